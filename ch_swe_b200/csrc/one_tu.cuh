// one_tu.cuh -- definitions of OneTU (swe_one_launch.cuh), included by the one_*.cu
// translation units only.
#pragma once

#include "swe_onepass.cuh"

namespace chswe {

#define CHSWE_ONE_EACH(X)               \
    if constexpr (sizeof(T) == 4) {     \
        CHSWE_ONE_CFGS_F(X)             \
    } else {                            \
        CHSWE_ONE_CFGS_D(X)             \
    }

// A block's warps are spread over the SM's four partitions of 16384 registers each.
static inline bool one_fits(int warps, int regs) { return (warps + 3) / 4 * 32 * regs <= 16384; }

template <class T, int XL, int TH, int REGS>
static cudaError_t one_optin()
{
    return cudaFuncSetAttribute(k_onepass<T, XL, TH, REGS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)OneLayout<T, XL, TH>::bytes(4));
}

template <class T>
cudaError_t OneTU<T>::optin()
{
    cudaError_t e = cudaSuccess;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS) \
    if (e == cudaSuccess) e = one_optin<T, XL, TH, REGS>();
    CHSWE_ONE_EACH(CHSWE_O)
#undef CHSWE_O
    return e;
}

template <class T>
bool OneTU<T>::box(int label, int occ, int &w, int &h)
{
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)        \
    if (label == LABEL && occ == OCC) {    \
        w = OneLayout<T, XL, TH>::SW;      \
        h = OneLayout<T, XL, TH>::SR;      \
        return true;                       \
    }
    CHSWE_ONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
bool OneTU<T>::grid(int label, int occ, int N, int members, OneGrid &g)
{
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)  \
    if (label == LABEL && occ == OCC)      \
        return one_grid<T>(N, members, XL, TH, OCC,        \
                           [](int sides) { return one_fits((OneLayout<T, XL, TH>::NM + sides * ONE_BAND) / 32, REGS); }, g);
    CHSWE_ONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
bool OneTU<T>::stage(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmM, const T *y, T *v0,
                     T *y1, T *acc, T *cmp, const Dims &d, const OneMetric<T> &om, const StageArgs &a, int *err,
                     cudaStream_t st)
{
    OneGrid og;
    if (!grid(label, occ, d.N, members, og)) return false;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)                                                                            \
    if (label == LABEL && occ == OCC) {                                                                              \
        launch_k(k_onepass<T, XL, TH, REGS>, og.g, dim3(OneLayout<T, XL, TH>::NM + og.sides * ONE_BAND),             \
                 OneLayout<T, XL, TH>::bytes(og.sides), st, tmY, tmM, y, v0, y1, acc, cmp, d, om, og.t, a, err);     \
        return true;                                                                                                 \
    }
    CHSWE_ONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
void OneTU<T>::tables(const T *fmet, T *side, const Dims &d, cudaStream_t st)
{
    k_one_tables<T><<<dim3((d.N + 1 + 127) / 128, 4), 128, 0, st>>>(fmet, side, d);
}

// This translation unit's copies of the panel links and the closure rows.
template <class T>
static cudaError_t one_upload(const Link *links)
{
    cudaError_t e = cudaMemcpyToSymbol(c_link, links, sizeof(Link) * NPAN * 4);
    double w[XROW_LEN];
    T wt[XROW_LEN];
    xrow42_table(w);
    for (int m = 0; m < XROW_LEN; m++) wt[m] = T(w[m]);
    if (e == cudaSuccess) {
        if constexpr (sizeof(T) == 4) e = cudaMemcpyToSymbol(g_xrow_f, wt, sizeof(wt));
        else e = cudaMemcpyToSymbol(g_xrow_d, wt, sizeof(wt));
    }
    return e;
}

template <class T>
cudaError_t OneTU<T>::upload_tables(const Link *links)
{
    return one_upload<T>(links);
}

}  // namespace chswe
