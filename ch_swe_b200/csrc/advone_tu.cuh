// advone_tu.cuh -- definitions of AdvOneTU (swe_adv_launch.cuh), included by the advone_*.cu
// translation units only.
#pragma once

#include "one_tu.cuh"
#include "swe_advone.cuh"

namespace chswe {

#define CHSWE_ADVONE_EACH(X)            \
    if constexpr (sizeof(T) == 4) {     \
        CHSWE_ADVONE_CFGS_F(X)          \
    } else {                            \
        CHSWE_ADVONE_CFGS_D(X)          \
    }

template <class T, int XL, int TH, int REGS>
static cudaError_t advone_optin()
{
    cudaError_t e = cudaFuncSetAttribute(k_adv_stage<T, XL, TH, REGS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)AdvLayout<T, XL, TH>::bytes(4));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_adv_co2<T, XL, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)CoLayout<T, XL, TH>::bytes());
    if constexpr (sizeof(T) == 4)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_adv_tend<T, XL, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)TendLayout<T, XL, TH>::bytes());
    return e;
}

template <class T>
cudaError_t AdvOneTU<T>::optin()
{
    cudaError_t e = cudaSuccess;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS) \
    if (e == cudaSuccess) e = advone_optin<T, XL, TH, REGS>();
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return e;
}

template <class T>
bool AdvOneTU<T>::box(int label, int occ, int &w, int &h)
{
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)  \
    if (label == LABEL && occ == OCC) {    \
        w = OneLayout<T, XL, TH>::SW;      \
        h = OneLayout<T, XL, TH>::SR;      \
        return true;                       \
    }
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
bool AdvOneTU<T>::grid(int label, int occ, int N, int members, OneGrid &g)
{
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)                   \
    if (label == LABEL && occ == OCC)                       \
        return one_grid<T>(N, members, XL, TH, OCC,         \
                           [](int sides) { return one_fits((AdvLayout<T, XL, TH>::NM + sides * ONE_BAND) / 32, REGS); }, g);
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
bool AdvOneTU<T>::co2(int label, int occ, int members, const CUtensorMap &tmY, T *w, const Dims &d, const OneMetric<T> &om,
                      const T *fmet, const double *dtm, int *err, cudaStream_t st)
{
    OneGrid og;
    if (!grid(label, occ, d.N, members, og)) return false;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)                                                                            \
    if (label == LABEL && occ == OCC) {                                                                              \
        launch_k(k_adv_co2<T, XL, TH>, og.g, dim3(CoLayout<T, XL, TH>::NM), CoLayout<T, XL, TH>::bytes(), st, tmY, w, \
                 d, om, fmet, og.t, dtm, err);                                                                       \
        return true;                                                                                                 \
    }
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
bool AdvOneTU<T>::tend(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmW, const T *vh, T *adt,
                       const Dims &d, const AdvView<T> &av, const OneMetric<T> &om, T inv_hxa, const double *dtm, int *err,
                       cudaStream_t st)
{
    OneGrid og;
    if (sizeof(T) == 8 || !grid(label, occ, d.N, members, og)) return false;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)                                                                               \
    if (label == LABEL && occ == OCC) {                                                                                 \
        if constexpr (sizeof(T) == 4)                                                                                   \
        launch_k(k_adv_tend<T, XL, TH>, og.g, dim3(TendLayout<T, XL, TH>::NM), TendLayout<T, XL, TH>::bytes(), st, tmY, \
                 tmW, vh, adt, d, av, om, inv_hxa, og.t, dtm, err);                                                     \
        return true;                                                                                                    \
    }
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
void AdvOneTU<T>::flux(int members, const T *y, const T *w, T *f, const Dims &d, const AdvView<T> &av, const MetricView<T> &m,
                       const double *dtm, cudaStream_t st)
{
    const int n = d.N + 1, nv = (n + OV<T>::W - 1) / OV<T>::W, gx = (nv + 31) / 32, ny = (n + 7) / 8;
    const int ne = (flux_edge_items(d.N, OV<T>::W) + 256 * gx - 1) / (256 * gx);
    launch_k(k_adv_flux<T>, dim3(gx, ny + ne, NPAN * members), dim3(32, 8), 0, st, y, w, f, d, av, m, ny, dtm);
}

template <class T>
bool AdvOneTU<T>::stage(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmW, const CUtensorMap &tmF,
                        const CUtensorMap &tmM, const T *w, T *v0, T *y1, T *acc, T *cmp, const Dims &d,
                        const OneMetric<T> &om, const StageArgs &a, int *err, cudaStream_t st)
{
    OneGrid og;
    if (!grid(label, occ, d.N, members, og)) return false;
#define CHSWE_O(LABEL, XL, TH, OCC, REGS)                                                                              \
    if (label == LABEL && occ == OCC) {                                                                                \
        launch_k(k_adv_stage<T, XL, TH, REGS>, og.g, dim3(AdvLayout<T, XL, TH>::NM + og.sides * ONE_BAND),             \
                 AdvLayout<T, XL, TH>::bytes(og.sides), st, tmY, tmW, tmF, tmM, w, v0, y1, acc, cmp, d, om, og.t, a, err); \
        return true;                                                                                                   \
    }
    CHSWE_ADVONE_EACH(CHSWE_O)
#undef CHSWE_O
    return false;
}

template <class T>
cudaError_t AdvOneTU<T>::upload_tables(const Link *links)
{
    return one_upload<T>(links);
}

}  // namespace chswe
