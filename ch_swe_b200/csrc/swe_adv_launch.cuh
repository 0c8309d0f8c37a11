// swe_adv_launch.cuh -- host-side entry points of the advective operator's vector kernels
// (swe_advone.cuh) of one precision.
#pragma once

#include "swe_advective.cuh"
#include "swe_one_launch.cuh"

namespace chswe {

// Configurations of k_adv_stage and k_adv_co2: (label, XL, TH, blocks per SM, registers).
#define CHSWE_ADVONE_CFGS_F(X) X(25, 15, 18, 2, 72) X(33, 9, 28, 2, 72)
#define CHSWE_ADVONE_CFGS_D(X) X(17, 18, 14, 2, 72) X(25, 14, 18, 2, 72) X(33, 18, 28, 1, 80)

template <class T>
struct AdvOneTU {
    static cudaError_t optin();
    static bool box(int label, int occ, int &w, int &h);
    static bool grid(int label, int occ, int N, int members, OneGrid &g);
    static bool co2(int label, int occ, int members, const CUtensorMap &tmY, T *w, const Dims &d, const OneMetric<T> &om,
                    const T *fmet, const double *dtm, int *err, cudaStream_t st);
    static void flux(int members, const T *y, const T *w, T *f, const Dims &d, const AdvView<T> &av, const MetricView<T> &m,
                     const double *dtm, cudaStream_t st);
    // FP32 only (C96 / C384 per RK4 step 82 / 252 us; with k_advt 89 / 278 and 95 / 315 at older tile
    // shapes).  FP64 runs the tiled k_advt; k_adv_tend there, measured at the present shapes: C48 73.5
    // against 75.2 us, C96 81.8 / 86.6, C128 124 / 139, C192 163 / 164, C256 226 / 222, C384 411 / 405, 16 x
    // C48 260 / 270: faster below C192, slower above.  false: not launched
    static bool tend(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmW, const T *vh, T *adt,
                     const Dims &d, const AdvView<T> &av, const OneMetric<T> &om, T inv_hxa, const double *dtm, int *err,
                     cudaStream_t st);
    static bool stage(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmW, const CUtensorMap &tmF,
                      const CUtensorMap &tmM, const T *w, T *v0, T *y1, T *acc, T *cmp, const Dims &d, const OneMetric<T> &om,
                      const StageArgs &a, int *err, cudaStream_t st);
    static cudaError_t upload_tables(const Link *links);
};

}  // namespace chswe
