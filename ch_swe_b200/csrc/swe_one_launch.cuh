// swe_one_launch.cuh -- host-side entry points of the one-launch stage (swe_onepass.cuh) of
// one precision, shared by the C ABI and the translation units that build it.
#pragma once

#include "swe_launch.cuh"
#include "swe_vec.cuh"

namespace chswe {

// Per panel side, along the side (k_one_tables): JQ12 at across nodes 1..5 (lines 0-4), J Qn at
// across centres 1..3 (5-7) and 1/J there (8-10), J Qt and 1/J on the edge line (11, 12).
constexpr int ONE_LINES = 13;
enum { OS_JQ12 = 0, OS_JQN = 5, OS_IJN = 8, OS_JQT = 11, OS_IJT = 12 };

// Edge vectors: the vectors that hold a closure output of an x stencil.  Their VW outputs
// are a dense combination of eight consecutive inputs (ONE_TAPS weights of VW values
// per operator and edge vector, xrow42 rows on the window); the difference of h adds a
// ninth, the neighbour's vertex value of the gradient SAT.
constexpr int ONE_TAPS = 9, ONE_EDGES = 6;

// Scales of the kernel's interpolations and differences (swe_onepass.cuh, one_row).
constexpr double ONE_IS = -16.0, ONE_DS = -24.0;

template <class T>
struct OneMetric {
    const T *side;           // [4][ONE_LINES][n]
    const T *we;             // [4 operators][ONE_EDGES][ONE_TAPS][VW], scaled
    const T *xr;             // xrow42_table's rows, scaled
    const T *ea, *ef;        // 1/(J a) and f J^2 of the boundary vertices (MetricView)
    const T *qb, *qt, *ql, *qr;
    T inv_hx;
    T cd, cg;                // 1 / (ONE_DS hx), -g / (ONE_DS hx a)
};

// The dense weights of the edge vectors of a cube of N cells (OneMetric::we), VW outputs per
// vector: [operator][edge vector][tap][output].
static inline void one_edge_table(int N, int VW, double *we)
{
    const int n = N + 1, HV = 4 / VW, vr = (n - 4) / VW;
    const double satw[3] = {sbp::SATI1, sbp::SATI2, sbp::SATI3};
    double tab[XROW_LEN];
    xrow42_table(tab);
    for (int q = 0; q < XROW_OPS * ONE_EDGES * ONE_TAPS * VW; q++) we[q] = 0.0;
    for (int op = 0; op < XROW_OPS; op++) {
        const bool c2i = op <= 1;
        const int nm = c2i ? n : N, nin = c2i ? N : n;     // outputs, inputs
        for (int v = 0; v < (n + VW - 1) / VW; v++) {
            int ve, b;
            if (v < HV) { ve = v; b = 1; }
            else if (v >= vr) { ve = HV + (v - vr); b = nin - 7; }
            else continue;
            for (int e = 0; e < VW; e++) {
                const int k = VW * v + 1 + e;
                if (k > nm) continue;
                int row, base;
                if (k <= (c2i ? 4 : 3)) { row = k - 1; base = 1; }
                else if (k > (c2i ? nm - 4 : nm - 3)) { row = 4 + nm - k; base = c2i ? nm - 5 : nm - 3; }
                else { row = 8; base = c2i ? k - 2 : k - 1; }
                double *w = we + ((size_t)op * ONE_EDGES + ve) * ONE_TAPS * VW + e;
                for (int m = 0; m < 5; m++) {
                    const double c = tab[(op * XROW_ROWS + row) * 5 + m];
                    if (c != 0.0) w[(base + m - b) * VW] += c;
                }
                // the gradient SAT: satw (h(1) - halo) on the first rows, satw (halo - h(n)) on the last
                if (op == 3 && k <= 3) { w[(1 - b) * VW] += satw[k - 1]; w[8 * VW] -= satw[k - 1]; }
                if (op == 3 && k >= N - 2) { w[(n - b) * VW] -= satw[N - k]; w[8 * VW] += satw[N - k]; }
                for (int m = 0; m < ONE_TAPS; m++) w[m * VW] *= (op & 1) ? ONE_DS : ONE_IS;
            }
        }
    }
}


// Configurations: (label, XL, TH, blocks per SM, registers per thread).  The label is the
// public tile size, at least the rows of the configuration's tiles.
#define CHSWE_ONE_CFGS_F(X) X(17, 15, 14, 2, 72) X(25, 15, 18, 2, 64) X(33, 9, 28, 2, 72)
#define CHSWE_ONE_CFGS_D(X) X(17, 29, 17, 1, 72) X(25, 14, 25, 1, 96) X(33, 18, 28, 1, 80)

// Balanced tiles: the first rx (ry) tiles hold qx + 1 vectors (qy + 1 rows), the others qx (qy).
struct OneTiles {
    int qx, rx, qy, ry;
};

struct OneGrid {
    dim3 g;
    OneTiles t;
    int sides;   // panel sides a tile can touch
};

constexpr int ONE_WAVE = 148;   // SMs: blocks of a kernel that takes an SM each

// Tiles of at most XL - 2 HV vectors by TH rows, balanced.  The rows per tile are the
// division with the least work on the busiest SM: blocks per SM times (rows + 6), the
// window rows that the widest pass computes.  A panel with several tiles per direction
// needs seven points in each of them.  fits(sides): whether a block with the band threads of that
// many panel sides fits the register file; a division whose blocks do not is passed over, so that
// the cube, not the number of its members, decides whether a configuration is available.
template <class T, class Fits>
static inline bool one_grid(int N, int members, int xl, int th, int occ, const Fits &fits, OneGrid &og)
{
    constexpr int VW = OV<T>::W, HV = 4 / VW;
    const int n = N + 1, nv = (n + VW - 1) / VW, wv = xl - 2 * HV;
    const int gx = (nv + wv - 1) / wv;
    if (gx > 1 && (nv / gx - 1) * VW + 1 < 9) return false;
    int best = 0;
    long long cost = 0;
    for (int gy = (n + th - 1) / th; gy <= n; gy++) {
        if (gy > 1 && n / gy < 7) break;
        const long long blocks = (long long)gx * gy * NPAN * members, per = (blocks + ONE_WAVE - 1) / ONE_WAVE;
        const long long c = per * ((n + gy - 1) / gy + 6);
        if (fits((gx == 1 ? 2 : 1) + (gy == 1 ? 2 : 1)) && (!best || c < cost)) { best = gy; cost = c; }
        if (best && blocks > 8LL * ONE_WAVE * occ) break;
    }
    if (!best) return false;
    og.g = dim3(gx, best, NPAN * members);
    og.t = OneTiles{nv / gx, nv % gx, n / best, n % best};
    og.sides = (gx == 1 ? 2 : 1) + (best == 1 ? 2 : 1);
    return true;
}

template <class T>
struct OneTU {
    static cudaError_t optin();
    // box width and rows of the tile loads of configuration (label, occ); false: not built
    static bool box(int label, int occ, int &w, int &h);
    static bool grid(int label, int occ, int N, int members, OneGrid &g);
    static bool stage(int label, int occ, int members, const CUtensorMap &tmY, const CUtensorMap &tmM, const T *y, T *v0,
                      T *y1, T *acc, T *cmp, const Dims &d, const OneMetric<T> &om, const StageArgs &a, int *err,
                      cudaStream_t st);
    static void tables(const T *fmet, T *side, const Dims &d, cudaStream_t st);
    static cudaError_t upload_tables(const Link *links);
};

}  // namespace chswe
