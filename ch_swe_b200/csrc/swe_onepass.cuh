// swe_onepass.cuh -- the one-launch stage of the linear operator on the Ch grid (SBP 4-2):
// one kernel per RK stage computes everything from the stage input -- contravariant
// components (co2contra_Ch_mod.f90:27-94), gradient with its SAT, Coriolis term with the
// ECS vector edge sync (ecs_Ah_vec_sync_mod.f90:62-125), divergence with its SAT and
// scalar edge sync (halo_Ah_scalar_sync_mod.f90:43-98), the tendency
// (operator_swm_lin_mod.f90:66-108) and the RK4 update (rk4_mod.f90:28-40).
//
// A tile that touches a panel edge computes the neighbour panel's raw boundary values
// itself, from a band of the neighbour's (u, v) along the shared side, so a stage needs no
// edge-strip and no edge-sync launch before it: an RK4 step is four launches.
//
// Lanes work on vectors of VW consecutive columns (one 16-byte word: four FP32 or two FP64
// points).  Point (i, j) of a panel box lies at column i + 3, so vector v holds the points
// VW v + 1 .. VW v + VW and is 16-byte aligned in global and in shared memory.  A block
// owns a tile of up to XL - 2 HV vectors by TH rows; its windows (h, u, v and seven metric
// boxes, the tile plus four points on every side) come by TMA.  Main thread (x, y) takes
// window vector x and row y of every pass: y stencils read four vectors of the column, x
// stencils the own vector and the three points beside it.  ONE_BAND further threads per
// touched side carry the boundary through loads, contravariant components and syncs beside
// the passes and meet the main threads twice (named barriers): for the own panel's copies
// after P2, and before P4.
//
// What bounds it, and why it has this shape (B200, C192 FP32 unless said otherwise).  The
// former stage was three dependent launches (edge strips or contravariant components, edge
// sync, tiles), about 21 us at any cube size up to C192, of which the kernels' own work was
// under half: an RK4 step took 86 us, C24 55 us.  One launch takes 7.6 us per stage (30.6 us
// per step; 22.3 us per step with three contexts at once).  A first version with 192 threads
// per block, two rows per thread and the boundary as a loop of the same threads ran 17 us per
// stage even at C24: the boundary's chain of dependent loads stood in the passes' way; its
// threads of their own brought C24 to 6 us.  A stage's time now is one memory round trip for the
// windows (0.8 us), four passes of 0.4 to 0.9 us and the RK4 stores; ncu counts 21 % of the L2
// throughput, 58 % of the L1's and 39 % of the shared-memory wavefronts at C384, issue slots 36 %
// busy: latency and shared-memory traffic, not arithmetic (three instead of four operations per stencil and
// packed FP32 changed nothing at C192).  Assigning the vectors of a pass to threads one after
// another, without idle lanes, saved 14 % of the instructions and ran 5 to 25 % slower: the
// rows' ends conflict in shared memory and fewer warps hide the latency.
//
// Ranges of the passes (x; y is symmetric) for tile [i0, i1), clipped to the panel:
//   vq  = JQ12 I_c2i,y(v)          nodes   [i0-3, i1+3)
//   uq  = JQ12 I_c2i,x(u)          nodes   [i0-1, i1+2)
//   Jut = JQ11 u + I_i2c,x(vq)     centres [i0-2, i1+1)     (ut = Jut / J)
//   Jvt = JQ22 v + I_i2c,y(uq)     nodes   [i0-1, i1+2)     (vt = Jvt / J)
//   up  = fJ2 I_c2i,y(vt)          nodes   [i0-1, i1+2)
//   vp  = -fJ2 I_c2i,x(ut)         nodes   [i0, i1)
//   div = (D_c2i,x Jut + D_c2i,y Jvt) / (hx J a)  on the tile
// Tiles are at least 7 points wide and high whenever a panel holds more than one, so the
// points computed beyond a tile that is not the last take interior rows only.
#pragma once

#include "swe_one_launch.cuh"

namespace chswe {


// XL: window vectors per row; TH: maximal tile rows.  Main threads: XL x YG, one window row
// each in every pass (YG >= TH + 6, the rows of the widest pass), whole warps; then
// ONE_BAND threads per touched panel side, one per along-edge point of its band.
// The shape decides more than anything else: it has to divide the panels without a remainder
// wave or idle lanes.  FP32 7 x 28 (XL 9) against 8 x 30 (XL 10), per RK4 step: C192 30.6 /
// 33.4 us (294 blocks, two per SM, either way), 256 x C48 577 / 639; FP64 14 x 28 against
// 12 x 30: C192 69 / 84 us (two full waves / three).
constexpr int ONE_BAND = 64;

template <class T, int XL, int TH>
struct OneLayout {
    static constexpr int VW = OV<T>::W, HV = 4 / VW;      // points per vector, halo vectors per side
    static constexpr int WV = XL - 2 * HV;                // tile vectors
    static constexpr int SW = XL * VW, SR = TH + 8;       // window points per row, rows
    static constexpr int YG = TH + 6, NM = (XL * YG + 31) / 32 * 32;
    static constexpr int BOX_BYTES = SW * SR * (int)sizeof(T);
    static constexpr int SLOT_BYTES = (BOX_BYTES + 127) / 128 * 128;
    static constexpr int SLOT = SLOT_BYTES / (int)sizeof(T);
    static constexpr int NLOAD = 10, NSLOT = 14;
    static constexpr int TP = TH > WV * VW ? TH : WV * VW;  // points of a tile along a side
    static constexpr int LB = ONE_BAND + 8;               // band line: lanes and the reach of closure taps
    static constexpr int BAND = 8 * LB;                   // TF 0..4, nq, J t, t of one side
    static constexpr int HL = TP + 8;
    static constexpr int HALO = NSLOT * SLOT;             // four lines: the neighbours' h
    static constexpr int DIVB = HALO + 4 * HL;            // four lines: the synchronised divergence
    static constexpr int BAR = DIVB + 4 * HL;             // the mbarrier (16 bytes)
    static constexpr int XR = BAR + VW;                   // the closure rows (xrow42_table)
    static constexpr int WE = XR + (XROW_LEN + VW - 1) / VW * VW;   // the edge-vector weights
    static constexpr int CORN = WE + XROW_OPS * ONE_EDGES * ONE_TAPS * VW;   // corner exchange, 4 x 2 x 8
    static constexpr int BANDS = CORN + 64;
    static_assert(TP + 6 <= ONE_BAND, "a side's band is one point per thread");
    static size_t bytes(int sides) { return (size_t)(BANDS + sides * BAND) * sizeof(T); }
};

// Band lines
enum { OB_TF = 0, OB_NQ = 5, OB_JT = 6, OB_T = 7 };

// Named barriers: the main threads' passes; main to band (J ut, J vt are there); band to
// main (the boundary vertices are there); all band threads (corners); one per side.
// bar.sync and bar.arrive are the aligned forms: every thread of the warp has to execute the
// same one together, so the warp reconverges first (the barriers follow divergent branches:
// thread 0's tile loads, the band threads' boundary and corner points).
enum { BAR_MAIN = 1, BAR_P2 = 2, BAR_BND = 3, BAR_CORN = 4, BAR_SIDE = 5 };
__device__ __forceinline__ void nbar_sync(int id, int cnt)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(cnt) : "memory");
}
__device__ __forceinline__ void nbar_arrive(int id, int cnt)
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(cnt) : "memory");
}

// The inputs of VW consecutive outputs of an interior x row: c2i own-2 .. own+VW (SH = -2),
// i2c own-1 .. own+VW+1 (SH = -1).
template <int SH, class T>
__device__ __forceinline__ void one_window(const T *p, T (&w)[OV<T>::W + 3])
{
    constexpr int W = OV<T>::W;
    const OV<T> o = *reinterpret_cast<const OV<T> *>(p);
#pragma unroll
    for (int e = 0; e < W; e++) w[e - SH] = o.a[e];
    if constexpr (sizeof(T) == 4) {
        if constexpr (SH == -2) {
            const float2 l = *reinterpret_cast<const float2 *>(p - 2);
            w[0] = l.x;
            w[1] = l.y;
            w[W + 2] = p[W];
        } else {
            const float2 r = *reinterpret_cast<const float2 *>(p + W);
            w[0] = p[-1];
            w[W + 1] = r.x;
            w[W + 2] = r.y;
        }
    } else {
        if constexpr (SH == -2) {
            const OV<T> l = *reinterpret_cast<const OV<T> *>(p - 2);
            w[0] = l.a[0];
            w[1] = l.a[1];
            w[W + 2] = p[W];
        } else {
            const OV<T> r = *reinterpret_cast<const OV<T> *>(p + W);
            w[0] = p[-1];
            w[W + 1] = r.a[0];
            w[W + 2] = r.a[1];
        }
    }
}

// Interior rows.  Every operator of this kernel is scaled, interpolations by -16 and
// differences by -24: three operations per output, the scales folded into the constants
// and metric products that follow (ONE_IS, ONE_DS; the closure weights carry them too).
template <bool D, class T>
__device__ __forceinline__ T one_row(T v0, T v1, T v2, T v3)
{
    return D ? fma(T(-27), v2 - v1, v3 - v0) : fma(T(-9), v2 + v1, v3 + v0);
}
template <bool D, class T>
__device__ __forceinline__ OV<T> one_row4(const OV<T> &a, const OV<T> &b, const OV<T> &c, const OV<T> &d)
{
    if constexpr (D) return ov_fma(ov_all(T(-27)), ov_sub(c, b), ov_sub(d, a));
    else return ov_fma(ov_all(T(-9)), ov_add(c, b), ov_add(d, a));
}

// An edge vector: the dense weights of operator OP on the inputs row[0 .. 7].  Most are zero, so
// an infinity or NaN among the inputs reaches all outputs of the vector (and all rows that share
// the five taps of a y closure or of a band).  Forming such sums again without the zero taps
// gives the split kernels' pattern and costs 2 to 12 % of an RK4 step (C192 FP32 30.7 -> 33.2
// us): the check stands in every pass's chain.
template <int OP, class T>
__device__ __forceinline__ OV<T> one_edge(const T *row, const T *we)
{
    constexpr int W = OV<T>::W;
    OV<T> r = ov_mul(*reinterpret_cast<const OV<T> *>(we), ov_all(row[0]));
#pragma unroll
    for (int m = 1; m < 8; m++) r = ov_fma(*reinterpret_cast<const OV<T> *>(we + m * W), ov_all(row[m]), r);
    return r;
}

// Operator OP (0 I_c2i, 1 D_c2i, 2 I_i2c, 3 D_i2c) along x on the VW outputs at p; ve >= 0:
// an edge vector, whose inputs start eo points from p.
template <int OP, class T>
__device__ __forceinline__ OV<T> one_x(const T *p, int ve, int eo, const T *we)
{
    constexpr int W = OV<T>::W;
    if (ve >= 0) return one_edge<OP, T>(p + eo, we + (OP * ONE_EDGES + ve) * ONE_TAPS * W);
    T w[W + 3];
    one_window<(OP <= 1 ? -2 : -1)>(p, w);
    OV<T> r;
#pragma unroll
    for (int e = 0; e < W; e++)
        r.a[e] = one_row<(OP & 1) != 0>(w[e], w[e + 1], w[e + 2], w[e + 3]);
    return r;
}

// The weight row of operator op (xrow42's rows) at output k of nm: first input and the table's row.
__device__ __forceinline__ void one_rowsel(int op, int k, int nm, int &base, int &w)
{
    const bool c2i = op <= 1;
    int row;
    if (k <= (c2i ? 4 : 3)) { row = k - 1; base = 1; }
    else if (k > (c2i ? nm - 4 : nm - 3)) { row = 4 + nm - k; base = c2i ? nm - 5 : nm - 3; }
    else { row = 8; base = c2i ? k - 2 : k - 1; }
    w = (op * XROW_ROWS + row) * 5;
}

// Operator OP along y at output l of nm on the column col (points at row index 0; times col2
// when MUL), rows SW apart: interior rows on four vectors, closure rows on five with the table xr.
template <int OP, bool MUL, int SW, class T>
__device__ __forceinline__ OV<T> one_y(const T *col, const T *col2, int l, int nm, const T *xr)
{
    constexpr bool C2I = OP <= 1, D = (OP & 1) != 0;
    auto at = [&](int r) {
        OV<T> v = ov_ld(col + r * SW);
        if constexpr (MUL) v = ov_mul(v, ov_ld(col2 + r * SW));
        return v;
    };
    if (C2I ? (l >= 5 && l <= nm - 4) : (l >= 4 && l <= nm - 3)) {
        const int b = C2I ? l - 2 : l - 1;
        return one_row4<D>(at(b), at(b + 1), at(b + 2), at(b + 3));
    }
    int base, w;
    one_rowsel(OP, l, nm, base, w);
    OV<T> r = ov_mul(ov_all(xr[w]), at(base));
#pragma unroll
    for (int m = 1; m < 5; m++) r = ov_fma(ov_all(xr[w + m]), at(base + m), r);
    return r;
}

// Raw quantities of one copy of a panel-boundary vertex in side coordinates (across the
// side, along it):
//   A = sum ic1 n, B = sum dc1 Jn, C = sum r1 Jn over the depths 1..3 of the normal component;
//   T1 = I_c2i(t), T2 = D_c2i(J t) along the edge line; K = sum r1 J t over the three centres
//   next to a panel corner.
template <class T>
struct OneRaw {
    T A, B, C, T1, T2, K;
};
// up / vp of a copy on side s from its raw quantities (coriolis_Ch_mod.f90:97-120).
template <class T>
__device__ __forceinline__ void one_vec(const OneRaw<T> &r, int s, T f, T &up, T &vp)
{
    up = f * (s <= SIDE_R ? r.T1 : r.A);
    vp = -f * (s <= SIDE_R ? r.A : r.T1);
}
// The divergence part across side s: the first c2i row and the SAT against the jump C - Ch.
template <class T>
__device__ __forceinline__ T one_across(const OneRaw<T> &r, int s, T Ch)
{
    const T sat = T(SbpOrder<42>::SATC) * (r.C - Ch);
    return (s == SIDE_L || s == SIDE_B) ? r.B + sat : -r.B - sat;
}

//   MODE 0: out = A(y);   1: Y1 = V0 + dt/2 k, ACC = dt/6 k;   2: Y1 = V0 + dt/2 k, ACC += dt/3 k;
//   3: Y1 = V0 + dt k, ACC += dt/3 k;   4: V0 += ACC + dt/6 k (FP32: Kahan with compensation CMP)
// Mode 1 takes V0 from the windows: its stage input is V0.
// The mode is an argument: one kernel serves the four stages of a step, whose code then
// stays in the instruction caches from one stage to the next.
template <class T, int XL, int TH, int REGS>
__global__ void __maxnreg__(REGS)
    k_onepass(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmM, const T *__restrict__ Yin,
              T *V0, T *Y1, T *ACC, T *CMP, Dims d, OneMetric<T> om, OneTiles ot, StageArgs a, int *err)
{
    using L = OneLayout<T, XL, TH>;
    using SB = SbpOrder<42>;
    using V = OV<T>;
    constexpr int VW = L::VW, HV = L::HV, SW = L::SW, NM = L::NM;
    extern __shared__ __align__(128) unsigned char osm_raw[];
    T *const sm = reinterpret_cast<T *>(osm_raw);
    T *const sH = sm, *const sU = sm + L::SLOT, *const sV = sm + 2 * L::SLOT, *const sJQ12 = sm + 3 * L::SLOT,
             *const sJQ11 = sm + 4 * L::SLOT, *const siJy = sm + 5 * L::SLOT, *const sJQ22 = sm + 6 * L::SLOT,
             *const siJx = sm + 7 * L::SLOT, *const sF = sm + 8 * L::SLOT, *const siJa = sm + 9 * L::SLOT,
             *const sVQ = sm + 10 * L::SLOT, *const sUQ = sm + 11 * L::SLOT, *const sJVT = sm + 12 * L::SLOT,
             *const sUT = sm + 13 * L::SLOT;
    // slots reused once their first contents are dead
    T *const sJUT = sJQ12, *const sUP = sVQ, *const sVP = sUQ;
    T *const hh = sm + L::HALO, *const db = sm + L::DIVB, *const xr = sm + L::XR, *const we = sm + L::WE;
    uint64_t *const bar = reinterpret_cast<uint64_t *>(sm + L::BAR);

    const int N = d.N, n = N + 1, P = d.P;
    const int t = blockIdx.z % NPAN, mem = blockIdx.z / NPAN;
    if (member_frozen(a.dtm, mem)) return;
    const int NV = (n + VW - 1) / VW, bx = blockIdx.x, by = blockIdx.y;
    const int v0 = bx * ot.qx + min(bx, ot.rx), v1 = v0 + ot.qx + (bx < ot.rx);
    const int i0 = 1 + VW * v0, i1 = min(1 + VW * v1, n + 1);
    const int j0 = 1 + by * ot.qy + min(by, ot.ry), j1 = j0 + ot.qy + (by < ot.ry);
    const int tid = threadIdx.x;
    const int rows = N + 1 + 2 * MG;
    // slot offset of point (i, j)
    auto SI = [&](int i, int j) { return (j - j0 + 4) * SW + (i - i0 + 4); };
    const T *const ym = Yin + (int64_t)mem * d.ms;
    // sides of the panel that the tile touches
    const unsigned touch = (i0 == 1 ? 1u : 0u) | (i1 == n + 1 ? 2u : 0u) | (j0 == 1 ? 4u : 0u) | (j1 == n + 1 ? 8u : 0u);
    const int nband = __popc(touch) * ONE_BAND;           // band threads at work in this block

    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(bar, (uint32_t)(L::NLOAD * L::BOX_BYTES));
        const int mr = j0 - 1, ax = i0 - 1;
        tma_load_2d(sJQ12, &tmM, bar, ax, FM_JQ12 * rows + mr);
        tma_load_2d(sJQ11, &tmM, bar, ax, FM_JQ11Y * rows + mr);
        tma_load_2d(siJy, &tmM, bar, ax, FM_IJY * rows + mr);
        tma_load_2d(sJQ22, &tmM, bar, ax, FM_JQ22X * rows + mr);
        tma_load_2d(siJx, &tmM, bar, ax, FM_IJX * rows + mr);
        tma_load_2d(sF, &tmM, bar, ax, (FM_FJ2 + t) * rows + mr);
        tma_load_2d(siJa, &tmM, bar, ax, FM_IJA * rows + mr);
        // the stage input: after the previous stage
        pdl_wait();
        const int yr = (mem * 3 * NPAN + t) * rows + (j0 - 1), fr = NPAN * rows;
        tma_load_2d(sH, &tmY, bar, ax, yr);
        tma_load_2d(sU, &tmY, bar, ax, yr + fr);
        tma_load_2d(sV, &tmY, bar, ax, yr + 2 * fr);
    }

    if (tid >= NM) {
        // =================== the band threads: the neighbours' copies of the boundary ===================
        // Thread b of a side takes the along-edge index al = a0 - 3 + b in this panel's order (node al
        // and centre al); the neighbour's line runs the other way when the link is reversed.
        const int bt = tid - NM, slot = bt / ONE_BAND, b = bt % ONE_BAND;
        if (bt >= nband) return;
        int s = 0;                                        // the slot-th touched side
        for (int q = 0, c = -1; q < 4; q++)
            if (touch >> q & 1) {
                c++;
                if (c == slot) s = q;
            }
        const Link K = c_link[t][s];
        const bool lr = s <= SIDE_R, nlr = K.nside <= SIDE_R, far = (K.nside == SIDE_R || K.nside == SIDE_T);
        const int a0 = lr ? j0 : i0, a1 = lr ? j1 : i1, al = a0 - 3 + b;
        T *const bd = sm + L::BANDS + slot * L::BAND;
        const bool node = al >= 1 && al <= n && al <= a1 + 2, cen = al >= 1 && al <= N && al <= a1 + 2;
        const int y = K.rev ? n + 1 - al : al, yc = K.rev ? N + 1 - al : al;     // the neighbour's node and centre
        // ---- before the previous stage completes: metric and weight rows of this point
        T q12[5], qn[3], ijn[3], qt = T(0), ijt = T(0), wI[5], wD[5], wC[5];
        T fo = T(0), fn = T(0), eao = T(0), ean = T(0), qs = T(0);
        int bI = 1, bC = 1;
        const T *const tab = om.side + K.nside * ONE_LINES * n - 1;
#pragma unroll
        for (int x = 0; x < 5; x++) q12[x] = node ? __ldg(tab + (OS_JQ12 + x) * n + y) : T(0);
#pragma unroll
        for (int x = 0; x < 3; x++) {
            qn[x] = node ? __ldg(tab + (OS_JQN + x) * n + y) : T(0);
            ijn[x] = node ? __ldg(tab + (OS_IJN + x) * n + y) : T(0);
        }
#pragma unroll
        for (int m = 0; m < 5; m++) wI[m] = wD[m] = wC[m] = T(0);
        const T *const gx = xrow_table<T>();
        if (node) {
            fo = T(ONE_IS) * __ldg(om.ef + (t * 4 + s) * n + al - 1);
            fn = T(ONE_IS) * __ldg(om.ef + (K.nb * 4 + K.nside) * n + y - 1);
            eao = __ldg(om.ea + s * n + al - 1);
            ean = __ldg(om.ea + K.nside * n + y - 1);
            qs = __ldg((s == SIDE_L ? om.ql : (s == SIDE_R ? om.qr : (s == SIDE_B ? om.qb : om.qt))) + al - 1);
            int w, w2, b2;
            one_rowsel(0, al, n, bI, w);
            one_rowsel(1, al, n, b2, w2);
#pragma unroll
            for (int m = 0; m < 5; m++) {
                wI[m] = __ldg(gx + w + m);
                wD[m] = __ldg(gx + w2 + m);
            }
        }
        if (cen) {
            qt = __ldg(tab + OS_JQT * n + yc);
            ijt = __ldg(tab + OS_IJT * n + yc);
            int w;
            one_rowsel(2, al, N, bC, w);
#pragma unroll
            for (int m = 0; m < 5; m++) wC[m] = __ldg(gx + w + m);
        }
        // a panel corner: the third panel is the neighbour across s2 (this thread's other side); the
        // signs of the second SATs
        const bool corner = al == 1 || al == n;
        const int s2 = lr ? (al == 1 ? SIDE_B : SIDE_T) : SIDE_L;
        T sn2 = T(0), sgx = T(0), sgy = T(0);
        bool y1 = false, y21 = false;
        if (corner && lr) {
            const Link K2 = c_link[t][s2];
            const int kc = s == SIDE_L ? 1 : n, y2 = K2.rev ? n + 1 - kc : kc;
            y1 = y == 1;
            y21 = y2 == 1;
            sn2 = T(K2.sn);
            sgx = T(c_link[K.nb][nlr ? (y1 ? SIDE_B : SIDE_T) : (y1 ? SIDE_L : SIDE_R)].sn);
            sgy = T(c_link[K2.nb][K2.nside <= SIDE_R ? (y21 ? SIDE_B : SIDE_T) : (y21 ? SIDE_L : SIDE_R)].sn);
        }
        // zeros beyond the band, which taps of weight zero read
        for (int q = b; q < L::BAND; q += ONE_BAND) bd[q] = T(0);
        nbar_sync(BAR_SIDE + slot, ONE_BAND);
        pdl_wait();
        // ---- the neighbour's band: TF at across nodes 1..5 (centre al), NF at across centres 1..3
        // (node al), h at the vertex
        const T *const yp = ym + (int64_t)K.nb * d.ps;
        const T *const gN = yp + (nlr ? 1 : 2) * d.fs, *const gT = yp + (nlr ? 2 : 1) * d.fs;
        T tf[5], nf[3];
#pragma unroll
        for (int x = 0; x < 5; x++) {
            const int xx = far ? n - x : x + 1;
            tf[x] = cen ? ld_cg(gT + (nlr ? box_off32(P, xx, yc) : box_off32(P, yc, xx))) : T(0);
        }
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const int xx = far ? n - (x + 1) : x + 1;
            nf[x] = node ? ld_cg(gN + (nlr ? box_off32(P, xx, y) : box_off32(P, y, xx))) : T(0);
        }
        if (al >= a0 && al < a1) {
            const int xx = far ? n : 1;
            hh[s * L::HL + al - a0] = ld_cg(yp + (nlr ? box_off32(P, xx, y) : box_off32(P, y, xx)));
        }
        // line offset of index i: i - a0 + 3
        auto ln = [&](int line) { return bd + line * L::LB - a0 + 3; };
#pragma unroll
        for (int x = 0; x < 5; x++) ln(OB_TF + x)[al] = tf[x];
        ln(OB_NQ)[al] = q12[0] * (T(SB::ic1(1)) * nf[0] + T(SB::ic1(2)) * nf[1] + T(SB::ic1(3)) * nf[2]);
        nbar_sync(BAR_SIDE + slot, ONE_BAND);
        // nodes whose stencils the band holds: the tile's and one before, one after
        const bool vx = node && al >= a0 - 1 && al <= a1 + 1;
        OneRaw<T> rn{};
        if (vx) {
            T tq[5], jn[3];
#pragma unroll
            for (int x = 0; x < 5; x++) {
                const T *f = ln(OB_TF + x) + bI;
                T v = T(0);
#pragma unroll
                for (int m = 0; m < 5; m++) v += wI[m] * f[m];
                tq[x] = q12[x] * v;
            }
            using namespace sbp;
            jn[0] = qn[0] * nf[0] + (T(II11) * tq[0] + T(II12) * tq[1] + T(II13) * tq[2] + T(II14) * tq[3]);
            jn[1] = qn[1] * nf[1] + (T(II21) * tq[0] + T(II22) * tq[1] + T(II23) * tq[2] + T(II24) * tq[3]);
            jn[2] = qn[2] * nf[2] + (T(II31) * tq[0] + T(II32) * tq[1] + T(II33) * tq[2] + T(II34) * tq[3] + T(II35) * tq[4]);
            rn.A = T(SB::ic1(1)) * (jn[0] * ijn[0]) + T(SB::ic1(2)) * (jn[1] * ijn[1]) + T(SB::ic1(3)) * (jn[2] * ijn[2]);
            rn.B = T(SB::dc1(1)) * jn[0] + T(SB::dc1(2)) * jn[1] + T(SB::dc1(3)) * jn[2];
            rn.C = T(SB::r1(1)) * jn[0] + T(SB::r1(2)) * jn[1] + T(SB::r1(3)) * jn[2];
        }
        if (cen && al >= a0 - 2 && al <= a1) {
            const T *f = ln(OB_NQ) + bC;
            T v = T(0);
#pragma unroll
            for (int m = 0; m < 5; m++) v += wC[m] * f[m];
            const T jt = qt * tf[0] + v;
            ln(OB_JT)[al] = jt;
            ln(OB_T)[al] = jt * ijt;
        }
        nbar_sync(BAR_SIDE + slot, ONE_BAND);
        const bool full = node && al >= a0 && al < a1;
        if (full) {
            const T *fj = ln(OB_JT) + bI, *ft = ln(OB_T) + bI;
#pragma unroll
            for (int m = 0; m < 5; m++) {
                rn.T1 += wI[m] * ft[m];
                rn.T2 += wD[m] * fj[m];
            }
            if (K.rev) rn.T2 = -rn.T2;
            const T *fk = ln(OB_JT);
            if (al == 1) rn.K = T(SB::r1(1)) * fk[1] + T(SB::r1(2)) * fk[2] + T(SB::r1(3)) * fk[3];
            if (al == n) rn.K = T(SB::r1(1)) * fk[N] + T(SB::r1(2)) * fk[N - 1] + T(SB::r1(3)) * fk[N - 2];
        }
        T un, vn, uh = T(0), vh = T(0);
        one_vec(rn, K.nside, fn, un, vn);
        halo_vec(t, s, un, vn, uh, vh);
        // ---- the own copy, from the tile's J ut, J vt
        nbar_sync(BAR_P2, NM + nband);
        OneRaw<T> ro{};
        int kk, ll;
        side_vertex(N, s, al, 0, kk, ll);
        if (vx) {
            const int o = s == SIDE_L ? SI(0, al) : (s == SIDE_R ? SI(n, al) : (s == SIDE_B ? SI(al, 0) : SI(al, n)));
            const int sd = s == SIDE_L ? 1 : (s == SIDE_R ? -1 : (s == SIDE_B ? SW : -SW));
            const T *const pj = (lr ? sJUT : sJVT) + o, *const pi = (lr ? siJy : siJx) + o;
            const T j1_ = pj[sd], j2_ = pj[2 * sd], j3_ = pj[3 * sd];
            ro.A = T(SB::ic1(1)) * (j1_ * pi[sd]) + T(SB::ic1(2)) * (j2_ * pi[2 * sd]) + T(SB::ic1(3)) * (j3_ * pi[3 * sd]);
            ro.B = T(SB::dc1(1)) * j1_ + T(SB::dc1(2)) * j2_ + T(SB::dc1(3)) * j3_;
            ro.C = T(SB::r1(1)) * j1_ + T(SB::r1(2)) * j2_ + T(SB::r1(3)) * j3_;
        }
        if (full) {
            const int sc = lr ? SW : 1, o = lr ? SI(kk, 0) : SI(0, ll);
            const T *const pt = (lr ? sJVT : sJUT) + o, *const pi = (lr ? siJx : siJy) + o;
#pragma unroll
            for (int m = 0; m < 5; m++) {
                // the fifth weight of an interior row is zero and its input may not exist
                const bool use = m < 4 || wI[4] != T(0) || wD[4] != T(0);
                const T v = use ? pt[(bI + m) * sc] : T(0), w = use ? v * pi[(bI + m) * sc] : T(0);
                ro.T1 += wI[m] * w;
                ro.T2 += wD[m] * v;
            }
            if (al == 1) ro.K = T(SB::r1(1)) * pt[sc] + T(SB::r1(2)) * pt[2 * sc] + T(SB::r1(3)) * pt[3 * sc];
            if (al == n) ro.K = T(SB::r1(1)) * pt[N * sc] + T(SB::r1(2)) * pt[(N - 1) * sc] + T(SB::r1(3)) * pt[(N - 2) * sc];
        }
        T up, vp;
        one_vec(ro, s, fo, up, vp);
        const T dn = one_across(rn, K.nside, T(K.sn) * ro.C) + rn.T2, dv = one_across(ro, s, T(K.sn) * rn.C) + ro.T2;
        if (vx && !full) {
            // beyond the tile only the component along the side is read
            if (lr) sVP[SI(kk, ll)] = T(0.5) * (vp + vh);
            else sUP[SI(kk, ll)] = T(0.5) * (up + uh);
        } else if (full && !corner) {
            sUP[SI(kk, ll)] = lr ? T(0.5) * (up + uh + qs * vh) : T(0.5) * (up + uh);
            sVP[SI(kk, ll)] = lr ? T(0.5) * (vp + vh) : T(0.5) * (vp + vh + qs * uh);
            db[s * L::HL + al - a0] = T(0.5) * (dv * om.inv_hx * eao + dn * om.inv_hx * ean);
        }
        const bool cornered = (touch & 3u) && (touch & 12u);
        if (cornered) {
            // the panel corners: the bottom / top side's thread hands its copy to the left / right side's
            const int end = al == 1 ? 0 : 1;
            if (full && corner && !lr) {
                T *c = sm + L::CORN + (s * 2 + end) * 8;
                c[0] = uh; c[1] = vh; c[2] = rn.C; c[3] = rn.K; c[4] = dn; c[5] = qs; c[6] = ean;
            }
            nbar_sync(BAR_CORN, nband);
            if (full && corner && lr) {
                const T *c = sm + L::CORN + (s2 * 2 + (kk == 1 ? 0 : 1)) * 8;
                const T satc = T(SB::SATC);
                // the second SAT at the corner, of every copy: own across s2 (its normal component next
                // to the corner is the tangential one of side s), the neighbour's toward the third panel
                // and the third panel's toward the neighbour
                const T jo = satc * (ro.K - sn2 * c[2]), jx = satc * (rn.K - sgx * c[3]), jy = satc * (c[3] - sgy * rn.K);
                const T d0 = al == 1 ? dv + jo : dv - jo, d1 = y1 ? dn + jx : dn - jx, d2 = y21 ? c[4] + jy : c[4] - jy;
                const T sdiv = (d0 * om.inv_hx * eao + d1 * om.inv_hx * ean + d2 * om.inv_hx * c[6]) / T(3);
                sUP[SI(kk, ll)] = (up + uh + c[0] + qs * vh) / T(3);
                sVP[SI(kk, ll)] = (vp + vh + c[1] + c[5] * c[0]) / T(3);
                db[s * L::HL + al - a0] = sdiv;
                db[s2 * L::HL + kk - i0] = sdiv;
            }
        }
        __threadfence_block();
        nbar_arrive(BAR_BND, NM + nband);
        return;
    }

    // =================== the main threads ===================
    const int tx = tid % XL, ty = tid / XL;
    const int k = i0 - 4 + VW * tx;                       // first point of this thread's vector
    const bool lane_ok = ty < L::YG;
    const bool in_tile = lane_ok && tx >= HV && tx < HV + (v1 - v0);
    // edge vectors of the x stencils (closures at outputs 1..4 and n-3..n)
    int ve = -1, ec = 0, ei = 0;                          // index, first input of the c2i / i2c rows (from k)
    {
        const int v = v0 - HV + tx, vr = (n - 4) / VW;
        if (v >= 0 && v < HV) { ve = v; ec = ei = 1 - k; }
        else if (v >= vr && v < NV) { ve = HV + (v - vr); ec = N - 7 - k; ei = n - 7 - k; }
    }
    if (touch) {
        for (int q = tid; q < XROW_LEN; q += NM) xr[q] = __ldg(om.xr + q);
        for (int q = tid; q < XROW_OPS * ONE_EDGES * ONE_TAPS && (touch & 3u); q += NM)
            ov_st(we + q * VW, *reinterpret_cast<const V *>(om.we + q * VW));
    }
    const T H = T(__ldg(a.Hm + mem)), dt = T(a.dtm ? __ldg(a.dtm + mem) : a.dt);
    // the first warp waits for the tile loads (its first thread initialised the barrier), the others
    // at the named barrier, where they take no issue slots
    __syncwarp();
    if (tid < 32 && !mbar_wait(bar, 0, FUSED_WAIT_NS)) {
        // the tile loads did not arrive: record it, wait once more (bounded), and finish on
        // whatever the windows hold
        *(volatile int *)err = 1;
        mbar_wait(bar, 0, FUSED_WAIT_NS);
    }
    nbar_sync(BAR_MAIN, NM);
    pdl_wait();                                           // (the loads waited already)

    // ---- P1: vq = JQ12 I_c2i,y(v) on rows [j0-1, j1+2), uq = JQ12 I_c2i,x(u) on rows [j0-3, j1+3)
    {
        const int l = max(j0 - 1, 1) + ty;
        if (lane_ok && l < min(j1 + 2, n + 1)) {
            const int o = SI(k, l);
            ov_st(sVQ + o, ov_mul(ov_ld(sJQ12 + o), one_y<0, false, SW>(sV + SI(k, 0), (const T *)nullptr, l, n, xr)));
        }
        const int m = max(j0 - 3, 1) + ty;
        if (lane_ok && m < min(j1 + 3, n + 1)) {
            const int o = SI(k, m);
            ov_st(sUQ + o, ov_mul(ov_ld(sJQ12 + o), one_x<0>(sU + o, ve, ec, we)));
        }
    }
    nbar_sync(BAR_MAIN, NM);

    // ---- P2: J ut = JQ11 u + I_i2c,x(vq) on u points, rows [j0-1, j1+2); ut = J ut / J
    //          J vt = JQ22 v + I_i2c,y(uq) on v points, rows [j0-2, j1+1)
    {
        const V s2 = ov_all(T(1.0 / (ONE_IS * ONE_IS)));
        const int l = max(j0 - 1, 1) + ty;
        if (lane_ok && l < min(j1 + 2, n + 1)) {
            const int o = SI(k, l);
            const V I = one_x<2>(sVQ + o, ve, ei, we);
            const V r = ov_fma(I, s2, ov_mul(ov_ld(sJQ11 + o), ov_ld(sU + o)));
            ov_st(sJUT + o, r);
            ov_st(sUT + o, ov_mul(r, ov_ld(siJy + o)));
        }
        const int m = max(j0 - 2, 1) + ty;
        if (lane_ok && m < min(j1 + 1, N + 1)) {
            const int o = SI(k, m);
            const V I = one_y<2, false, SW>(sUQ + SI(k, 0), (const T *)nullptr, m, N, xr);
            ov_st(sJVT + o, ov_fma(I, s2, ov_mul(ov_ld(sJQ22 + o), ov_ld(sV + o))));
        }
    }
    nbar_sync(BAR_MAIN, NM);
    if (touch) {
        __threadfence_block();
        nbar_arrive(BAR_P2, NM + nband);
    }

    // ---- P3: the Coriolis vertex vectors away from the panel boundary
    {
        // a point of this vector lies on the panel boundary (columns 1 and n)
        const bool bcol = k <= 1 ? k + VW > 1 : (k <= n && k + VW > n);
        auto put = [&](T *out, const V &r) {
            if (!bcol) ov_st(out, r);
            else
#pragma unroll
                for (int e = 0; e < VW; e++)
                    if (k + e != 1 && k + e != n) out[e] = r.a[e];
        };
        const int l = j0 + ty;
        if (lane_ok && l < j1 && l != 1 && l != n) {
            const int o = SI(k, l);
            put(sUP + o, ov_mul(ov_ld(sF + o), one_y<0, true, SW>(sJVT + SI(k, 0), siJx + SI(k, 0), l, n, xr)));
        }
        const int m = max(j0 - 1, 1) + ty;
        if (in_tile && m < min(j1 + 2, n + 1) && m != 1 && m != n) {
            const int o = SI(k, m);
            const V I = one_x<0>(sUT + o, ve, ec, we), f = ov_ld(sF + o);
            V r;
#pragma unroll
            for (int e = 0; e < VW; e++) r.a[e] = -f.a[e] * I.a[e];
            put(sVP + o, r);
        }
    }
    // ---- RK4 operands of this thread's points, in flight across the barrier; in mode 1 V0 is the
    // stage input, in the windows
    const int mode = a.mode;
    const int j = j0 + ty;
    const bool work = in_tile && j < j1;
    const int so = SI(k, j);
    const int64_t po = (int64_t)mem * d.ms + (int64_t)t * d.ps + box_off32(P, k, j);
    const int64_t fs = d.fs;
    V pv[3]{}, pa[3]{}, kh, ku, kv;
    if (work) {
        if (mode >= 2) {
#pragma unroll
            for (int f = 0; f < 3; f++) {
                pv[f] = ov_ld(V0 + po + f * fs);
                pa[f] = ov_ld(ACC + po + f * fs);
            }
        }
        // the parts that need no boundary value: divergence and gradient (without the SAT's
        // neighbour terms)
        kh = ov_mul(ov_mul(ov_add(one_x<1>(sJUT + so, ve, ec, we),
                                  one_y<1, false, SW>(sJVT + SI(k, 0), (const T *)nullptr, j, n, xr)),
                           ov_all(om.cd)),
                    ov_ld(siJa + so));
        ku = one_x<3>(sH + so, ve, ei, we);
        kv = ov_zero<T, VW>();
        if (j <= N) kv = one_y<3, false, SW>(sH + SI(k, 0), (const T *)nullptr, j, N, xr);
    }
    if (touch) nbar_sync(BAR_BND, NM + nband);
    else nbar_sync(BAR_MAIN, NM);
    if (!work) return;

    // ---- P4: the tendencies of the tile's points and the RK4 update
    if (touch) {
        // the synchronised divergence of the boundary vertices; the gradient SAT across the edges
        const bool edgecol = k <= 1 || k + VW > n;
        if (j == 1 || j == n) {
#pragma unroll
            for (int e = 0; e < VW; e++) kh.a[e] = db[(j == 1 ? SIDE_B : SIDE_T) * L::HL + k + e - i0];
        }
        if (edgecol) {
#pragma unroll
            for (int e = 0; e < VW; e++) {
                if (k + e == 1) kh.a[e] = db[SIDE_L * L::HL + j - j0];
                if (k + e == n) kh.a[e] = db[SIDE_R * L::HL + j - j0];
            }
        }
        if (ve >= 0) {
            const T hx = hh[(ve < HV ? SIDE_L : SIDE_R) * L::HL + j - j0];
            ku = ov_fma(ov_ld(we + ((3 * ONE_EDGES + ve) * ONE_TAPS + 8) * VW), ov_all(hx), ku);
        }
        if (j <= SB::NSAT || (j >= N + 1 - SB::NSAT && j <= N)) {
            const bool lo = j <= SB::NSAT;
            const V hb = ov_ld(sH + SI(k, lo ? 1 : n));
            const T *const ho = hh + (lo ? SIDE_B : SIDE_T) * L::HL + k - i0;
            const T w = T(ONE_DS * (lo ? SB::satw(j) : -SB::satw(N + 1 - j)));
#pragma unroll
            for (int e = 0; e < VW; e++) kv.a[e] += w * (hb.a[e] - ho[e]);
        }
    }
    {
        const V s2 = ov_all(T(1.0 / (ONE_IS * ONE_IS))), cg = ov_all(om.cg);
        kh = ov_mul(kh, ov_all(-H));
        ku = ov_fma(ov_mul(one_x<2>(sUP + so, ve, ei, we), ov_ld(siJy + so)), s2, ov_mul(ku, cg));
        if (j <= N)
            kv = ov_fma(ov_mul(one_y<2, false, SW>(sVP + SI(k, 0), (const T *)nullptr, j, N, xr), ov_ld(siJx + so)), s2,
                        ov_mul(kv, cg));
        if (k + VW > n)
#pragma unroll
            for (int e = 0; e < VW; e++) {
                if (k + e > N) ku.a[e] = T(0);
                if (k + e > n) kh.a[e] = kv.a[e] = T(0);
            }
    }
    // elements beyond the fields' extent hold zeros and stay zero
    if (mode == 0) {
        ov_st(Y1 + po, kh);
        ov_st(Y1 + po + fs, ku);
        ov_st(Y1 + po + 2 * fs, kv);
    } else if (mode <= 3) {
        const T ca = (mode == 3) ? dt : T(0.5) * dt, cb = (mode == 1) ? dt / T(6) : dt / T(3);
        if (mode == 1) {
            pv[0] = ov_ld(sH + so);
            pv[1] = ov_ld(sU + so);
            pv[2] = ov_ld(sV + so);
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const V &kk = f == 0 ? kh : (f == 1 ? ku : kv);
            pv[f] = ov_fma(ov_all(ca), kk, pv[f]);
            pa[f] = ov_fma(ov_all(cb), kk, pa[f]);   // (zero before, in mode 1)
            ov_st(Y1 + po + f * fs, pv[f]);
            ov_st(ACC + po + f * fs, pa[f]);
        }
    } else {
        const T cb = dt / T(6);
        V cm[3];
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int f = 0; f < 3; f++) cm[f] = ov_ld(CMP + po + f * fs);
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const V &kk = f == 0 ? kh : (f == 1 ? ku : kv);
#pragma unroll
            for (int e = 0; e < VW; e++) {
                const T inc = pa[f].a[e] + cb * kk.a[e];
                if constexpr (sizeof(T) == 4) kahan_add(pv[f].a[e], cm[f].a[e], inc);
                else pv[f].a[e] = pv[f].a[e] + inc;
            }
            ov_st(V0 + po + f * fs, pv[f]);
            if constexpr (sizeof(T) == 4) ov_st(CMP + po + f * fs, cm[f]);
        }
    }
}

// The side lines of OneMetric from the fused metric boxes: [side][line][along].
template <class T>
__global__ void k_one_tables(const T *__restrict__ base, T *__restrict__ side, Dims d)
{
    const int N = d.N, n = N + 1, P = d.P, s = blockIdx.y;
    const int y = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (y > n) return;
    const bool lr = s <= SIDE_R, far = (s == SIDE_R || s == SIDE_T);
    const int64_t box = d.ps;
    T *o = side + s * ONE_LINES * n + y - 1;
    auto node = [&](int x) { const int xx = far ? n + 1 - x : x; return lr ? box_off32(P, xx, y) : box_off32(P, y, xx); };
    auto cen = [&](int x) { const int xx = far ? n - x : x; return lr ? box_off32(P, xx, y) : box_off32(P, y, xx); };
    for (int x = 1; x <= 5; x++) o[(OS_JQ12 + x - 1) * n] = base[FM_JQ12 * box + node(x)];
    for (int x = 1; x <= 3; x++) {
        o[(OS_JQN + x - 1) * n] = base[(lr ? FM_JQ11Y : FM_JQ22X) * box + cen(x)];
        o[(OS_IJN + x - 1) * n] = base[(lr ? FM_IJY : FM_IJX) * box + cen(x)];
    }
    o[OS_JQT * n] = y <= N ? base[(lr ? FM_JQ22X : FM_JQ11Y) * box + node(1)] : T(0);
    o[OS_IJT * n] = y <= N ? base[(lr ? FM_IJX : FM_IJY) * box + node(1)] : T(0);
}


}  // namespace chswe
