// swe_advone.cuh -- the advective operator's stage (covariant Ch branch, SBP 4-2) on 16-byte
// vectors of points, the form of swe_onepass.cuh:
//   k_adv_co2   contravariant components ut, vt (co2contra_Ch_mod.f90:27-94)
//   k_adv_flux  J times the up4 mass flux on the u and v points (massflux_ch_mod.f90:80-121)
//   k_adv_tend  up4 advection and Christoffel terms (vector_advection_Ch_mod.f90:33-115)
//   k_adv_stage divergence of the flux with its SAT and scalar edge sync, gradient of the
//               total depth, Coriolis with the vector edge sync, the advective tendencies and
//               the RK4 update (operator_adv_swm_mod.f90:62-96, rk4_mod.f90:28-40)
// A tile of k_adv_stage that touches a panel edge reads the neighbour panel's contravariant
// components and flux beside the edge itself, so the stage needs no edge strips and no
// edge-sync launch; k_advhalo (swe_advective.cuh) is shared with the split stage.
//
// Measured at C384 FP32 per launch (B200, cold L2, ncu): k_co2contra 22.8 -> k_adv_co2 9.8 us,
// k_stage 55.2 -> k_adv_stage 24.8 us, k_advt 27.8 -> k_adv_tend 15.2 us, k_edge 6.0 us and its
// strips gone; an RK4 step alone 444 us autotuned -> 252 (33, 2) or 220 (25, 2), with three
// contexts beside one another 367 -> 176.  The kernels wait for memory latency between
// short passes (the stage's windows and metric are nine TMA boxes per tile; the flux reads
// seven vectors per thread): more bytes in flight, not fewer operations, would shorten them.
#pragma once

#include "swe_advective.cuh"
#include "swe_adv_launch.cuh"
#include "swe_onepass.cuh"

namespace chswe {

// ---------------------------------------------------------------------------
// k_adv_co2: ut = Qi11 u + J^-1 I_i2c,x(J Qi12 I_c2i,y(v)), vt = Qi22 v + J^-1 I_i2c,y(J Qi12 I_c2i,x(u))
// ---------------------------------------------------------------------------
template <class T, int XL, int TH>
struct CoLayout {
    using L = OneLayout<T, XL, TH>;
    static constexpr int YG = TH + 3, NM = (XL * YG + 31) / 32 * 32;
    static constexpr int XR = 4 * L::SLOT, WE = XR + (XROW_LEN + L::VW - 1) / L::VW * L::VW,
                         BAR = WE + XROW_OPS * ONE_EDGES * ONE_TAPS * L::VW, TOTAL = BAR + L::VW;
    static size_t bytes() { return (size_t)TOTAL * sizeof(T); }
};

template <class T, int XL, int TH>
__global__ void __launch_bounds__(CoLayout<T, XL, TH>::NM)
    k_adv_co2(const __grid_constant__ CUtensorMap tmY, T *__restrict__ W, Dims d, OneMetric<T> om, const T *__restrict__ fmet,
              OneTiles ot, const double *__restrict__ dtm, int *err)
{
    using C = CoLayout<T, XL, TH>;
    using L = OneLayout<T, XL, TH>;
    using V = OV<T>;
    constexpr int VW = L::VW, HV = L::HV, SW = L::SW, NM = C::NM;
    extern __shared__ __align__(128) unsigned char osm_raw[];
    T *const sm = reinterpret_cast<T *>(osm_raw);
    T *const sU = sm, *const sV = sm + L::SLOT, *const sVQ = sm + 2 * L::SLOT, *const sUQ = sm + 3 * L::SLOT;
    T *const xr = sm + C::XR, *const we = sm + C::WE;
    uint64_t *const bar = reinterpret_cast<uint64_t *>(sm + C::BAR);
    const int N = d.N, n = N + 1, P = d.P, NV = (n + VW - 1) / VW, bx = blockIdx.x, by = blockIdx.y;
    const int t = blockIdx.z % NPAN, mem = blockIdx.z / NPAN;
    if (member_frozen(dtm, mem)) return;
    const int v0 = bx * ot.qx + min(bx, ot.rx), v1 = v0 + ot.qx + (bx < ot.rx);
    const int i0 = 1 + VW * v0, i1 = min(1 + VW * v1, n + 1);
    const int j0 = 1 + by * ot.qy + min(by, ot.ry), j1 = j0 + ot.qy + (by < ot.ry);
    const int tid = threadIdx.x, rows = N + 1 + 2 * MG;
    auto SI = [&](int i, int j) { return (j - j0 + 4) * SW + (i - i0 + 4); };
    const unsigned touch = (i0 == 1 ? 1u : 0u) | (i1 == n + 1 ? 2u : 0u) | (j0 == 1 ? 4u : 0u) | (j1 == n + 1 ? 8u : 0u);
    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(bar, (uint32_t)(2 * L::BOX_BYTES));
        pdl_wait();
        const int yr = (mem * 3 * NPAN + t) * rows + (j0 - 1), fr = NPAN * rows;
        tma_load_2d(sU, &tmY, bar, i0 - 1, yr + fr);
        tma_load_2d(sV, &tmY, bar, i0 - 1, yr + 2 * fr);
    }
    const int tx = tid % XL, ty = tid / XL, k = i0 - 4 + VW * tx;
    const bool lane_ok = ty < C::YG, in_tile = lane_ok && tx >= HV && tx < HV + (v1 - v0);
    int ve = -1, ec = 0, ei = 0;
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
    // the metric of this thread's points, in flight beside the loads.  Vectors of the halo beyond
    // the panel box hold no metric (their columns may leave the row) and are not read.
    const int64_t box = d.ps;
    const int l1 = j0 + ty, l2 = max(j0 - 1, 1) + ty, j = j0 + ty;
    const bool halo_ok = lane_ok && k >= 1 - VW * HV && k <= n;
    const bool w1 = halo_ok && l1 < j1, w2 = in_tile && l2 < min(j1 + 2, n + 1), w3 = in_tile && j < j1;
    V m1 = ov_all(T(0)), m2 = m1, a11 = m1, ay = m1, a22 = m1, ax = m1;
    if (w1) m1 = ov_ld(fmet + FM_JQ12 * box + box_off32(P, k, l1));
    if (w2) m2 = ov_ld(fmet + FM_JQ12 * box + box_off32(P, k, l2));
    if (w3) {
        const int o = box_off32(P, k, j);
        a11 = ov_ld(fmet + FM_JQ11Y * box + o);
        ay = ov_ld(fmet + FM_IJY * box + o);
        a22 = ov_ld(fmet + FM_JQ22X * box + o);
        ax = ov_ld(fmet + FM_IJX * box + o);
    }
    __syncwarp();
    if (tid < 32 && !mbar_wait(bar, 0, FUSED_WAIT_NS)) {
        *(volatile int *)err = 1;
        mbar_wait(bar, 0, FUSED_WAIT_NS);
    }
    __syncthreads();
    // vq = JQ12 I_c2i,y(v) on the tile's rows, the columns the i2c rows read; uq = JQ12 I_c2i,x(u)
    // on the tile's columns and rows [j0-1, j1+2)
    if (w1) ov_st(sVQ + SI(k, l1), ov_mul(m1, one_y<0, false, SW>(sV + SI(k, 0), (const T *)nullptr, l1, n, xr)));
    if (w2) ov_st(sUQ + SI(k, l2), ov_mul(m2, one_x<0>(sU + SI(k, l2), ve, ec, we)));
    __syncthreads();
    if (!w3) return;
    const V s2 = ov_all(T(1.0 / (ONE_IS * ONE_IS)));
    const int so = SI(k, j);
    const int64_t po = (int64_t)mem * d.ms + (int64_t)t * d.ps + box_off32(P, k, j);
    V ut = ov_mul(ov_fma(one_x<2>(sVQ + so, ve, ei, we), s2, ov_mul(a11, ov_ld(sU + so))), ay);
    if (k + VW > n)
#pragma unroll
        for (int e = 0; e < VW; e++)
            if (k + e > N) ut.a[e] = T(0);
    ov_st(W + po + d.fs, ut);
    if (j <= N) {
        V vt = ov_mul(ov_fma(one_y<2, false, SW>(sUQ + SI(k, 0), (const T *)nullptr, j, N, xr), s2, ov_mul(a22, ov_ld(sV + so))), ax);
        if (k + VW > n)
#pragma unroll
            for (int e = 0; e < VW; e++)
                if (k + e > n) vt.a[e] = T(0);
        ov_st(W + po + 2 * d.fs, vt);
    }
}

// ---------------------------------------------------------------------------
// k_adv_flux: J F on the u (field 1) and v points (field 2), one vector of points per thread
// ---------------------------------------------------------------------------
// Blocks with blockIdx.y < ny take 8 rows of 32 vectors and every flux whose six points lie in
// the panel.  The vectors beside columns 1 and n (u points) and the rows beside rows 1 and n
// (v points) read virtual points interpolated along the neighbour's grid lines, a chain of
// dependent loads: they are items of the further blocks, so that no other warp waits for them.
__host__ __device__ __forceinline__ int flux_first_edge(int n, int VW)
{
    // the first vector whose six-point windows reach beyond column n
    return n - VW - 3 < 0 ? 1 : ((n - VW - 3) / VW + 1 > 1 ? (n - VW - 3) / VW + 1 : 1);
}
__host__ __device__ __forceinline__ int flux_edge_items(int N, int VW)
{
    const int n = N + 1;
    return n * (VW + n - VW * flux_first_edge(n, VW)) + 4 * n;
}

template <class T>
__global__ void __launch_bounds__(256) k_adv_flux(const T *__restrict__ Y, const T *__restrict__ W, T *__restrict__ F, Dims d,
                                                  AdvView<T> av, MetricView<T> m, int ny, const double *__restrict__ dtm)
{
    using V = OV<T>;
    constexpr int VW = V::W;
    const int N = d.N, n = N + 1, P = d.P, NV = (n + VW - 1) / VW, vre = flux_first_edge(n, VW);
    const int mem = blockIdx.z / NPAN, t = blockIdx.z % NPAN;
    if (member_frozen(dtm, mem)) return;
    const int64_t po = mem * d.ms + t * d.ps;
    const T *const h = Y + mem * d.ms;
    pdl_trigger();
    if ((int)blockIdx.y < ny) {
        const int v = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y + 1, k = 1 + VW * v;
        const int64_t o = box_off(P, k, j);
        const bool ok = v < NV && j <= n, fx = ok && v >= 1 && v < vre, fy = ok && j >= 3 && j <= N - 2;
        V jy = ov_all(T(0)), jx = jy;
        if (fx) jy = ov_ld(m.Jy + o);
        if (fy) jx = ov_ld(m.Jx + o);
        pdl_wait();
        const T *const hr = h + t * d.ps + o;
        if (fx) {
            const V a = ov_ld(hr - 4 + (VW == 2 ? 2 : 0)), c = ov_ld(W + po + d.fs + o);
            T w[VW + 5];   // h(k-2 .. k+VW+2)
            w[0] = a.a[VW - 2];
            w[1] = a.a[VW - 1];
#pragma unroll
            for (int q = 0; q < VW + 3; q++) w[q + 2] = __ldg(hr + q);
            V f;
#pragma unroll
            for (int e = 0; e < VW; e++) f.a[e] = up4_flux(c.a[e], w[e], w[e + 1], w[e + 2], w[e + 3], w[e + 4], w[e + 5]);
            ov_st(F + po + d.fs + o, ov_mul(f, jy));
        }
        if (fy) {
            V g[6], f;
#pragma unroll
            for (int q = 0; q < 6; q++) g[q] = ov_ld(hr + (q - 2) * P);
            const V c = ov_ld(W + po + 2 * d.fs + o);
#pragma unroll
            for (int e = 0; e < VW; e++)
                f.a[e] = up4_flux(c.a[e], g[0].a[e], g[1].a[e], g[2].a[e], g[3].a[e], g[4].a[e], g[5].a[e]);
            ov_st(F + po + 2 * d.fs + o, ov_mul(f, jx));   // (zeros beyond column n, where W holds zeros)
        }
        return;
    }
    pdl_wait();
    // one edge point per thread
    const int q0 = ((blockIdx.y - ny) * gridDim.x + blockIdx.x) * 256 + threadIdx.y * 32 + threadIdx.x;
    const int wx = VW + n - VW * vre, nx = n * wx;   // u points of a row: 1..VW and VW vre + 1 .. n
    int i, j, f;
    if (q0 < nx) {
        f = 1;
        j = 1 + q0 / wx;
        i = 1 + q0 - (j - 1) * wx;
        if (i > VW) i += VW * (vre - 1);
        if (i > N) return;
    } else if (q0 < nx + 4 * n) {
        f = 2;
        const int r = (q0 - nx) / n;
        i = 1 + q0 - nx - r * n;
        j = r < 2 ? 1 + r : N - 3 + r;               // v points of the rows 1, 2, N-1, N
    } else return;
    const int64_t o = box_off(P, i, j);
    const T c = __ldg(W + po + f * d.fs + o), J = __ldg((f == 1 ? m.Jy : m.Jx) + o);
    T w[6];
#pragma unroll
    for (int q = 0; q < 6; q++) w[q] = h_ext(h, d, av, t, f == 1 ? i - 2 + q : i, f == 1 ? j : j - 2 + q);
    F[po + f * d.fs + o] = up4_flux(c, w[0], w[1], w[2], w[3], w[4], w[5]) * J;
}

// ---------------------------------------------------------------------------
// k_adv_tend: A_u, A_v = up4 advection + Christoffel terms before the edge sync (k_advt's values)
// ---------------------------------------------------------------------------
template <class T, int XL, int TH>
struct TendLayout {
    using L = OneLayout<T, XL, TH>;
    static constexpr int YG = TH + 3, NM = (XL * YG + 31) / 32 * 32;
    static constexpr int XR = 6 * L::SLOT, WE = XR + (XROW_LEN + L::VW - 1) / L::VW * L::VW,
                         BAR = WE + XROW_OPS * ONE_EDGES * ONE_TAPS * L::VW, TOTAL = BAR + L::VW;
    static size_t bytes() { return (size_t)TOTAL * sizeof(T); }
};

// 12 |c| times the upwind derivative of f along c at the middle of f[0..6] (up4_diff: the sign
// of c picks the stencil or its mirror, c times the sign is |c|)
template <class T>
__device__ __forceinline__ T up4_adv(T c, T f0, T f1, T f2, T f3, T f4, T f5, T f6)
{
    const bool p = c >= T(0);
    const T a = p ? f4 : f2, b = p ? f2 : f4, e = p ? f1 : f5, g = p ? f0 : f6;
    return fabs(c) * (T(3) * a + T(10) * f3 - T(18) * b + T(6) * e - g);
}

template <class T, int XL, int TH>
__global__ void __launch_bounds__(TendLayout<T, XL, TH>::NM, 2)
    k_adv_tend(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmW, const T *__restrict__ VH,
               T *__restrict__ A, Dims d, AdvView<T> av, OneMetric<T> om, T inv_hxa, OneTiles ot, const double *__restrict__ dtm,
               int *err)
{
    static_assert(sizeof(T) == 4, "FP64 tendencies: k_advt (AdvOneTU::tend)");
    using C = TendLayout<T, XL, TH>;
    using L = OneLayout<T, XL, TH>;
    using V = OV<T>;
    constexpr int VW = L::VW, HV = L::HV, SW = L::SW, NM = C::NM;
    extern __shared__ __align__(128) unsigned char osm_raw[];
    T *const sm = reinterpret_cast<T *>(osm_raw);
    T *const sU = sm, *const sV = sm + L::SLOT, *const sUT = sm + 2 * L::SLOT, *const sVT = sm + 3 * L::SLOT,
             *const sVH = sm + 4 * L::SLOT, *const sUH = sm + 5 * L::SLOT;
    T *const xr = sm + C::XR, *const we = sm + C::WE;
    uint64_t *const bar = reinterpret_cast<uint64_t *>(sm + C::BAR);
    const int N = d.N, n = N + 1, P = d.P, NV = (n + VW - 1) / VW, bx = blockIdx.x, by = blockIdx.y;
    const int t = blockIdx.z % NPAN, mem = blockIdx.z / NPAN;
    if (member_frozen(dtm, mem)) return;
    const int v0 = bx * ot.qx + min(bx, ot.rx), v1 = v0 + ot.qx + (bx < ot.rx);
    const int i0 = 1 + VW * v0, i1 = min(1 + VW * v1, n + 1);
    const int j0 = 1 + by * ot.qy + min(by, ot.ry), j1 = j0 + ot.qy + (by < ot.ry);
    const int tid = threadIdx.x, rows = N + 1 + 2 * MG;
    auto SI = [&](int i, int j) { return (j - j0 + 4) * SW + (i - i0 + 4); };
    const unsigned touch = (i0 == 1 ? 1u : 0u) | (i1 == n + 1 ? 2u : 0u) | (j0 == 1 ? 4u : 0u) | (j1 == n + 1 ? 8u : 0u);
    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(bar, (uint32_t)(4 * L::BOX_BYTES));
        pdl_wait();
        const int yr = (mem * 3 * NPAN + t) * rows + (j0 - 1), fr = NPAN * rows;
        tma_load_2d(sUT, &tmW, bar, i0 - 1, yr + fr);
        tma_load_2d(sVT, &tmW, bar, i0 - 1, yr + 2 * fr);
        tma_load_2d(sU, &tmY, bar, i0 - 1, yr + fr);
        tma_load_2d(sV, &tmY, bar, i0 - 1, yr + 2 * fr);
    }
    const int tx = tid % XL, ty = tid / XL, k = i0 - 4 + VW * tx, j = j0 + ty;
    const bool lane_ok = ty < C::YG, in_tile = lane_ok && tx >= HV && tx < HV + (v1 - v0), work = in_tile && j < j1;
    int ve = -1, ec = 0, ei = 0;
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
    V g11 = ov_all(T(0)), g21 = g11, g22 = g11;
    const int o = box_off32(P, k, j);
    if (work) {
        g11 = ov_ld(av.S + o);
        g21 = ov_ld(av.S + d.ps + o);
        g22 = ov_ld(av.S + 2 * d.ps + o);
    }
    __syncwarp();
    if (tid < 32 && !mbar_wait(bar, 0, FUSED_WAIT_NS)) {
        *(volatile int *)err = 1;
        mbar_wait(bar, 0, FUSED_WAIT_NS);
    }
    __syncthreads();
    // ---- vh = I_c2i,y(vt) on the tile's rows and the columns the i2c rows read; uh = I_c2i,x(ut)
    // on the tile's columns and rows [j0-1, j1+2); the winds beyond the panel from the halo points
    if (lane_ok && j < j1) ov_st(sVH + SI(k, j), one_y<0, false, SW>(sVT + SI(k, 0), (const T *)nullptr, j, n, xr));
    {
        const int m = max(j0 - 1, 1) + ty;
        if (in_tile && m < min(j1 + 2, n + 1)) ov_st(sUH + SI(k, m), one_x<0>(sUT + SI(k, m), ve, ec, we));
    }
    if (touch) {
        pdl_wait();
        const T *const vh = VH + ((int64_t)mem * NPAN + t) * av.hp;
        const int tw = i1 - i0, th = j1 - j0;
        if (touch & 3u)
            for (int q = tid; q < 3 * th; q += NM) {
                const int c = q / th, l = j0 + q - c * th;   // c + 1 points beyond the panel
                if (touch & 1u) {
                    sU[SI(-c, l)] = vh[vh_u_w(N) + c * (N + 1) + (l - 1)];
                    if (l <= N) sV[SI(-c, l)] = vh[vh_v_w(N) + c * N + (l - 1)];
                }
                if (touch & 2u) {
                    sU[SI(N + 1 + c, l)] = vh[vh_u_e(N) + c * (N + 1) + (l - 1)];
                    if (l <= N) sV[SI(N + 2 + c, l)] = vh[vh_v_e(N) + c * N + (l - 1)];
                }
            }
        if (touch & 12u)
            for (int q = tid; q < 3 * tw; q += NM) {
                const int c = q / tw, i = i0 + q - c * tw;
                if (touch & 4u) {
                    if (i <= N) sU[SI(i, -c)] = vh[vh_u_s(N) + c * N + (i - 1)];
                    sV[SI(i, -c)] = vh[vh_v_s(N) + c * (N + 1) + (i - 1)];
                }
                if (touch & 8u) {
                    if (i <= N) sU[SI(i, N + 2 + c)] = vh[vh_u_n(N) + c * N + (i - 1)];
                    sV[SI(i, N + 1 + c)] = vh[vh_v_n(N) + c * (N + 1) + (i - 1)];
                }
            }
    }
    __syncthreads();
    if (!work) return;
    const int64_t po = (int64_t)mem * d.ms + (int64_t)t * d.ps + o;
    const int so = SI(k, j);
    const T s2 = T(1.0 / ONE_IS), ca = -inv_hxa * T(1.0 / 12.0), cr = -av.inv_neg_radius;
    // the tendency of one wind component f with the advecting (a, b) there
    auto tend = [&](const T *f, const V &a, const V &b) {
        T x[VW + 6];
        {
            const V l = ov_ld(f - 4), h = ov_ld(f + 4);
            const V c = ov_ld(f);
#pragma unroll
            for (int e = 0; e < 3; e++) { x[e] = l.a[e + 1]; x[VW + 3 + e] = h.a[e]; }
#pragma unroll
            for (int e = 0; e < VW; e++) x[3 + e] = c.a[e];
        }
        V y[7], r;
#pragma unroll
        for (int q = 0; q < 7; q++) y[q] = ov_ld(f + (q - 3) * SW);
#pragma unroll
        for (int e = 0; e < VW; e++) {
            const T ae = a.a[e], be = b.a[e];
            const T s = up4_adv(ae, x[e], x[e + 1], x[e + 2], x[e + 3], x[e + 4], x[e + 5], x[e + 6]) +
                        up4_adv(be, y[0].a[e], y[1].a[e], y[2].a[e], y[3].a[e], y[4].a[e], y[5].a[e], y[6].a[e]);
            r.a[e] = s * ca + (ae * ae * g11.a[e] + T(2) * ae * be * g21.a[e] + be * be * g22.a[e]) * cr;
        }
        return r;
    };
    {
        // u points: ut and v_at_u = I_i2c,x(vh)
        V b = one_x<2>(sVH + so, ve, ei, we);
#pragma unroll
        for (int e = 0; e < VW; e++) b.a[e] *= s2 * s2;
        V r = tend(sU + so, ov_ld(sUT + so), b);
        if (k + VW > n)
#pragma unroll
            for (int e = 0; e < VW; e++)
                if (k + e > N) r.a[e] = T(0);
        ov_st(A + po + d.fs, r);
    }
    if (j <= N) {
        // v points: u_at_v = I_i2c,y(uh) and vt
        const T *S = av.S + 3 * d.ps + o;
        g11 = ov_ld(S);
        g21 = ov_ld(S + d.ps);
        g22 = ov_ld(S + 2 * d.ps);
        V a = one_y<2, false, SW>(sUH + SI(k, 0), (const T *)nullptr, j, N, xr);
#pragma unroll
        for (int e = 0; e < VW; e++) a.a[e] *= s2 * s2;
        V r = tend(sV + so, a, ov_ld(sVT + so));
        if (k + VW > n)
#pragma unroll
            for (int e = 0; e < VW; e++)
                if (k + e > n) r.a[e] = T(0);
        ov_st(A + po + 2 * d.fs, r);
    }
}

// ---------------------------------------------------------------------------
// k_adv_stage
// ---------------------------------------------------------------------------
template <class T, int XL, int TH>
struct AdvLayout {
    using L = OneLayout<T, XL, TH>;
    static constexpr int YG = TH + 3, NM = (XL * YG + 31) / 32 * 32;
    static constexpr int NLOAD = 9, NSLOT = 11;
    static constexpr int LB = ONE_BAND + 8, BAND = 2 * LB;    // t and J F_t along one side
    static constexpr int HL = L::TP + 8;
    static constexpr int HALO = NSLOT * L::SLOT, DIVB = HALO + 4 * HL, BAR = DIVB + 4 * HL, XR = BAR + L::VW,
                         WE = XR + (XROW_LEN + L::VW - 1) / L::VW * L::VW, CORN = WE + XROW_OPS * ONE_EDGES * ONE_TAPS * L::VW,
                         BANDS = CORN + 64;
    static size_t bytes(int sides) { return (size_t)(BANDS + sides * BAND) * sizeof(T); }
};

// tmY: stage input (h); tmW: contravariant components; tmF: J F; tmM: fused metric; all with
// boxes of SW x SR.  a.A: advective tendencies, a.HB: boundary h before the averaging, a.HS:
// orography or null.
template <class T, int XL, int TH, int REGS>
__global__ void __maxnreg__(REGS)
    k_adv_stage(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmW,
                const __grid_constant__ CUtensorMap tmF, const __grid_constant__ CUtensorMap tmM, const T *__restrict__ Wc,
                T *V0, T *Y1, T *ACC, T *CMP, Dims d, OneMetric<T> om, OneTiles ot, StageArgs a, int *err)
{
    using L = OneLayout<T, XL, TH>;
    using G = AdvLayout<T, XL, TH>;
    using SB = SbpOrder<42>;
    using V = OV<T>;
    constexpr int VW = L::VW, HV = L::HV, SW = L::SW, NM = G::NM;
    extern __shared__ __align__(128) unsigned char osm_raw[];
    T *const sm = reinterpret_cast<T *>(osm_raw);
    T *const sH = sm, *const sUT = sm + L::SLOT, *const sVT = sm + 2 * L::SLOT, *const sFU = sm + 3 * L::SLOT,
             *const sFV = sm + 4 * L::SLOT, *const sF = sm + 5 * L::SLOT, *const siJy = sm + 6 * L::SLOT,
             *const siJx = sm + 7 * L::SLOT, *const siJa = sm + 8 * L::SLOT, *const sUP = sm + 9 * L::SLOT,
             *const sVP = sm + 10 * L::SLOT;
    T *const hh = sm + G::HALO, *const db = sm + G::DIVB, *const xr = sm + G::XR, *const we = sm + G::WE;
    uint64_t *const bar = reinterpret_cast<uint64_t *>(sm + G::BAR);

    const int N = d.N, n = N + 1, P = d.P;
    const int t = blockIdx.z % NPAN, mem = blockIdx.z / NPAN;
    if (member_frozen(a.dtm, mem)) return;
    const int NV = (n + VW - 1) / VW, bx = blockIdx.x, by = blockIdx.y;
    const int v0 = bx * ot.qx + min(bx, ot.rx), v1 = v0 + ot.qx + (bx < ot.rx);
    const int i0 = 1 + VW * v0, i1 = min(1 + VW * v1, n + 1);
    const int j0 = 1 + by * ot.qy + min(by, ot.ry), j1 = j0 + ot.qy + (by < ot.ry);
    const int tid = threadIdx.x, rows = N + 1 + 2 * MG;
    auto SI = [&](int i, int j) { return (j - j0 + 4) * SW + (i - i0 + 4); };
    const unsigned touch = (i0 == 1 ? 1u : 0u) | (i1 == n + 1 ? 2u : 0u) | (j0 == 1 ? 4u : 0u) | (j1 == n + 1 ? 8u : 0u);
    const int nband = __popc(touch) * ONE_BAND;
    const T *const HB = (const T *)a.HB, *const HS = (const T *)a.HS;

    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(bar, (uint32_t)(G::NLOAD * L::BOX_BYTES));
        const int mr = j0 - 1, ax = i0 - 1;
        tma_load_2d(sF, &tmM, bar, ax, (FM_FJ2 + t) * rows + mr);
        tma_load_2d(siJy, &tmM, bar, ax, FM_IJY * rows + mr);
        tma_load_2d(siJx, &tmM, bar, ax, FM_IJX * rows + mr);
        tma_load_2d(siJa, &tmM, bar, ax, FM_IJA * rows + mr);
        pdl_wait();
        const int yr = (mem * 3 * NPAN + t) * rows + (j0 - 1), fr = NPAN * rows;
        tma_load_2d(sUT, &tmW, bar, ax, yr + fr);
        tma_load_2d(sVT, &tmW, bar, ax, yr + 2 * fr);
        tma_load_2d(sFU, &tmF, bar, ax, yr + fr);
        tma_load_2d(sFV, &tmF, bar, ax, yr + 2 * fr);
        tma_load_2d(sH, &tmY, bar, ax, yr);
    }

    if (tid >= NM) {
        // =================== the band threads (swe_onepass.cuh) ===================
        const int bt = tid - NM, slot = bt / ONE_BAND, b = bt % ONE_BAND;
        if (bt >= nband) return;
        int s = 0;
        for (int q = 0, c = -1; q < 4; q++)
            if (touch >> q & 1) {
                c++;
                if (c == slot) s = q;
            }
        const Link K = c_link[t][s];
        const bool lr = s <= SIDE_R, nlr = K.nside <= SIDE_R, far = (K.nside == SIDE_R || K.nside == SIDE_T);
        const int a0 = lr ? j0 : i0, a1 = lr ? j1 : i1, al = a0 - 3 + b;
        T *const bd = sm + G::BANDS + slot * G::BAND;
        const bool node = al >= 1 && al <= n && al <= a1 + 2, cen = al >= 1 && al <= N && al <= a1 + 2;
        const int y = K.rev ? n + 1 - al : al, yc = K.rev ? N + 1 - al : al;
        const bool vx = node && al >= a0 - 1 && al <= a1 + 1, full = node && al >= a0 && al < a1;
        T wI[5], wD[5], fo = T(0), fn = T(0), eao = T(0), ean = T(0), qs = T(0);
        int bI = 1;
#pragma unroll
        for (int m = 0; m < 5; m++) wI[m] = wD[m] = T(0);
        if (node) {
            const T *const gx = xrow_table<T>();
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
        for (int q = b; q < G::BAND; q += ONE_BAND) bd[q] = T(0);
        nbar_sync(BAR_SIDE + slot, ONE_BAND);
        pdl_wait();
        // the neighbour's copies: the normal components of ut, vt and of J F at depths 1..3 (node al),
        // the tangential ones on the edge line (centre al), h before the averaging at the vertex
        const int64_t nb = (int64_t)mem * d.ms + (int64_t)K.nb * d.ps;
        const T *const pW = Wc + nb, *const pF = (const T *)a.F + nb;
        const int64_t fn_ = (nlr ? 1 : 2) * d.fs, ft_ = (nlr ? 2 : 1) * d.fs;
        OneRaw<T> rn{};
        T nf[3], jf[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const int xx = far ? n - (x + 1) : x + 1, o = nlr ? box_off32(P, xx, y) : box_off32(P, y, xx);
            nf[x] = vx ? ld_cg(pW + fn_ + o) : T(0);
            jf[x] = vx ? ld_cg(pF + fn_ + o) : T(0);
        }
        const int e1 = far ? n : 1;
        T tt = T(0), jt = T(0);
        if (cen) {
            const int o = nlr ? box_off32(P, e1, yc) : box_off32(P, yc, e1);
            tt = ld_cg(pW + ft_ + o);
            jt = ld_cg(pF + ft_ + o);
        }
        if (full) {
            T hv = ld_cg(HB + hb_index(N, mem, K.nb, K.nside, y));
            if (HS) hv += __ldg(HS + K.nb * d.ps + (nlr ? box_off32(P, e1, y) : box_off32(P, y, e1)));
            hh[s * G::HL + al - a0] = hv;
        }
        auto ln = [&](int line) { return bd + line * G::LB - a0 + 3; };
        ln(0)[al] = tt;
        ln(1)[al] = jt;
        rn.A = T(SB::ic1(1)) * nf[0] + T(SB::ic1(2)) * nf[1] + T(SB::ic1(3)) * nf[2];
        rn.B = T(SB::dc1(1)) * jf[0] + T(SB::dc1(2)) * jf[1] + T(SB::dc1(3)) * jf[2];
        rn.C = T(SB::r1(1)) * jf[0] + T(SB::r1(2)) * jf[1] + T(SB::r1(3)) * jf[2];
        nbar_sync(BAR_SIDE + slot, ONE_BAND);
        if (full) {
            const T *ft = ln(0) + bI, *fj = ln(1) + bI;
#pragma unroll
            for (int m = 0; m < 5; m++) {
                rn.T1 += wI[m] * ft[m];
                rn.T2 += wD[m] * fj[m];
            }
            if (K.rev) rn.T2 = -rn.T2;
            const T *fk = ln(1);
            if (al == 1) rn.K = T(SB::r1(1)) * fk[1] + T(SB::r1(2)) * fk[2] + T(SB::r1(3)) * fk[3];
            if (al == n) rn.K = T(SB::r1(1)) * fk[N] + T(SB::r1(2)) * fk[N - 1] + T(SB::r1(3)) * fk[N - 2];
        }
        T un, vn, uh = T(0), vh = T(0);
        one_vec(rn, K.nside, fn, un, vn);
        halo_vec(t, s, un, vn, uh, vh);
        // the own copy, from the tile's windows (the main threads' arrival: the barrier is initialised)
        nbar_sync(BAR_P2, NM + nband);
        if (!mbar_wait(bar, 0, FUSED_WAIT_NS)) {
            *(volatile int *)err = 1;
            mbar_wait(bar, 0, FUSED_WAIT_NS);
        }
        OneRaw<T> ro{};
        int kk, ll;
        side_vertex(N, s, al, 0, kk, ll);
        if (vx) {
            const int o = s == SIDE_L ? SI(0, al) : (s == SIDE_R ? SI(n, al) : (s == SIDE_B ? SI(al, 0) : SI(al, n)));
            const int sd = s == SIDE_L ? 1 : (s == SIDE_R ? -1 : (s == SIDE_B ? SW : -SW));
            const T *const pj = (lr ? sFU : sFV) + o, *const pi = (lr ? sUT : sVT) + o;
            const T j1_ = pj[sd], j2_ = pj[2 * sd], j3_ = pj[3 * sd];
            ro.A = T(SB::ic1(1)) * pi[sd] + T(SB::ic1(2)) * pi[2 * sd] + T(SB::ic1(3)) * pi[3 * sd];
            ro.B = T(SB::dc1(1)) * j1_ + T(SB::dc1(2)) * j2_ + T(SB::dc1(3)) * j3_;
            ro.C = T(SB::r1(1)) * j1_ + T(SB::r1(2)) * j2_ + T(SB::r1(3)) * j3_;
        }
        if (full) {
            const int sc = lr ? SW : 1, o = lr ? SI(kk, 0) : SI(0, ll);
            const T *const pt = (lr ? sFV : sFU) + o, *const pi = (lr ? sVT : sUT) + o;
#pragma unroll
            for (int m = 0; m < 5; m++) {
                const bool use = m < 4 || wI[4] != T(0) || wD[4] != T(0);
                ro.T1 += use ? wI[m] * pi[(bI + m) * sc] : T(0);
                ro.T2 += use ? wD[m] * pt[(bI + m) * sc] : T(0);
            }
            if (al == 1) ro.K = T(SB::r1(1)) * pt[sc] + T(SB::r1(2)) * pt[2 * sc] + T(SB::r1(3)) * pt[3 * sc];
            if (al == n) ro.K = T(SB::r1(1)) * pt[N * sc] + T(SB::r1(2)) * pt[(N - 1) * sc] + T(SB::r1(3)) * pt[(N - 2) * sc];
        }
        T up, vp;
        one_vec(ro, s, fo, up, vp);
        const T dn = one_across(rn, K.nside, T(K.sn) * ro.C) + rn.T2, dv = one_across(ro, s, T(K.sn) * rn.C) + ro.T2;
        if (vx && !full) {
            if (lr) sVP[SI(kk, ll)] = T(0.5) * (vp + vh);
            else sUP[SI(kk, ll)] = T(0.5) * (up + uh);
        } else if (full && !corner) {
            sUP[SI(kk, ll)] = lr ? T(0.5) * (up + uh + qs * vh) : T(0.5) * (up + uh);
            sVP[SI(kk, ll)] = lr ? T(0.5) * (vp + vh) : T(0.5) * (vp + vh + qs * uh);
            db[s * G::HL + al - a0] = T(0.5) * (dv * om.inv_hx * eao + dn * om.inv_hx * ean);
        }
        if ((touch & 3u) && (touch & 12u)) {
            const int end = al == 1 ? 0 : 1;
            if (full && corner && !lr) {
                T *c = sm + G::CORN + (s * 2 + end) * 8;
                c[0] = uh; c[1] = vh; c[2] = rn.C; c[3] = rn.K; c[4] = dn; c[5] = qs; c[6] = ean;
            }
            nbar_sync(BAR_CORN, nband);
            if (full && corner && lr) {
                const T *c = sm + G::CORN + (s2 * 2 + (kk == 1 ? 0 : 1)) * 8;
                const T satc = T(SB::SATC);
                const T jo = satc * (ro.K - sn2 * c[2]), jx = satc * (rn.K - sgx * c[3]), jy = satc * (c[3] - sgy * rn.K);
                const T d0 = al == 1 ? dv + jo : dv - jo, d1 = y1 ? dn + jx : dn - jx, d2 = y21 ? c[4] + jy : c[4] - jy;
                const T sdiv = (d0 * om.inv_hx * eao + d1 * om.inv_hx * ean + d2 * om.inv_hx * c[6]) / T(3);
                sUP[SI(kk, ll)] = (up + uh + c[0] + qs * vh) / T(3);
                sVP[SI(kk, ll)] = (vp + vh + c[1] + c[5] * c[0]) / T(3);
                db[s * G::HL + al - a0] = sdiv;
                db[s2 * G::HL + kk - i0] = sdiv;
            }
        }
        __threadfence_block();
        nbar_arrive(BAR_BND, NM + nband);
        return;
    }

    // =================== the main threads ===================
    if (touch) {
        __threadfence_block();
        nbar_arrive(BAR_P2, NM + nband);
    }
    const int tx = tid % XL, ty = tid / XL;
    const int k = i0 - 4 + VW * tx, j = j0 + ty;
    const bool lane_ok = ty < G::YG, in_tile = lane_ok && tx >= HV && tx < HV + (v1 - v0), work = in_tile && j < j1;
    int ve = -1, ec = 0, ei = 0;
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
    pdl_wait();
    // the RK4 operands and advective tendencies of this thread's points, in flight beside the loads
    const int mode = a.mode;
    const int64_t po = (int64_t)mem * d.ms + (int64_t)t * d.ps + box_off32(P, k, j);
    const int64_t fs = d.fs;
    const T *const Aa = (const T *)a.A;
    V pv[3]{}, pa[3]{}, au{}, aw{};
    if (work) {
        au = ov_ld(Aa + po + fs);
        aw = ov_ld(Aa + po + 2 * fs);
        if (touch) {
            // the duplicated edge points: the mean with the neighbour's tangential component
            if (j == 1 || j == n)
#pragma unroll
                for (int e = 0; e < VW; e++)
                    if (k + e <= N) au.a[e] = adv_edge_sync(Aa, d, mem, t, 1, k + e, j, au.a[e]);
#pragma unroll
            for (int e = 0; e < VW; e++)
                if ((k + e == 1 || k + e == n) && j <= N) aw.a[e] = adv_edge_sync(Aa, d, mem, t, 2, k + e, j, aw.a[e]);
        }
    }
    __syncwarp();
    if (tid < 32 && !mbar_wait(bar, 0, FUSED_WAIT_NS)) {
        *(volatile int *)err = 1;
        mbar_wait(bar, 0, FUSED_WAIT_NS);
    }
    nbar_sync(BAR_MAIN, NM);
    // ---- the gradient's input: h before the averaging on the panel boundary, plus the orography
    if (touch || HS) {
        for (int r = ty; r < (j1 - j0) + 8 && lane_ok; r += G::YG) {
            const int l = j0 - 4 + r;
            if (l < 1 || l > n || k > n || k + VW <= 1) continue;
            T *const p = sH + SI(k, l);
            V x = ov_ld(p);
            if (touch)
#pragma unroll
                for (int e = 0; e < VW; e++) {
                    const int i = k + e;
                    if (i < 1 || i > n || !(i == 1 || i == n || l == 1 || l == n)) continue;
                    x.a[e] = ld_cg(HB + (i == 1 || i == n ? hb_index(N, mem, t, i == 1 ? SIDE_L : SIDE_R, l)
                                                          : hb_index(N, mem, t, l == 1 ? SIDE_B : SIDE_T, i)));
                }
            if (HS) x = ov_add(x, ov_ld(HS + t * d.ps + box_off32(P, k, l)));
            ov_st(p, x);
        }
        nbar_sync(BAR_MAIN, NM);
    }
    // ---- P3: the Coriolis vertex vectors away from the panel boundary
    {
        const bool bcol = k <= 1 ? k + VW > 1 : (k <= n && k + VW > n);
        auto put = [&](T *out, const V &r) {
            if (!bcol) ov_st(out, r);
            else
#pragma unroll
                for (int e = 0; e < VW; e++)
                    if (k + e != 1 && k + e != n) out[e] = r.a[e];
        };
        if (lane_ok && j < j1 && j != 1 && j != n) {
            const int o = SI(k, j);
            put(sUP + o, ov_mul(ov_ld(sF + o), one_y<0, false, SW>(sVT + SI(k, 0), (const T *)nullptr, j, n, xr)));
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
    const int so = SI(k, j);
    V kh, ku, kv;
    if (work) {
        if (mode >= 1) {
#pragma unroll
            for (int f = 0; f < 3; f++) pv[f] = ov_ld(V0 + po + f * fs);
        }
        if (mode >= 2) {
#pragma unroll
            for (int f = 0; f < 3; f++) pa[f] = ov_ld(ACC + po + f * fs);
        }
        kh = ov_mul(ov_mul(ov_add(one_x<1>(sFU + so, ve, ec, we),
                                  one_y<1, false, SW>(sFV + SI(k, 0), (const T *)nullptr, j, n, xr)),
                           ov_all(om.cd)),
                    ov_ld(siJa + so));
        ku = one_x<3>(sH + so, ve, ei, we);
        kv = ov_all(T(0));
        if (j <= N) kv = one_y<3, false, SW>(sH + SI(k, 0), (const T *)nullptr, j, N, xr);
    }
    if (touch) nbar_sync(BAR_BND, NM + nband);
    else nbar_sync(BAR_MAIN, NM);
    if (!work) return;

    // ---- P4
    if (touch) {
        if (j == 1 || j == n) {
#pragma unroll
            for (int e = 0; e < VW; e++) kh.a[e] = db[(j == 1 ? SIDE_B : SIDE_T) * G::HL + k + e - i0];
        }
#pragma unroll
        for (int e = 0; e < VW; e++) {
            if (k + e == 1) kh.a[e] = db[SIDE_L * G::HL + j - j0];
            if (k + e == n) kh.a[e] = db[SIDE_R * G::HL + j - j0];
        }
        if (ve >= 0) {
            const T hx = hh[(ve < HV ? SIDE_L : SIDE_R) * G::HL + j - j0];
            ku = ov_fma(ov_ld(we + ((3 * ONE_EDGES + ve) * ONE_TAPS + 8) * VW), ov_all(hx), ku);
        }
        if (j <= SB::NSAT || (j >= N + 1 - SB::NSAT && j <= N)) {
            const bool lo = j <= SB::NSAT;
            const V hb = ov_ld(sH + SI(k, lo ? 1 : n));
            const T *const ho = hh + (lo ? SIDE_B : SIDE_T) * G::HL + k - i0;
            const T w = T(ONE_DS * (lo ? SB::satw(j) : -SB::satw(N + 1 - j)));
#pragma unroll
            for (int e = 0; e < VW; e++) kv.a[e] += w * (hb.a[e] - ho[e]);
        }
    }
    {
        const V s2 = ov_all(T(1.0 / (ONE_IS * ONE_IS))), cg = ov_all(om.cg);
        kh = ov_mul(kh, ov_all(-H));
        ku = ov_fma(ov_mul(one_x<2>(sUP + so, ve, ei, we), ov_ld(siJy + so)), s2, ov_fma(ku, cg, au));
        if (j <= N)
            kv = ov_fma(ov_mul(one_y<2, false, SW>(sVP + SI(k, 0), (const T *)nullptr, j, N, xr), ov_ld(siJx + so)), s2,
                        ov_fma(kv, cg, aw));
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
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const V &q = f == 0 ? kh : (f == 1 ? ku : kv);
            ov_st(Y1 + po + f * fs, ov_fma(ov_all(ca), q, pv[f]));
            ov_st(ACC + po + f * fs, ov_fma(ov_all(cb), q, pa[f]));
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
            const V &q = f == 0 ? kh : (f == 1 ? ku : kv);
#pragma unroll
            for (int e = 0; e < VW; e++) {
                const T inc = pa[f].a[e] + cb * q.a[e];
                if constexpr (sizeof(T) == 4) kahan_add(pv[f].a[e], cm[f].a[e], inc);
                else pv[f].a[e] = pv[f].a[e] + inc;
            }
            ov_st(V0 + po + f * fs, pv[f]);
            if constexpr (sizeof(T) == 4) ov_st(CMP + po + f * fs, cm[f]);
        }
    }
}

}  // namespace chswe
