// swe_vec.cuh -- 16-byte vectors of consecutive points: four FP32 or two FP64 values.
#pragma once

#include <cstdint>

namespace chswe {

// A 16-byte vector of T.
template <class T>
struct alignas(16) OV {
    static constexpr int W = 16 / (int)sizeof(T);
    T a[W];
};

template <class T, int W>
__device__ __forceinline__ OV<T> ov_zero()
{
    OV<T> r;
#pragma unroll
    for (int e = 0; e < W; e++) r.a[e] = T(0);
    return r;
}

// Packed arithmetic: two FP32 operations per instruction on aligned register pairs
// (fma.rn.f32x2), plain FP64.
__device__ __forceinline__ uint64_t pk(float x, float y) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y)); return r; }
__device__ __forceinline__ void upk(uint64_t v, float &x, float &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
#define CHSWE_OV_OP(NAME, F32, F64)                                                                            \
    __device__ __forceinline__ OV<float> NAME(const OV<float> &a, const OV<float> &b)                           \
    {                                                                                                          \
        OV<float> r;                                                                                           \
        _Pragma("unroll") for (int e = 0; e < 4; e += 2) {                                                     \
            uint64_t v;                                                                                        \
            asm(F32 " %0, %1, %2;" : "=l"(v) : "l"(pk(a.a[e], a.a[e + 1])), "l"(pk(b.a[e], b.a[e + 1])));        \
            upk(v, r.a[e], r.a[e + 1]);                                                                        \
        }                                                                                                      \
        return r;                                                                                              \
    }                                                                                                          \
    __device__ __forceinline__ OV<double> NAME(const OV<double> &a, const OV<double> &b)                        \
    {                                                                                                          \
        return OV<double>{{a.a[0] F64 b.a[0], a.a[1] F64 b.a[1]}};                                              \
    }
CHSWE_OV_OP(ov_add, "add.rn.f32x2", +)
CHSWE_OV_OP(ov_sub, "sub.rn.f32x2", -)
CHSWE_OV_OP(ov_mul, "mul.rn.f32x2", *)
#undef CHSWE_OV_OP
__device__ __forceinline__ OV<float> ov_fma(const OV<float> &a, const OV<float> &b, const OV<float> &c)
{
    OV<float> r;
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        uint64_t v;
        asm("fma.rn.f32x2 %0, %1, %2, %3;"
            : "=l"(v)
            : "l"(pk(a.a[e], a.a[e + 1])), "l"(pk(b.a[e], b.a[e + 1])), "l"(pk(c.a[e], c.a[e + 1])));
        upk(v, r.a[e], r.a[e + 1]);
    }
    return r;
}
__device__ __forceinline__ OV<double> ov_fma(const OV<double> &a, const OV<double> &b, const OV<double> &c)
{
    return OV<double>{{fma(a.a[0], b.a[0], c.a[0]), fma(a.a[1], b.a[1], c.a[1])}};
}
template <class T>
__device__ __forceinline__ OV<T> ov_all(T x)
{
    OV<T> r;
#pragma unroll
    for (int e = 0; e < OV<T>::W; e++) r.a[e] = x;
    return r;
}

template <class T>
__device__ __forceinline__ OV<T> ov_ld(const T *p) { return *reinterpret_cast<const OV<T> *>(p); }
template <class T>
__device__ __forceinline__ void ov_st(T *p, const OV<T> &v) { *reinterpret_cast<OV<T> *>(p) = v; }

}  // namespace chswe
