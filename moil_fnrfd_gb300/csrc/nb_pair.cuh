// nb_pair.cuh -- what the water kernels of nb_realspace.cu and nb_press.cu share: rows of the W1
// lists, sums over the lanes of a subgroup, and the Ewald pair terms on the packed two-lane FP32 pipe.
#pragma once
#include "nb_common.cuh"

namespace {

// water i's W1 row: entry v is the v-th in-cutoff molecule from the front for v < nn, then
// the skin-only molecules from the back of the row
template <typename E>
struct W1Row {
    const E *row;
    int nn, n, cap, base;
    __device__ W1Row(const int2 *__restrict__ cnt, const void *wl1, int cap_row, int i, int base_)
    {
        const int2 c = cnt[i];
        row = (const E *)wl1 + (size_t)i * cap_row;
        // an overflowed row (counts above the capacity) is read within the row; the
        // evaluation reports the overflow and is redone with larger rows
        nn = min(c.x, cap_row);
        n = min(c.x + c.y, cap_row);
        cap = cap_row;
        base = sizeof(E) == 2 ? base_ : 0;     // uint16 entries are offsets from the replica's first water
    }
    __device__ const E *addr(int v) const { return row + (v < nn ? v : cap - 1 - (v - nn)); }
    __device__ int at(int v) const { return base + (int)*addr(v); }
};

// Sum over the W lanes of a subgroup (W a power of two, all lanes of the warp present).
template <int W> __device__ __forceinline__ long long sub_sum(long long v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, W);
    return v;
}
template <int W> __device__ __forceinline__ int sub_sum(int v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, W);
    return v;
}
template <int W> __device__ __forceinline__ double sub_sum(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, W);
    return v;
}

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Real-space Ewald Coulomb of two site pairs (packed) and of one: the energy qq erfc(alpha r)/r
// and minus its (dE/dr)/r.  erfc(x) = exp(-x^2) t P(A t + B), t = 1 / (1 + P x), x = alpha r, with
// no clamp to the fitted range x <= 4.5: beyond it the fit extrapolates smoothly (relative
// error 1e-5 at x = 7, 2e-3 at x = 3500) and exp(-x^2) < 1e-8 makes the term negligible.
struct WaterK {
    float palpha, ex2c, c2a;
};
__device__ __forceinline__ float2 ewald2(const WaterK &K, float2 rr2, float2 qq, float2 &e)
{
    const float2 rinv = f2(nb_rsqrt_approx(rr2.x), nb_rsqrt_approx(rr2.y));
    const float2 arg = __fmul2_rn(rr2, f2(K.ex2c));
    const float2 den = __ffma2_rn(f2(K.palpha), __fmul2_rn(rr2, rinv), f2(1.f));
    const float2 tt = f2(nb_rcp_approx(den.x), nb_rcp_approx(den.y));
    const float2 u = __ffma2_rn(f2(ERFCX_A), tt, f2(ERFCX_B));
    const float C[ERFCX_NC] = ERFCX_COEFS;
    float2 p = f2(C[ERFCX_NC - 1]);
#pragma unroll
    for (int m = ERFCX_NC - 2; m >= 0; --m) p = __ffma2_rn(p, u, f2(C[m]));
    const float2 ex = f2(nb_ex2_approx(-arg.x), nb_ex2_approx(-arg.y));
    e = __fmul2_rn(__fmul2_rn(qq, __fmul2_rn(ex, __fmul2_rn(tt, p))), rinv);
    return __fmul2_rn(__ffma2_rn(__fmul2_rn(qq, f2(K.c2a)), ex, e), __fmul2_rn(rinv, rinv));
}
__device__ __forceinline__ float ewald1(const WaterK &K, float rr2, float rinv, float qq, float &e)
{
    const float tt = nb_rcp_approx(fmaf(K.palpha, rr2 * rinv, 1.f)), u = fmaf(ERFCX_A, tt, ERFCX_B);
    const float C[ERFCX_NC] = ERFCX_COEFS;
    float p = C[ERFCX_NC - 1];
#pragma unroll
    for (int m = ERFCX_NC - 2; m >= 0; --m) p = fmaf(p, u, C[m]);
    const float ex = nb_ex2_approx(-rr2 * K.ex2c);
    e = qq * (ex * (tt * p)) * rinv;
    return fmaf(qq * K.c2a, ex, e) * (rinv * rinv);
}
// a value the compiler holds instead of loading it again (the replica's constants inside the pair
// loops: 2.5% of the water stage)
__device__ __forceinline__ float held(float x)
{
    asm volatile("" : "+f"(x));
    return x;
}
// hi + lo += v (TwoSum, Knuth: the rounding error of hi + v collects in lo)
__device__ __forceinline__ void two_add(float2 &a, float v)
{
    const float sm = a.x + v, bb = sm - a.x;
    a = make_float2(sm, a.y + ((a.x - (sm - bb)) + (v - bb)));
}
template <int W> __device__ __forceinline__ float2 sub_two_sum(float2 a)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
        const float hi = __shfl_xor_sync(0xffffffffu, a.x, o, W), lo = __shfl_xor_sync(0xffffffffu, a.y, o, W);
        two_add(a, hi);
        a.y += lo;
    }
    return a;
}

}  // namespace
