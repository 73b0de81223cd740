// nb_pair.cuh -- what the pair kernels of nb_realspace.cu, nb_press.cu and nb_adjoint.cu share: rows of the W1
// lists, sums over the lanes of a subgroup, the Ewald pair terms on the packed two-lane FP32 pipe and
// the FP32 pairs of non-water atoms.
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
// the same for two sums at once, (hi.x, lo.x) and (hi.y, lo.y), on the packed pipe
__device__ __forceinline__ void two_add2(float2 &hi, float2 &lo, float2 v)
{
    const float2 m1 = f2(-1.f), sm = __fadd2_rn(hi, v), bb = __ffma2_rn(hi, m1, sm);
    const float2 eh = __ffma2_rn(__ffma2_rn(bb, m1, sm), m1, hi), ev = __ffma2_rn(bb, m1, v);
    lo = __fadd2_rn(lo, __fadd2_rn(eh, ev));
    hi = sm;
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

template <typename T>
__device__ __forceinline__ void lj_switch_apply(const RepDev &R, T r2, T &e1, T &df1)
{
    if (R.lj_switch && r2 > (T)R.ron2) {
        T d = (T)R.rv2 - r2;
        T sw = d * d * ((T)R.rv2 + (T)2 * r2 - (T)3 * (T)R.ron2) * (T)R.swden;
        T dsw = (T)12 * d * ((T)R.ron2 - r2) * (T)R.swden;
        df1 = df1 * sw + e1 * dsw;
        e1 *= sw;
    }
}

// FP32 pairs of non-water semantics (nb_realspace.cu, atom_pair): a replica's constants held in registers, since a
// pair's arithmetic is no longer than loading them again each time.
struct AtomK {
    float iL0, iL1, iL2, L0, L1, L2, m0, m1, m2, rmax2, rv2, re2, ke;
    WaterK K;
    bool arith, tiny, sw;        // tiny: the hvdw0 rule applies (geometric rule, small-sigma hydrogens)
    __device__ void rules(const RepDev &R)
    {
        re2 = R.re2; ke = held((float)R.epstmp);
        arith = R.arith != 0; tiny = !R.arith && R.hvdw0; sw = R.lj_switch != 0;
    }
    __device__ AtomK(const RepDev &R)
        : iL0(held(R.invL[0])), iL1(held(R.invL[1])), iL2(held(R.invL[2])), L0(held(R.L[0])), L1(held(R.L[1])),
          L2(held(R.L[2])), m0(held(R.Llo[0])), m1(held(R.Llo[1])), m2(held(R.Llo[2])), rmax2(held(R.rmax2)),
          rv2(held(R.rv2)), K{held(ERFCX_P * R.alpha), held(R.ex2c), held(R.c2a)}
    {
        rules(R);
    }
    // values that the caller holds already
    __device__ AtomK(const RepDev &R, float a0, float a1, float a2, float b0, float b1, float b2, float c0, float c1,
                     float c2, float rm, float rv, WaterK k)
        : iL0(a0), iL1(a1), iL2(a2), L0(b0), L1(b1), L2(b2), m0(c0), m1(c1), m2(c2), rmax2(rm), rv2(rv), K(k)
    {
        rules(R);
    }
    // (x + 1.5*2^23) - 1.5*2^23 rounds x to nearest (|x| < 2^22)
    __device__ void image(float &dx, float &dy, float &dz, bool &img) const
    {
        const float nx = fmaf(dx, iL0, 12582912.f) - 12582912.f, ny = fmaf(dy, iL1, 12582912.f) - 12582912.f,
                    nz = fmaf(dz, iL2, 12582912.f) - 12582912.f;
        dx = fmaf(-nx, m0, fmaf(-nx, L0, dx)); dy = fmaf(-ny, m1, fmaf(-ny, L1, dy)); dz = fmaf(-nz, m2, fmaf(-nz, L2, dz));
        img = (nx != 0.f) | (ny != 0.f) | (nz != 0.f);
    }
    // two at once
    __device__ void image2(float2 &x, float2 &y, float2 &z, float2 &nx, float2 &ny, float2 &nz) const
    {
        const float2 mg = f2(12582912.f), nm = f2(-12582912.f);
        nx = __fadd2_rn(__ffma2_rn(x, f2(iL0), mg), nm);
        ny = __fadd2_rn(__ffma2_rn(y, f2(iL1), mg), nm);
        nz = __fadd2_rn(__ffma2_rn(z, f2(iL2), mg), nm);
        x = __ffma2_rn(nx, f2(-m0), __ffma2_rn(nx, f2(-L0), x));
        y = __ffma2_rn(ny, f2(-m1), __ffma2_rn(ny, f2(-L1), y));
        z = __ffma2_rn(nz, f2(-m2), __ffma2_rn(nz, f2(-L2), z));
    }
    // LJ of a pair inside the LJ cutoff: its energy, and minus (dE/dr)/r as the result.  r^-6 and r^-12
    // amplify the approximate rsqrt's error 6 and 12 times: one Newton step first
    __device__ float lj(const RepDev &R, float r2, float rinv, float2 a, float2 b, float &e1) const
    {
        const float ri = fmaf(-0.5f * rinv, fmaf(r2, rinv * rinv, -1.f), rinv), s2 = ri * ri, s6 = s2 * s2 * s2;
        float A, B;
        if (!arith) {
            A = a.x * b.x * s6 * s6;
            B = a.y * b.y * s6;
        } else {
            const float aa = a.x * b.x, sg = 0.5f * (a.y + b.y);
            float b1 = sg * sg * sg;
            b1 = b1 * b1;
            B = aa * b1 * s6;
            A = B * b1 * s6;
        }
        e1 = A - B;
        float df = -6.f * s2 * (A + e1);
        if (sw) lj_switch_apply<float>(R, r2, e1, df);
        return -df;
    }
    // one pair (charges times each other and ke in qq): minus (dE/dr)/r
    __device__ float pair(const RepDev &R, float r2, float qq, float2 a, float2 b, bool t, float &eel, float &elj,
                          float &vir, int &npair) const
    {
        const bool in_lj = r2 < rv2 && !(t && r2 < re2), in_el = r2 < rmax2 && qq != 0.f;
        eel = 0.f; elj = 0.f; vir = 0.f;
        float m = 0.f;
        if (in_lj || in_el) {
            ++npair;
            const float rinv = nb_rsqrt_approx(r2);
            if (in_el) m = ewald1(K, r2, rinv, qq, eel);
            if (in_lj) {
                const float l = lj(R, r2, rinv, a, b, elj);
                vir = l * r2;
                m += l;
            }
        }
        return m;
    }
};

}  // namespace
