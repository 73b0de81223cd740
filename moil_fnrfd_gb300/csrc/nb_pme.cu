// nb_pme.cu -- PME reciprocal sum (pot/ewald_receip.f:101-1080), GB300 layout.
//
// The reference spreads into a padded complex grid, runs two full 3D C2C FFTs
// (pubz3d / FFTPACK) with the influence function in between (scalar_sum) and gathers.
// Here the real-space charge grid never exists in HBM:
//   pme_site       (in the coordinate preparation) fractional coordinates
//                  fr = n (w - anint(w) + 1/2) (:250-260) and, one byte per site, int(fr3),
//                  the last z plane of the site's stencil
//   plane_fwd      one CTA per (replica, z plane): the sites whose z stencil touches the plane
//                  are picked from the replica's z bytes (plane_sites), their 4x4 x-y stencils
//                  accumulated in shared memory in 32-bit fixed point (order independent,
//                  hence deterministic), then R2C along x and C2C along y in shared memory;
//                  the half-complex plane goes to HBM as [z][kx][ky]
//   zconv          one CTA per (replica, kx, run of ky): C2C along z, the influence function
//                  exp(-pi^2 m^2 / alpha^2) / (pi V B(m) m^2) with the FP64 energy sum
//                  (scalar_sum, :723-812), inverse C2C along z, written back in place
//   plane_inv      one CTA per (replica, z plane): inverse C2C along y, C2R along x in shared
//                  memory; FP32: the real plane back to HBM for pme_gather; FP64: each atom's
//                  share of the gradient from this plane (grad_sum, :815-970) into its own slot --
//                  four planes, four slots, summed at the end
//   pme_gather     (FP32) each site's gradient from the real planes
// FFTs (FP32 path): Stockham autosort with radices up to 10 (two passes per line for most lengths:
// the composite codelets of nb_fft.cuh); every pass transforms all lines of a tile at once, the block's threads spread over (line, butterfly) pairs, with the
// index arithmetic (twiddle step, destination) read from per-stage tables built on the host
// and the line number obtained by a multiply-high by a precomputed magic constant.  The
// last pass of a direction stores transposed, so the next direction reads contiguous lines.
// The plain FP64 path runs the same passes in FP64.
// Inverse transforms are conj(FFT(conj(x))), unnormalised like FFTPACK's cfftb.
#include <mutex>

#include "nb_fft.cuh"
#include "nb_internal.h"

namespace {

__host__ __device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// ---------------------------------------------------------------------------------
// PME records and z bytes of every site (handles whose coordinate preparation does not write
// them, nb_fused_sites)
template <typename T>
__global__ void __launch_bounds__(256) k_pme_sites(int nsite, const int *__restrict__ site_rep,
                                                   const RepDev *__restrict__ reps, const void *pos_v, const void *q_v,
                                                   void *fr_v, unsigned char *__restrict__ zidx)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsite) return;
    typedef typename vec4<T>::type T4;
    const T4 p = ((const T4 *)pos_v)[s];
    const T x[3] = {p.x, p.y, p.z};
    unsigned char z;
    ((T4 *)fr_v)[s] = pme_site(reps[site_rep[s]], x, ((const T *)q_v)[s], z);
    zidx[s] = z;
}

// ---------------------------------------------------------------------------------
// Which of 16 sites' z bytes reach plane z: bit e set where (byte e - z) mod n3 < 4
__device__ __forceinline__ unsigned z_hits(uint4 v, int z, int n3)
{
    const unsigned u[4] = {v.x, v.y, v.z, v.w};
    unsigned m = 0u;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        unsigned x;
        if (z + 3 < n3) {
            // bytes below 128 each: (b | 0x80) - z never borrows from its neighbour, and bits 2-6
            // with the inverted top bit are zero exactly for 0 <= b - z < 4
            x = (((u[w] | 0x80808080u) - 0x01010101u * (unsigned)z) ^ 0x80808080u) & 0xfcfcfcfcu;
            x = ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);          // 0x80 in zero bytes
        } else {
            x = 0u;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int d = (int)((u[w] >> (8 * e)) & 0xffu) - z;
                d += d < 0 ? n3 : 0;
                x |= (d < 4 ? 0x80u : 0u) << (8 * e);
            }
        }
        m |= ((((x >> 7) * 0x01020408u) >> 24) & 0xfu) << (4 * w);
    }
    return m;
}

// The sites of replica R whose stencil reaches plane z: fn(n) is called by the whole block with n
// entries (site << 2 | plane within the stencil, 0 = the last) in queue, cap ints of shared memory
// that are free for this; several times when they do not fit at once or the replica has more
// than 64 sites per thread.  A thread tests 16 sites' z bytes per load, so a block reads one byte
// per site of its replica (5 KB for 5,000 sites, from L2) where lists of sites per plane took
// four launches (binning, scan, scatter and a memset: 18 us before the planes of a small system
// could start) and 70 bytes of traffic per site.  The order of the entries varies, which the
// integer planes do not show.
#define NB_ZLOADS 4
template <typename Fn>
__device__ __forceinline__ void plane_sites(const RepDev &R, int nW, int z, const unsigned char *__restrict__ zidx,
                                            int *queue, int cap, Fn fn)
{
    __shared__ int count;
    const int t = threadIdx.x, n3 = R.n3;
    if (t == 0) count = 0;
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
        // the water sites, then the others
        const int s0 = r == 0 ? 3 * R.wat0 : 3 * nW + R.oth0, s1 = s0 + (r == 0 ? 3 * R.nwat : R.noth);
#pragma unroll 1
        for (int c = s0 & ~15; c < s1; c += 16 * NB_ZLOADS * blockDim.x) {
            uint4 v[NB_ZLOADS];
            unsigned m[NB_ZLOADS];
#pragma unroll
            for (int q = 0; q < NB_ZLOADS; ++q) {
                const int s = c + 16 * (t + q * (int)blockDim.x);
                v[q] = s < s1 ? *reinterpret_cast<const uint4 *>(zidx + s) : make_uint4(0u, 0u, 0u, 0u);
            }
            int hits = 0;
#pragma unroll
            for (int q = 0; q < NB_ZLOADS; ++q) {
                const int s = c + 16 * (t + q * (int)blockDim.x);
                m[q] = 0u;
                if (s < s1) {
                    m[q] = z_hits(v[q], z, n3);
                    if (s < s0) m[q] &= 0xffffu << (s0 - s);
                    if (s + 16 > s1) m[q] &= 0xffffu >> (s + 16 - s1);
                    hits += __popc(m[q]);
                }
            }
            __syncthreads();           // count is zero; the queue is free
            const int p = hits ? atomicAdd(&count, hits) : 0;
            __syncthreads();
            const int total = count;
#pragma unroll 1
            for (int base = 0; base < total; base += cap) {
                if (hits) {
                    int k = p - base;
#pragma unroll 1
                    for (int q = 0; q < NB_ZLOADS; ++q) {
                        const int s = c + 16 * (t + q * (int)blockDim.x);
                        unsigned b = q == 0 ? m[0] : (q == 1 ? m[1] : (q == 2 ? m[2] : m[3]));
                        while (b) {
                            const int e = s + __ffs(b) - 1;
                            b &= b - 1u;
                            if (k >= 0 && k < cap) {
                                int d = (int)zidx[e] - z;
                                d += d < 0 ? n3 : 0;
                                queue[k] = e << 2 | d;
                            }
                            ++k;
                        }
                    }
                }
                __syncthreads();
                fn(min(cap, total - base));
                __syncthreads();
            }
            if (t == 0) count = 0;     // everyone has read total (a barrier since, or it was zero)
        }
    }
}

// plane accumulation.  FP32: int32 fixed point; the caller pre-multiplies by the replica's
// spread_scale (nb_spread_exp) so one contribution stays below 2^25 and rounds it to the
// nearest integer.  Integer addition makes the plane independent of the order of the
// atomics.  FP64: FP64 atomics.
template <typename T> struct Acc;
template <> struct Acc<float> {
    typedef int type;
    __device__ static void add(type *p, float x) { atomicAdd(p, __float2int_rn(x)); }
    __device__ static float get(type v, float inv) { return __int2float_rn(v) * inv; }
};
template <> struct Acc<double> {
    typedef double type;
    __device__ static void add(type *p, double v) { atomicAdd(p, v); }
    __device__ static double get(type v, double) { return v; }
};

// Order-4 weights of fractional offset w in closed form (the cardinal cubic B-spline that
// fill_bspline's recursion evaluates, ewald_receip.f:1022-1080):
//   th = ((1-w)^3, 4 - 6w^2 + 3w^3, 1 + 3w + 3w^2 - 3w^3, w^3) / 6
//   dth = (-(1-w)^2, 3w^2 - 4w, 1 + 2w - 3w^2, w^2) / 2
template <typename T>
__device__ __forceinline__ void bsp4_th(T w, T th[4])
{
    const T w2 = w * w, w3 = w2 * w, m = (T)1 - w, s = (T)(1.0 / 6.0);
    th[0] = s * m * m * m;
    th[1] = s * ((T)4 - (T)6 * w2 + (T)3 * w3);
    th[2] = s * ((T)1 + (T)3 * (w + w2 - w3));
    th[3] = s * w3;
}
// 6 th: the same weights without the factor 1/6, whose FP32 rounding (2.98e-8 high) would
// raise every spread charge by 9e-8 and the reciprocal energy by 1.8e-7; the FP32 spread
// applies 1/216 once per site (spread216)
__device__ __forceinline__ void bsp4_th6(float w, float th[4])
{
    const float w2 = w * w, w3 = w2 * w, m = 1.f - w;
    th[0] = m * m * m;
    th[1] = 4.f - 6.f * w2 + 3.f * w3;
    th[2] = 1.f + 3.f * (w + w2 - w3);
    th[3] = w3;
}
template <typename T>
__device__ __forceinline__ void bsp4_dth(T w, T d[4])
{
    const T w2 = w * w, m = (T)1 - w;
    d[0] = (T)-0.5 * m * m;
    d[1] = (T)0.5 * w * ((T)3 * w - (T)4);
    d[2] = (T)0.5 * ((T)1 + (T)2 * w - (T)3 * w2);
    d[3] = (T)0.5 * w2;
}
// grid index i in [-3, n] wrapped into [0, n)
__device__ __forceinline__ int pme_wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// the 4x4 x-y stencil of n queued sites (plane_sites) into the plane; one site per thread
template <typename T>
__device__ __forceinline__ void spread_sites(const RepDev &R, const int *queue, int n,
                                             const typename vec4<T>::type *fr, typename Acc<T>::type *acc, T scale)
{
    typedef typename vec4<T>::type T4;
    const int n1 = R.n1, n2 = R.n2;
    for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
        const int e = queue[idx], t3 = 3 - (e & 3);
        const T4 f = fr[e >> 2];
        int i1, i2, i3;
        T w1, w2, w3;
        pme_fr_split(f.x, i1, w1);
        pme_fr_split(f.y, i2, w2);
        pme_fr_split(f.z, i3, w3);
        T th1[4], th2[4], th3[4];
        if constexpr (sizeof(T) == 4) {
            bsp4_th6(w1, th1);
            bsp4_th6(w2, th2);
            bsp4_th6(w3, th3);
        } else {
            bsp4_th<T>(w1, th1);
            bsp4_th<T>(w2, th2);
            bsp4_th<T>(w3, th3);
        }
        const T qz = (t3 == 0 ? th3[0] : (t3 == 1 ? th3[1] : (t3 == 2 ? th3[2] : th3[3]))) * (f.w * scale);
        int xs[4];
#pragma unroll
        for (int t1 = 0; t1 < 4; ++t1) xs[t1] = pme_wrap(i1 - 3 + t1, n1);
#pragma unroll
        for (int t2 = 0; t2 < 4; ++t2) {
            typename Acc<T>::type *row = acc + pme_wrap(i2 - 3 + t2, n2) * n1;
            const T v = th2[t2] * qz;
#pragma unroll
            for (int t1 = 0; t1 < 4; ++t1) Acc<T>::add(row + xs[t1], v * th1[t1]);
        }
    }
}

// gradient (or potential) share of one plane (real values Rp[ky][x]) for n queued sites
template <typename T>
__device__ __forceinline__ void gather_sites(const RepDev &R, const int *queue, int n,
                                             const typename vec4<T>::type *fr, const T *Rp, T *__restrict__ part,
                                             bool pot)
{
    typedef typename vec4<T>::type T4;
    const int n1 = R.n1, n2 = R.n2;
    for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
        const int e = queue[idx], s = e >> 2, t3 = 3 - (e & 3);
        const T4 f = fr[s];
        int i1, i2, i3;
        T w1, w2, w3;
        pme_fr_split(f.x, i1, w1);
        pme_fr_split(f.y, i2, w2);
        pme_fr_split(f.z, i3, w3);
        T th1[4], dt1[4], th2[4], dt2[4], th3[4], dt3[4];
        bsp4_th<T>(w1, th1); bsp4_dth<T>(w1, dt1);
        bsp4_th<T>(w2, th2); bsp4_dth<T>(w2, dt2);
        bsp4_th<T>(w3, th3); bsp4_dth<T>(w3, dt3);
        const T z0 = t3 == 0 ? th3[0] : (t3 == 1 ? th3[1] : (t3 == 2 ? th3[2] : th3[3]));
        const T z1 = t3 == 0 ? dt3[0] : (t3 == 1 ? dt3[1] : (t3 == 2 ? dt3[2] : dt3[3]));
        int xs[4];
#pragma unroll
        for (int t1 = 0; t1 < 4; ++t1) xs[t1] = pme_wrap(i1 - 3 + t1, n1);
        T gx = 0, gy = 0, gz = 0;
#pragma unroll
        for (int t2 = 0; t2 < 4; ++t2) {
            const T *row = Rp + pme_wrap(i2 - 3 + t2, n2) * n1;
            T sx = 0, sy = 0;
#pragma unroll
            for (int t1 = 0; t1 < 4; ++t1) {
                const T q = row[xs[t1]];
                sx += q * dt1[t1];
                sy += q * th1[t1];
            }
            gx += sx * th2[t2];
            gy += sy * dt2[t2];
            gz += sy * th2[t2];
        }
        if (pot) {
            // the potential share of this plane (parameter derivatives): one slot per plane
            part[4 * (size_t)s + t3] = gz * z0;
            continue;
        }
        T *o = part + 12 * (size_t)s + 3 * t3;
        o[0] = gx * z0;
        o[1] = gy * z0;
        o[2] = gz * z1;
    }
}

// influence function (scalar_sum): m folded as MOIL does (k > ceil(n/2) - 1 -> k - n)
template <typename T>
__device__ __forceinline__ T eterm_of(const RepDev &R, const T *bsp, int kx, int ky, int kz)
{
    if (kx == 0 && ky == 0 && kz == 0) return (T)0;
    const int nf2 = (R.n2 + 1) / 2, nf3 = (R.n3 + 1) / 2;
    int m2 = ky < nf2 ? ky : ky - R.n2, m3 = kz < nf3 ? kz : kz - R.n3;
    T mh1 = (T)kx * rep_invL<T>(R, 0), mh2 = (T)m2 * rep_invL<T>(R, 1), mh3 = (T)m3 * rep_invL<T>(R, 2);
    T msq = mh1 * mh1 + mh2 * mh2 + mh3 * mh3;
    return exp(-(T)R.pme_fac * msq) /
           ((T)R.pivol * bsp[kx] * bsp[R.n1 + ky] * bsp[R.n1 + R.n2 + kz] * msq);
}

// =================================================================================
// FP32 path: block-cooperative table-driven Stockham passes

#define NB_TKF 32     // z lines per zconv CTA (FP32 path)
#define NB_TK 16      // (FP64 path)

// Shared-memory layout of the intermediate results between Stockham stages: element e of a
// buffer is stored at e + e/16 (one spare slot per 16 float2, i.e. per 128 bytes), so the
// strided stores of the early stages (stride R for radix R) and the strided reads of the
// later ones spread over all banks.  Inputs and outputs of a transform keep the caller's
// layout.
__host__ __device__ __forceinline__ int swz(int e) { return e + (e >> 4); }
// float2 slots that hold m elements in the spread layout
__host__ __device__ __forceinline__ int swz_elems(int m) { return m + (m >> 4) + 1; }

// Where a transform's first stage reads and its last one writes, besides the shared-memory buffers
enum FftIn { IN_LINES, IN_SPREAD, IN_CONJ, IN_PLANE };
enum FftOut { OUT_LINES, OUT_SPREAD, OUT_TRANSPOSED, OUT_ROWS };
template <typename T> struct FftEnds {
    typedef typename cplx<T>::type C;
    const C *in = nullptr;   // IN_CONJ: lines in global memory, conjugated
    const typename Acc<T>::type *acc = nullptr;     // IN_PLANE: the charge plane, rows 2l and 2l + 1 as line l
    T inv = 0;
    int rows = 0;                 // rows of the plane (IN_PLANE, OUT_ROWS)
    C *out = nullptr;        // OUT_LINES: to global memory
    T *real = nullptr;        // OUT_ROWS: Re and -Im of line l as rows 2l and 2l + 1
};

// One Stockham stage over L lines of length n = RADIX * nb.  Source line l at src + l*ss (contiguous)
// or in the spread layout (IN_SPREAD); destination dst + l*ds, in the spread layout (OUT_SPREAD) or
// transposed (dst[k*ds + l]); or the ends above.  CONJ_OUT conjugates the stored values.  tab / tw
// point into shared memory (fft_ctx_load).
template <int RADIX, int IN, int OUT, bool CONJ_OUT, typename T, typename C>
__device__ __forceinline__ void fft_pass_r(const C *__restrict__ src, C *__restrict__ dst, const FftEnds<T> &E,
                                           int L, int ss, int ds, int Ns, int nb, unsigned magic,
                                           const int2 *__restrict__ tab, const C *__restrict__ tw)
{
    const int total = L * nb;
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        int line = nb == 1 ? b : (int)__umulhi((unsigned)b, magic);
        int j = b - line * nb;
        int2 e = tab[j];
        const int s0 = line * ss + j;
        C v[RADIX];
        if (IN == IN_PLANE) {
            const typename Acc<T>::type *a0 = E.acc + 2 * line * ss + j, *a1 = a0 + ss;
            const bool two = 2 * line + 1 < E.rows;
#pragma unroll
            for (int r = 0; r < RADIX; ++r)
            {
                v[r].x = Acc<T>::get(a0[r * nb], E.inv);
                v[r].y = two ? Acc<T>::get(a1[r * nb], E.inv) : (T)0;
            }
        } else {
#pragma unroll
            for (int r = 0; r < RADIX; ++r)
                v[r] = IN == IN_CONJ ? cconj(E.in[s0 + r * nb]) : src[IN == IN_SPREAD ? swz(s0 + r * nb) : s0 + r * nb];
        }
        if (IN == IN_SPREAD) {          // (a first stage's twiddles are all one)
#pragma unroll
            for (int r = 1; r < RADIX; ++r) v[r] = cmul(v[r], tw[r * e.x]);
        }
        bfly<RADIX>(v);
#pragma unroll
        for (int r = 0; r < RADIX; ++r) {
            C o = CONJ_OUT ? cconj(v[r]) : v[r];
            int k = e.y + r * Ns;
            if (OUT == OUT_TRANSPOSED) {
                dst[k * ds + line] = o;
            } else if (OUT == OUT_ROWS) {
                E.real[2 * line * ds + k] = o.x;
                if (2 * line + 1 < E.rows) E.real[(2 * line + 1) * ds + k] = -o.y;
            } else {
                const int d = line * ds + k;
                dst[OUT == OUT_SPREAD ? swz(d) : d] = o;
            }
        }
    }
    __syncthreads();
}

template <int IN, int OUT, bool CONJ_OUT, typename T, typename C>
__device__ __forceinline__ void fft_pass(int R, const C *src, C *dst, const FftEnds<T> &E, int L, int ss, int ds,
                                         int Ns, int nb, unsigned magic, const int2 *tab, const C *tw)
{
    switch (R) {
    case 2: fft_pass_r<2, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 3: fft_pass_r<3, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 4: fft_pass_r<4, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 5: fft_pass_r<5, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 6: fft_pass_r<6, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 8: fft_pass_r<8, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    case 9: fft_pass_r<9, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    default: fft_pass_r<10, IN, OUT, CONJ_OUT>(src, dst, E, L, ss, ds, Ns, nb, magic, tab, tw); break;
    }
}

// A plan with its twiddles and stage table, staged in shared memory by fft_ctx_load so the
// butterflies read them without global-memory latency.
template <typename C> struct FftCtx {
    const FftPlanDev *p;
    const int2 *tab;      // plan-local: stage s at tab + p->off[s]
    const C *tw;     // plan-local twiddles, n entries
};

// shared-memory bytes of one staged plan of length n
size_t fft_ctx_bytes(int n, size_t elem);

// copies from global to shared memory that no register and no thread waits for until async_wait
__device__ __forceinline__ void async_copy16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copy8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// the tables of a plan of length n: len 16-byte units (plan, twiddles, stage table); complete after
// async_wait and a barrier
template <typename C>
__device__ __forceinline__ unsigned char *fft_ctx_load(unsigned char *dst, const int4 *__restrict__ src, int len, int n,
                                                       FftCtx<C> &ctx)
{
    for (int k = threadIdx.x; k < len; k += blockDim.x) async_copy16(dst + 16 * k, src + k);
    ctx.p = (const FftPlanDev *)dst;
    ctx.tw = (const C *)(dst + align16(sizeof(FftPlanDev)));
    ctx.tab = (const int2 *)((const unsigned char *)ctx.tw + align16(n * sizeof(C)));
    return dst + 16 * (size_t)len;
}

// Full forward FFT of L lines of length n held in a (line stride in_ss), or read as IN says; b is
// scratch.  The last pass stores as OUT says with stride out_ds (OUT_TRANSPOSED: the transposed row
// stride); the stages between keep the spread layout.  Returns the buffer holding the result;
// CONJ_LAST conjugates the final output (second half of an inverse transform).
template <int IN, int OUT, bool CONJ_LAST, typename T, typename C>
__device__ C *fft_lines(const FftCtx<C> &c, C *a, C *b, const FftEnds<T> &E, int L, int in_ss, int out_ds)
{
    const FftPlanDev &p = *c.p;
    C *src = a, *dst = b;
    const int n = p.n, nst = p.nst;
    for (int s = 0; s < nst; ++s) {
        const int2 *t = c.tab + p.off[s];
        C *o = s + 1 == nst && E.out ? E.out : dst;
        if (s + 1 < nst) {
            if (s == 0)
                fft_pass<IN, OUT_SPREAD, false>(p.rad[s], src, o, E, L, in_ss, n, p.ns[s], p.nb[s], p.magic[s], t, c.tw);
            else
                fft_pass<IN_SPREAD, OUT_SPREAD, false>(p.rad[s], src, o, E, L, n, n, p.ns[s], p.nb[s], p.magic[s], t, c.tw);
        } else if (s == 0) {
            fft_pass<IN, OUT, CONJ_LAST>(p.rad[s], src, o, E, L, in_ss, out_ds, p.ns[s], p.nb[s], p.magic[s], t, c.tw);
        } else {
            fft_pass<IN_SPREAD, OUT, CONJ_LAST>(p.rad[s], src, o, E, L, n, out_ds, p.ns[s], p.nb[s], p.magic[s], t, c.tw);
        }
        C *x = src; src = dst; dst = x;
    }
    return src;
}

// complex slots of each of the two plane buffers of the plane kernels: the packed rows
// (ceil(n2/2) lines of n1), the half spectrum (n1/2+1 lines of n2, stored with the odd row
// stride n2|1 after the forward x pass), the transposed inverse y output (n2 rows of stride
// (n1/2+1)|1), and either kind in the spread layout of the stages between; even, so the
// buffers after it stay 16-byte aligned
__host__ __device__ __forceinline__ int plane_buf_elems(int n1, int n2)
{
    const int n1h = n1 / 2 + 1, a = ((n2 + 1) / 2) * n1, b = n1h * n2;
    int m = swz_elems(a > b ? a : b);
    m = m > n1h * (n2 | 1) ? m : n1h * (n2 | 1);
    m = m > n2 * (n1h | 1) ? m : n2 * (n1h | 1);
    return (m + 1) & ~1;
}

// complex slots of each zconv buffer: the tile's lines of n3 at the odd stride n3|1 or spread
template <typename T> __host__ __device__ constexpr int col_tile() { return sizeof(T) == 4 ? NB_TKF : NB_TK; }
template <typename T> __host__ __device__ __forceinline__ int zconv_buf_elems(int n3)
{
    const int tk = col_tile<T>(), a = swz_elems(tk * n3), b = tk * (n3 | 1);
    return ((a > b ? a : b) + 1) & ~1;
}

// Charge plane z: the sites' stencils into an int32 plane, then the x and y transforms.  Bound: instruction
// issue and the shared-memory pipe; of 180 us for 9,535 planes of about 37 x 37 (256 replicas) the
// transforms take 65, the selection of the sites 48, their stencils 42.  Two passes per axis (wide
// radices), the first from the int32 plane and the last to the grid, without a staging copy at either
// end: 512 replicas 1981 -> 1939 us per evaluation with the inverse's, 24 images 94.5 -> 90.6.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 2) k_plane_fwd(const PlaneWork *__restrict__ work, const RepDev *__restrict__ reps,
                                                     const int4 *__restrict__ blob,
                                                     int nW, const unsigned char *__restrict__ zidx,
                                                     const typename vec4<T>::type *__restrict__ fr,
                                                     typename cplx<T>::type *__restrict__ grid)
{
    typedef typename cplx<T>::type C;
    typedef typename Acc<T>::type A;
    extern __shared__ __align__(16) unsigned char smem[];
    const PlaneWork w = work[blockIdx.x];
    const RepDev &R = reps[w.rep];
    const int n1 = w.n1, n2 = w.n2, n1h = n1 / 2 + 1, n2p = (n2 + 1) >> 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    C *B0 = (C *)smem, *B1 = B0 + plane_buf_elems(n1, n2);
    A *acc = (A *)B0;                            // the charge plane lives in B0 until it is packed
    FftCtx<C> c1, c2;
    unsigned char *ctx = (unsigned char *)(B1 + plane_buf_elems(n1, n2));
    ctx = fft_ctx_load(ctx, blob + w.bx, w.lx, n1, c1);
    fft_ctx_load(ctx, blob + w.by, w.ly, n2, c2);
    for (int k = threadIdx.x; k < n1 * n2; k += blockDim.x) acc[k] = 0;
    plane_sites(R, nW, w.z, zidx, (int *)B1, (int)(sizeof(C) / 4) * plane_buf_elems(n1, n2),
                [&](int n) { spread_sites<T>(R, (const int *)B1, n, fr, acc, sizeof(T) == 4 ? (T)R.spread216 : (T)1); });
    async_wait();
    __syncthreads();
    // x transform of real rows two at a time: line p carries row 2p as its real part and
    // row 2p+1 as its imaginary part, read from the int32 plane
    FftEnds<T> ex, ey;
    ex.acc = acc; ex.inv = sizeof(T) == 4 ? (T)R.spread_inv : (T)1; ex.rows = n2;
    C *Z = fft_lines<IN_PLANE, OUT_LINES, false>(c1, B0, B1, ex, n2p, n1, n1);
    C *X = Z == B1 ? B0 : B1;
    // separate the two real transforms (X_2p = (Z_k + conj Z_-k)/2, X_2p+1 = -i (Z_k - conj Z_-k)/2)
    // and keep kx < n1h, transposed to [kx][y] lines of n2 at the odd row stride sT (the lanes'
    // stores then fall in distinct banks)
    const int sT = n2 | 1;
    for (int p = warp; p < n2p; p += nwarp)
        for (int k = lane; k < n1h; k += 32) {
            const C a = Z[p * n1 + k], b = Z[p * n1 + (k == 0 ? 0 : n1 - k)];
            const T h = (T)0.5;
            C u, v;
            u.x = h * (a.x + b.x); u.y = h * (a.y - b.y);
            v.x = h * (a.y + b.y); v.y = h * (b.x - a.x);
            X[k * sT + 2 * p] = u;
            if (2 * p + 1 < n2) X[k * sT + 2 * p + 1] = v;
        }
    __syncthreads();
    // y: n1h lines of n2, to the grid
    ey.out = grid + w.g0 + (size_t)w.z * n1h * n2;
    fft_lines<IN_LINES, OUT_LINES, false>(c2, X, Z, ey, n1h, sT, n2);
}

__global__ void __launch_bounds__(256, 6) k_zconv_f(const ColWork *__restrict__ work, const RepDev *__restrict__ reps,
                                                 const int4 *__restrict__ blob,
                                                 const float *__restrict__ etab_all, float2 *__restrict__ grid,
                                                 double *__restrict__ e_col)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[8];
    const ColWork w = work[blockIdx.x];
    const RepDev &R = reps[w.rep];
    const int n1 = w.n1, n2 = w.n2, n3 = w.n3, n1h = n1 / 2 + 1;
    const int tk = w.nky;
    const float *etab = etab_all + w.bsp0;
    float2 *A = (float2 *)smem, *B = A + zconv_buf_elems<float>(n3);
    FftCtx<float2> c3;
    fft_ctx_load((unsigned char *)(B + zconv_buf_elems<float>(n3)), blob + w.bz, w.lz, n3, c3);
    const int sA = n3 | 1;    // odd line stride of the columns as loaded and stored
    float2 *g = grid + w.g0 + (size_t)w.kx * n2 + w.ky0;
    const size_t zs = (size_t)n1h * n2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int kz = warp; kz < n3; kz += 8)
        if (lane < tk) async_copy8(A + lane * sA + kz, g + kz * zs + lane);
    async_wait();
    __syncthreads();
    float2 *F = fft_lines<IN_LINES, OUT_LINES, false>(c3, A, B, FftEnds<float>(), tk, sA, n3);
    float2 *Fo = F == A ? B : A;
    const float wgt = (w.kx == 0 || 2 * w.kx == n1) ? 1.f : 2.f;
    // influence function exp(-pi^2 m^2 / alpha^2) / (pi V B(m) m^2): the exponential and the
    // B-spline moduli factor per dimension, so they come from a per-dimension table
    // etab[k] = exp(-pi^2 m_k^2 / (alpha^2 L^2)) / B(k) formed in FP64 (no approximate
    // exponential in the energy); m^2 = sum_d k_d^2 / L_d^2 from exact integer squares and
    // 1/L_d^2 as hi + lo, and the reciprocal of pi V m^2 to within an ulp (one Newton step on
    // the approximate reciprocal, its residual formed exactly by an FMA)
    const float pivol = R.pivolf;
    const int nf2 = (n2 + 1) / 2, nf3 = (n3 + 1) / 2;
    const float m1s = (float)(w.kx * w.kx), t1 = etab[w.kx];
    const float c2h = R.msq_c[2][0], c2l = R.msq_c[2][1];
    float en = 0.f;
    for (int c = warp; c < tk; c += 8) {
        const int ky = w.ky0 + c;
        const int m2 = ky < nf2 ? ky : ky - n2;
        const float m2s = (float)(m2 * m2);
        const float t12 = t1 * etab[n1 + ky];
        const float m12 = fmaf(m1s, R.msq_c[0][0], fmaf(m2s, R.msq_c[1][0], fmaf(m1s, R.msq_c[0][1], m2s * R.msq_c[1][1])));
        for (int kz = lane; kz < n3; kz += 32) {
            const int m3 = kz < nf3 ? kz : kz - n3;
            const float m3s = (float)(m3 * m3);
            const float msq = fmaf(m3s, c2h, fmaf(m3s, c2l, m12));
            const float den = pivol * msq;
            float rd = nb_rcp_approx(den);
            rd = fmaf(rd, fmaf(-den, rd, 1.f), rd);
            const float et = (w.kx == 0 && ky == 0 && kz == 0) ? 0.f : (t12 * etab[n1 + n2 + kz]) * rd;
            float2 v = F[c * n3 + kz];
            en += wgt * et * (v.x * v.x + v.y * v.y);
            F[c * n3 + kz] = make_float2(v.x * et, -v.y * et);    // conj: the inverse runs forward
        }
    }
    __syncthreads();
    float2 *I = fft_lines<IN_LINES, OUT_LINES, true>(c3, F, Fo, FftEnds<float>(), tk, n3, sA);
    for (int kz = warp; kz < n3; kz += 8)
        if (lane < tk) g[kz * zs + lane] = I[lane * sA + kz];
    // fixed-order reduction: each thread's few terms in FP32, then FP64 across the warp and
    // over the 8 warp sums; pivol_corr and pme_qcorr remove the FP32 rounding of pi V and of the
    // spread charges from the sum
    double ed = (double)en;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ed += __shfl_down_sync(0xffffffffu, ed, o);
    if (lane == 0) red[warp] = ed;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < 8; ++k) sum += red[k];
        e_col[blockIdx.x] = sum * (R.pivol_corr * R.pme_qcorr);
    }
}

// Reciprocal virial of the pressure analysis (ewald_receip.f:799-807, pressON): the z
// transform of k_zconv_f's columns, then per m the diagonal terms
// E(m) (1 - 2 (1 + pi^2 m^2 / alpha^2) m_a^2 / m^2) with E(m) = wgt * eterm * |S(m)|^2 as the
// energy sum forms it; three FP64 partial sums per column work item (fixed-order reduction)
__global__ void __launch_bounds__(256) k_press_zvir_f(const ColWork *__restrict__ work, const RepDev *__restrict__ reps,
                                                      const int4 *__restrict__ blob, const float *__restrict__ bsp_all,
                                                      const float2 *__restrict__ grid, double *__restrict__ v_col)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[3][8];
    const ColWork w = work[blockIdx.x];
    const RepDev &R = reps[w.rep];
    const int n1 = w.n1, n2 = w.n2, n3 = w.n3, n1h = n1 / 2 + 1;
    const int tk = w.nky;
    const float *bsp = bsp_all + w.bsp0;
    float2 *A = (float2 *)smem, *B = A + zconv_buf_elems<float>(n3);
    FftCtx<float2> c3;
    fft_ctx_load((unsigned char *)(B + zconv_buf_elems<float>(n3)), blob + w.bz, w.lz, n3, c3);
    const int sA = n3 | 1;
    const float2 *g = grid + w.g0 + (size_t)w.kx * n2 + w.ky0;
    const size_t zs = (size_t)n1h * n2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int kz = warp; kz < n3; kz += 8)
        if (lane < tk) async_copy8(A + lane * sA + kz, g + kz * zs + lane);
    async_wait();
    __syncthreads();
    const float2 *F = fft_lines<IN_LINES, OUT_LINES, false>(c3, A, B, FftEnds<float>(), tk, sA, n3);
    const float wgt = (w.kx == 0 || 2 * w.kx == n1) ? 1.f : 2.f;
    const float fac2 = R.pme_fac2f, pivol = R.pivolf, fac = (float)R.pme_fac;
    const int nf2 = (n2 + 1) / 2, nf3 = (n3 + 1) / 2;
    const float iL0 = R.invL[0], iL1 = R.invL[1], iL2 = R.invL[2];
    const float mh1 = (float)w.kx * iL0, pb1 = pivol * bsp[w.kx];
    float v0 = 0.f, v1 = 0.f, v2 = 0.f;
    for (int c = warp; c < tk; c += 8) {
        const int ky = w.ky0 + c;
        const float mh2 = (float)(ky < nf2 ? ky : ky - n2) * iL1;
        const float pb12 = pb1 * bsp[n1 + ky], m12 = mh1 * mh1 + mh2 * mh2;
        for (int kz = lane; kz < n3; kz += 32) {
            if (w.kx == 0 && ky == 0 && kz == 0) continue;
            const float mh3 = (float)(kz < nf3 ? kz : kz - n3) * iL2;
            const float msq = fmaf(mh3, mh3, m12);
            const float et = nb_ex2_approx(-fac2 * msq) * nb_rcp_approx(pb12 * bsp[n1 + n2 + kz] * msq);
            const float2 v = F[c * n3 + kz];
            const float e = wgt * et * (v.x * v.x + v.y * v.y), b = 2.f * (1.f + fac * msq) / msq;
            v0 += e * (1.f - b * mh1 * mh1);
            v1 += e * (1.f - b * mh2 * mh2);
            v2 += e * (1.f - b * mh3 * mh3);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_down_sync(0xffffffffu, v0, o);
        v1 += __shfl_down_sync(0xffffffffu, v1, o);
        v2 += __shfl_down_sync(0xffffffffu, v2, o);
    }
    if (lane == 0) { red[0][warp] = v0; red[1][warp] = v1; red[2][warp] = v2; }
    __syncthreads();
    if (threadIdx.x < 3) {
        double sum = 0.0;
        for (int k = 0; k < 8; ++k) sum += red[threadIdx.x][k];
        v_col[3 * (size_t)blockIdx.x + threadIdx.x] = sum;
    }
}

// Inverse y and x transforms of plane z: the first pass reads the grid and the last one stores the real
// rows (k_plane_fwd).  FP32: the real potential plane (n1 x n2 floats) goes over the plane's own complex storage,
// which this block alone reads, for k_pme_gather_f; FP64: the block gathers its sites' shares itself.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 2) k_plane_inv(const PlaneWork *__restrict__ work,
                                                     const int4 *__restrict__ blob,
                                                     typename cplx<T>::type *__restrict__ grid, const RepDev *__restrict__ reps, int nW,
                                                     const unsigned char *__restrict__ zidx,
                                                     const typename vec4<T>::type *__restrict__ fr,
                                                     T *__restrict__ part, int pot)
{
    typedef typename cplx<T>::type C;
    extern __shared__ __align__(16) unsigned char smem[];
    const PlaneWork w = work[blockIdx.x];
    const int n1 = w.n1, n2 = w.n2, n1h = n1 / 2 + 1, n2p = (n2 + 1) >> 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    C *B0 = (C *)smem, *B1 = B0 + plane_buf_elems(n1, n2);
    FftCtx<C> c1, c2;
    unsigned char *ctx = (unsigned char *)(B1 + plane_buf_elems(n1, n2));
    ctx = fft_ctx_load(ctx, blob + w.bx, w.lx, n1, c1);
    fft_ctx_load(ctx, blob + w.by, w.ly, n2, c2);
    C *g = grid + w.g0 + (size_t)w.z * n1h * n2;
    async_wait();
    __syncthreads();
    // y: n1h lines [kx][ky] of n2 from the grid, conjugated (inverse through the forward transform); the
    // last pass conjugates back and stores transposed to H[ky][kx] at the odd row stride hs
    const int hs = n1h | 1;
    FftEnds<T> ey, ex;
    ey.in = g;
    C *H = fft_lines<IN_CONJ, OUT_TRANSPOSED, true>(c2, B1, B0, ey, n1h, n2, hs);
    C *Zc = H == B0 ? B1 : B0;
    // x inverse of two real rows at a time: Z = H_2p + i H_2p+1 over the full Hermitian line of
    // n1, conjugated so the forward transform inverts it; row 2p = Re, row 2p+1 = -Im of the result
    for (int p = warp; p < n2p; p += nwarp)
        for (int k = lane; k < n1; k += 32) {
            const bool lo = k < n1h;
            const int kk = lo ? k : n1 - k;
            C a = H[2 * p * hs + kk], b;
            b.x = b.y = (T)0;
            if (2 * p + 1 < n2) b = H[(2 * p + 1) * hs + kk];
            if (!lo) { a = cconj(a); b = cconj(b); }
            C z;
            z.x = a.x - b.y; z.y = -(a.y + b.x);
            Zc[p * n1 + k] = z;
        }
    __syncthreads();
    ex.rows = n2;
    if constexpr (sizeof(T) == 4) {
        // the real potential plane over the plane's own complex storage (this block alone reads it)
        ex.real = (T *)g;
        fft_lines<IN_LINES, OUT_ROWS, false>(c1, Zc, H, ex, n2p, n1, n1);
    } else {
        // the real plane in the buffer that the last pass does not read, the other one for the queue
        C *rows = (c1.p->nst & 1) ? H : Zc, *queue = rows == H ? Zc : H;
        ex.real = (T *)rows;
        fft_lines<IN_LINES, OUT_ROWS, false>(c1, Zc, H, ex, n2p, n1, n1);
        plane_sites(reps[w.rep], nW, w.z, zidx, (int *)queue, (int)(sizeof(C) / 4) * plane_buf_elems(n1, n2), [&](int n) {
            gather_sites<T>(reps[w.rep], (const int *)queue, n, fr, (const T *)rows, part, pot != 0);
        });
    }
}

// PME gradient of each site from the real potential grid (grad_sum,
// ewald_receip.f:815-970): order-4 weights and derivatives once per site, the 4x4x4 stencil
// read from the grid planes k_plane_inv left in place; result (x, y, z) per site, to be
// scaled by q * fc * n_d / L_d in the finalize.  LPS lanes per site, a share of the stencil's planes
// each (their sums are added in plane order, so the result does not depend on LPS).  Bound: latency
// of the 16 row loads while the sites do not fill the GPU, the issue of the stencil arithmetic
// beyond.
template <int LPS>
__global__ void __launch_bounds__(256, 4) k_pme_gather_f(int nsite, const int *__restrict__ site_rep,
                                                      const RepDev *__restrict__ reps, const float4 *__restrict__ fr,
                                                      const float2 *__restrict__ grid, float4 *__restrict__ part)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x, sub = idx & (LPS - 1);
    const int s = idx / LPS;
    if (s >= nsite) return;
    const float4 f = fr[s];
    if (f.w == 0.f) { if (sub == 0) part[s] = make_float4(0.f, 0.f, 0.f, 0.f); return; }
    const RepDev &R = reps[site_rep[s]];
    const int n1 = R.n1, n2 = R.n2, n3 = R.n3;
    const size_t zs = (size_t)R.n1h * n2 * 2;    // floats per plane
    const float *Q = (const float *)(grid + R.g0);
    int i1, i2, i3;
    float w1, w2, w3;
    pme_fr_split(f.x, i1, w1);
    pme_fr_split(f.y, i2, w2);
    pme_fr_split(f.z, i3, w3);
    float th1[4], dt1[4], th2[4], dt2[4], th3[4], dt3[4];
    bsp4_th<float>(w1, th1); bsp4_dth<float>(w1, dt1);
    bsp4_th<float>(w2, th2); bsp4_dth<float>(w2, dt2);
    bsp4_th<float>(w3, th3); bsp4_dth<float>(w3, dt3);
    int xs[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) xs[t] = pme_wrap(i1 - 3 + t, n1);
    // without an x wrap the four stencil points of a row are contiguous: two aligned float4
    // loads hold them, one when they start 16-byte aligned (the grid allocation ends 16 bytes
    // past its last plane for the second).
    // fr1 can round to n1 itself (index n1 wraps to 0), which takes the wrapped path.
    const bool contig = i1 >= 3 && i1 < n1;
    float gx = 0.f, gy = 0.f, gz = 0.f, h3[4 / LPS][3];
#pragma unroll
    for (int u = 0; u < 4 / LPS; ++u) {
        const int t3 = sub * (4 / LPS) + u;
        const float *P = Q + pme_wrap(i3 - 3 + t3, n3) * zs;
        float hx = 0.f, hy = 0.f, hz = 0.f;
#pragma unroll
        for (int t2 = 0; t2 < 4; ++t2) {
            const float *row = P + pme_wrap(i2 - 3 + t2, n2) * n1;
            float q4[4];
            if (contig) {
                const uintptr_t a = (uintptr_t)(row + i1 - 3);
                const float4 *p4 = (const float4 *)(a & ~(uintptr_t)15);
                const int sh = (int)((a >> 2) & 3);
                const float4 c0 = __ldg(p4);
                const float4 c1 = sh != 0 ? __ldg(p4 + 1) : c0;     // an aligned row needs one load
                q4[0] = sh == 0 ? c0.x : (sh == 1 ? c0.y : (sh == 2 ? c0.z : c0.w));
                q4[1] = sh == 0 ? c0.y : (sh == 1 ? c0.z : (sh == 2 ? c0.w : c1.x));
                q4[2] = sh == 0 ? c0.z : (sh == 1 ? c0.w : (sh == 2 ? c1.x : c1.y));
                q4[3] = sh == 0 ? c0.w : (sh == 1 ? c1.x : (sh == 2 ? c1.y : c1.z));
            } else {
#pragma unroll
                for (int t1 = 0; t1 < 4; ++t1) q4[t1] = row[xs[t1]];
            }
            float sx = 0.f, sy = 0.f;
#pragma unroll
            for (int t1 = 0; t1 < 4; ++t1) {
                const float q = q4[t1];
                sx = fmaf(q, dt1[t1], sx);
                sy = fmaf(q, th1[t1], sy);
            }
            hx = fmaf(sx, th2[t2], hx);
            hy = fmaf(sy, dt2[t2], hy);
            hz = fmaf(sy, th2[t2], hz);
        }
        h3[u][0] = hx; h3[u][1] = hy; h3[u][2] = hz;
    }
    // (the site's lanes are here together: they left together or not at all)
    const unsigned mates = LPS == 1 ? 0u : ((1u << LPS) - 1u) << ((threadIdx.x & 31) & ~(LPS - 1));
#pragma unroll
    for (int t3 = 0; t3 < 4; ++t3) {
        float h[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            h[d] = LPS == 1 ? h3[t3 % (4 / LPS)][d] : __shfl_sync(mates, h3[t3 % (4 / LPS)][d], t3 / (4 / LPS), LPS);
        gx = fmaf(h[0], th3[t3], gx);
        gy = fmaf(h[1], th3[t3], gy);
        gz = fmaf(h[2], dt3[t3], gz);
    }
    if (sub == 0) part[s] = make_float4(gx, gy, gz, 0.f);
}

// =================================================================================
// FP64 (plain) path: the same planes and passes in FP64; the influence function with its exponential
// and division per point, in FP64.  One warp per line with a butterfly per lane used 5 lanes in 32 of
// the FP64 pipe for lines of 20: PME stages of 216 waters 131 us, 1,334 waters 211; shared by the block,
// two real rows per x transform, 62 and 109.
__global__ void __launch_bounds__(256) k_zconv_d(const ColWork *__restrict__ work, const RepDev *__restrict__ reps,
                                                 const int4 *__restrict__ blob, const double *__restrict__ bsp_all,
                                                 double2 *__restrict__ grid, double *__restrict__ e_col)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[256];
    const ColWork w = work[blockIdx.x];
    const RepDev &R = reps[w.rep];
    const int n1 = w.n1, n2 = w.n2, n3 = w.n3, n1h = n1 / 2 + 1, tk = w.nky;
    const double *bsp = bsp_all + w.bsp0;
    double2 *A = (double2 *)smem, *B = A + zconv_buf_elems<double>(n3);
    FftCtx<double2> c3;
    fft_ctx_load((unsigned char *)(B + zconv_buf_elems<double>(n3)), blob + w.bz, w.lz, n3, c3);
    const int sA = n3 | 1;
    double2 *g = grid + w.g0 + (size_t)w.kx * n2 + w.ky0;
    const size_t zs = (size_t)n1h * n2;
    for (int idx = threadIdx.x; idx < tk * n3; idx += blockDim.x) {
        const int kz = idx / tk, c = idx - kz * tk;
        A[c * sA + kz] = g[kz * zs + c];
    }
    async_wait();
    __syncthreads();
    double2 *F = fft_lines<IN_LINES, OUT_LINES, false>(c3, A, B, FftEnds<double>(), tk, sA, n3);
    double2 *Fo = F == A ? B : A;
    const double wgt = (w.kx == 0 || 2 * w.kx == n1) ? 1.0 : 2.0;
    double en = 0.0;
    for (int idx = threadIdx.x; idx < tk * n3; idx += blockDim.x) {
        const int c = idx / n3, kz = idx - c * n3;
        const double et = eterm_of<double>(R, bsp, w.kx, w.ky0 + c, kz);
        const double2 v = F[idx];
        en += wgt * et * (v.x * v.x + v.y * v.y);
        F[idx] = make_double2(v.x * et, -v.y * et);      // conj: the inverse runs forward
    }
    __syncthreads();
    double2 *I = fft_lines<IN_LINES, OUT_LINES, true>(c3, F, Fo, FftEnds<double>(), tk, n3, sA);
    for (int idx = threadIdx.x; idx < tk * n3; idx += blockDim.x) {
        const int kz = idx / tk, c = idx - kz * tk;
        g[kz * zs + c] = I[c * sA + kz];
    }
    red[threadIdx.x] = en;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) e_col[blockIdx.x] = red[0];
}

// reciprocal virial of the pressure analysis on the plain path: the z transform of k_zconv_d's
// columns, then per m the diagonal terms
// E(m) (1 - 2 (1 + pi^2 m^2 / alpha^2) m_a^2 / m^2) (ewald_receip.f:799-807), E(m) as the
// energy sum forms it; three FP64 sums per column work item
__global__ void __launch_bounds__(256) k_press_zvir_d(const ColWork *__restrict__ work, const RepDev *__restrict__ reps,
                                                      const int4 *__restrict__ blob, const double *__restrict__ bsp_all,
                                                      const double2 *__restrict__ grid, double *__restrict__ v_col)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[3][256];
    const ColWork w = work[blockIdx.x];
    const RepDev &R = reps[w.rep];
    const int n1 = w.n1, n2 = w.n2, n3 = w.n3, n1h = n1 / 2 + 1, tk = w.nky;
    const double *bsp = bsp_all + w.bsp0;
    double2 *A = (double2 *)smem, *B = A + zconv_buf_elems<double>(n3);
    FftCtx<double2> c3;
    fft_ctx_load((unsigned char *)(B + zconv_buf_elems<double>(n3)), blob + w.bz, w.lz, n3, c3);
    const int sA = n3 | 1;
    const double2 *g = grid + w.g0 + (size_t)w.kx * n2 + w.ky0;
    const size_t zs = (size_t)n1h * n2;
    for (int idx = threadIdx.x; idx < tk * n3; idx += blockDim.x) {
        const int kz = idx / tk, c = idx - kz * tk;
        A[c * sA + kz] = g[kz * zs + c];
    }
    async_wait();
    __syncthreads();
    const double2 *F = fft_lines<IN_LINES, OUT_LINES, false>(c3, A, B, FftEnds<double>(), tk, sA, n3);
    double v[3] = {0.0, 0.0, 0.0};
    const double wgt = (w.kx == 0 || (2 * w.kx == n1)) ? 1.0 : 2.0;
    const int nf2 = (n2 + 1) / 2, nf3 = (n3 + 1) / 2;
    for (int idx = threadIdx.x; idx < tk * n3; idx += blockDim.x) {
        const int c = idx / n3, kz = idx - c * n3, ky = w.ky0 + c;
        if (w.kx == 0 && ky == 0 && kz == 0) continue;
        const double mh[3] = {(double)w.kx * R.invLd[0], (double)(ky < nf2 ? ky : ky - n2) * R.invLd[1],
                              (double)(kz < nf3 ? kz : kz - n3) * R.invLd[2]};
        const double msq = mh[0] * mh[0] + mh[1] * mh[1] + mh[2] * mh[2];
        const double et = eterm_of<double>(R, bsp, w.kx, ky, kz);
        const double2 q = F[idx];
        const double e = wgt * et * (q.x * q.x + q.y * q.y), b = 2.0 * (1.0 + R.pme_fac * msq) / msq;
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] += e * (1.0 - b * mh[d] * mh[d]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) red[d][threadIdx.x] = v[d];
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
#pragma unroll
            for (int d = 0; d < 3; ++d) red[d][threadIdx.x] += red[d][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x < 3) v_col[3 * (size_t)blockIdx.x + threadIdx.x] = red[threadIdx.x][0];
}

template <typename T>
void pme_t(NbCtx *c)
{
    cudaStream_t s = c->stream;
    if (c->timing) cudaEventRecord(c->ev[6], s);
    if (c->d_pos && !nb_fused_sites(c)) {
        k_pme_sites<T><<<(int)((c->nsite + 255) / 256), 256, 0, s>>>((int)c->nsite, c->d_site_rep, c->d_reps, c->d_pos,
                                                                    c->d_site_q, c->d_fr, c->d_zidx);
        c->launches++;
    }
    typedef typename cplx<T>::type C;
    typedef typename vec4<T>::type T4;
    const int np = (int)c->planes.size(), nc = (int)c->cols.size();
    k_plane_fwd<T><<<np, 256, c->smem_plane, s>>>(c->d_planes, c->d_reps, c->d_blob, (int)c->nW, c->d_zidx,
                                                      (const T4 *)c->d_fr, (C *)c->d_grid);
    if (c->timing) cudaEventRecord(c->ev[7], s);
    if constexpr (sizeof(T) == 4)
        k_zconv_f<<<nc, 256, c->smem_zconv, s>>>(c->d_cols, c->d_reps, c->d_blob, c->d_etab, (float2 *)c->d_grid,
                                                 c->d_e_col);
    else
        k_zconv_d<<<nc, 256, c->smem_zconv, s>>>(c->d_cols, c->d_reps, c->d_blob, (const double *)c->d_bsp,
                                                 (double2 *)c->d_grid, c->d_e_col);
    if (c->timing) cudaEventRecord(c->ev[8], s);
    k_plane_inv<T><<<np, 256, c->smem_plane, s>>>(c->d_planes, c->d_blob, (C *)c->d_grid, c->d_reps, (int)c->nW,
                                                      c->d_zidx, (const T4 *)c->d_fr, (T *)c->d_part, 0);
    if constexpr (sizeof(T) == 4) {
        // four lanes per site while they all fit the GPU at once (an evaluation of 216 waters 50.7 / 47.2 us
        // with 1 / 4, 460 waters and 203 atoms 65.0 / 61.1, 42,000 waters 148 / 148, 229,000 558 / 576)
        const int lps = c->nsite <= 40000 ? 4 : 1;
        (lps == 4 ? k_pme_gather_f<4> : k_pme_gather_f<1>)<<<(int)((c->nsite * lps + 255) / 256), 256, 0, s>>>(
            (int)c->nsite, c->d_site_rep, c->d_reps, (const float4 *)c->d_fr, (const float2 *)c->d_grid,
            (float4 *)c->d_part);
        c->launches++;
    }
    if (c->timing) cudaEventRecord(c->ev[9], s);
    c->launches += 3;
}

// radix plan and Stockham tables; returns 0 if n is not 2/3/5-smooth or too long.  Radices 2 to 10,
// the fewest passes (a line of up to 100 points in two), the most even split on ties.  tab receives
// (twiddle step, destination index) per butterfly.
// fewest factors of m from the wide radix set, at most `left` of them, and of those the smallest sum
// (the most even split: the longest butterfly sets the time of a pass); its count, -1 if none
int wide_factors(int m, int left, int *out)
{
    static const int R[8] = {10, 9, 8, 6, 5, 4, 3, 2};
    if (m == 1) return 0;
    if (left == 0) return -1;
    int best = -1, sum = 0, tmp[8];
    for (int k = 0; k < 8; ++k) {
        if (m % R[k]) continue;
        const int f = wide_factors(m / R[k], best < 0 ? left - 1 : best - 1, tmp);
        if (f < 0) continue;
        int s = R[k];
        for (int q = 0; q < f; ++q) s += tmp[q];
        if (best >= 0 && f + 1 == best && s >= sum) continue;
        best = f + 1;
        sum = s;
        out[0] = R[k];
        for (int q = 0; q < f; ++q) out[1 + q] = tmp[q];
    }
    return best;
}

int make_plan(int n, FftPlanDev *p, std::vector<int2> *tab)
{
    memset(p, 0, sizeof(*p));
    p->n = n;
    if (n < 2 || n > NB_MAX_FFT) return 0;
    const int k = wide_factors(n, 8, p->rad);
    if (k < 0) return 0;
    p->nst = k;
    int Ns = 1, off = 0;
    for (int s = 0; s < k; ++s) {
        int R = p->rad[s], nb = n / R, stride = n / (Ns * R);
        p->ns[s] = Ns;
        p->nb[s] = nb;
        p->off[s] = off;
        p->magic[s] = nb > 1 ? 0xFFFFFFFFu / (unsigned)nb + 1u : 0u;
        if (tab) {
            for (int j = 0; j < nb; ++j) {
                int jm = j % Ns;
                tab->push_back(make_int2(jm * stride, (j / Ns) * Ns * R + jm));
            }
        }
        off += nb;
        Ns *= R;
    }
    return 1;
}

size_t fft_ctx_bytes(int n, size_t elem)
{
    FftPlanDev p;
    if (!make_plan(n, &p, nullptr)) return 0;
    size_t ntab = (size_t)p.off[p.nst - 1] + p.nb[p.nst - 1];
    return align16(sizeof(FftPlanDev)) + align16(ntab * sizeof(int2)) + align16(n * elem);
}

template <typename T>
size_t plane_smem(int n1, int n2)
{
    const size_t e = sizeof(typename cplx<T>::type);
    return 2 * e * plane_buf_elems(n1, n2) + fft_ctx_bytes(n1, e) + fft_ctx_bytes(n2, e);
}
template <typename T>
size_t zconv_smem(int n3)
{
    const size_t e = sizeof(typename cplx<T>::type);
    return 2 * e * zconv_buf_elems<T>(n3) + fft_ctx_bytes(n3, e);
}
// the z-column work items of one kx: the n2 columns in ceil(n2 / tile) runs of equal length
// (within one), so no block of the column kernels works on a short remainder alone (n2 = 36
// gives two runs of 18, not 32 and 4: every Stockham pass of a run then fits one sweep of the
// block's threads)
void push_col_runs(std::vector<ColWork> &cols, ColWork w, int tile)
{
    const int n2 = w.n2;
    const int nrun = (n2 + tile - 1) / tile, base = n2 / nrun, extra = n2 % nrun;
    int ky0 = 0;
    for (int k = 0; k < nrun; ++k) {
        const int len = base + (k < extra ? 1 : 0);
        w.ky0 = ky0;
        w.nky = len;
        cols.push_back(w);
        ky0 += len;
    }
}

// one plan's tables as the kernels stage them (fft_ctx_load), appended to blob; its offset and
// length in 16-byte units
template <typename C>
void push_blob(std::vector<int4> &blob, const FftPlanDev &p, const std::vector<int2> &tab, const std::vector<C> &tw,
               int *off, int *len)
{
    const size_t b0 = align16(sizeof(FftPlanDev)), b1 = b0 + align16(p.n * sizeof(C)),
                 b2 = b1 + align16(tab.size() * sizeof(int2));
    *off = (int)blob.size();
    *len = (int)(b2 / 16);
    blob.resize(blob.size() + b2 / 16);
    unsigned char *d = (unsigned char *)(blob.data() + *off);
    memset(d, 0, b2);
    memcpy(d, &p, sizeof(p));
    memcpy(d + b0, tw.data(), p.n * sizeof(C));
    memcpy(d + b1, tab.data(), tab.size() * sizeof(int2));
}

// raise a kernel's dynamic shared-memory limit to at least `bytes` (never lower it)
template <typename K>
cudaError_t raise_smem_limit(K *kernel, size_t bytes)
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    if ((size_t)fa.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T>
cudaError_t raise_pme_limits(size_t sp, size_t sz)
{
    cudaError_t e;
    if ((e = raise_smem_limit(k_plane_fwd<T>, sp)) != cudaSuccess) return e;
    if ((e = raise_smem_limit(k_plane_inv<T>, sp)) != cudaSuccess) return e;
    if constexpr (sizeof(T) == 4) {
        if ((e = raise_smem_limit(k_zconv_f, sz)) != cudaSuccess) return e;
        return raise_smem_limit(k_press_zvir_f, sz);
    } else {
        if ((e = raise_smem_limit(k_zconv_d, sz)) != cudaSuccess) return e;
        return raise_smem_limit(k_press_zvir_d, sz);
    }
}

template <typename T>
int configure_t(NbCtx *c)
{
    typedef typename cplx<T>::type C;
    // plans by length: tables laid out as the kernels stage them
    std::vector<int> plan_n, boff, blen, rep_plan(3 * c->nrep, 0);
    std::vector<int4> blob;
    for (int r = 0; r < c->nrep; ++r) {
        int ns[3] = {c->rd[r].n1, c->rd[r].n2, c->rd[r].n3};
        for (int d = 0; d < 3; ++d) {
            int found = -1;
            for (size_t k = 0; k < plan_n.size(); ++k)
                if (plan_n[k] == ns[d]) found = (int)k;
            if (found < 0) {
                FftPlanDev p;
                std::vector<int2> tab;
                std::vector<C> tw(std::max(ns[d], 0));
                if (!make_plan(ns[d], &p, &tab)) return MOIL_NB_ERR_GRID;
                for (int t = 0; t < ns[d]; ++t) {
                    double ang = -2.0 * M_PI * (double)t / (double)ns[d];
                    tw[t].x = (T)cos(ang);
                    tw[t].y = (T)sin(ang);
                }
                boff.push_back(0);
                blen.push_back(0);
                push_blob(blob, p, tab, tw, &boff.back(), &blen.back());
                plan_n.push_back(ns[d]);
                found = (int)plan_n.size() - 1;
            }
            rep_plan[3 * r + d] = found;
        }
    }
    NB_CUDA_OK(c, cudaMalloc(&c->d_blob, sizeof(int4) * blob.size()));
    NB_CUDA_OK(c, cudaMemcpy(c->d_blob, blob.data(), sizeof(int4) * blob.size(), cudaMemcpyHostToDevice));
    std::vector<T> bsp(c->bsp_h.size());
    for (size_t k = 0; k < bsp.size(); ++k) bsp[k] = (T)c->bsp_h[k];
    NB_CUDA_OK(c, cudaMalloc(&c->d_bsp, sizeof(T) * bsp.size()));
    NB_CUDA_OK(c, cudaMemcpy(c->d_bsp, bsp.data(), sizeof(T) * bsp.size(), cudaMemcpyHostToDevice));
    if (sizeof(T) == 4) {
        std::vector<float> et(c->bsp_h.size());
        for (int r = 0; r < c->nrep; ++r) {
            const RepDev &R = c->rd[r];
            nb_pme_etab(R, c->bsp_h.data() + R.bsp0, et.data() + R.bsp0);
        }
        NB_CUDA_OK(c, cudaMalloc(&c->d_etab, sizeof(float) * et.size()));
        NB_CUDA_OK(c, cudaMemcpy(c->d_etab, et.data(), sizeof(float) * et.size(), cudaMemcpyHostToDevice));
    }
    // work lists: planes (replica, z) and z columns (replica, kx, ky run)
    c->planes.clear();
    c->cols.clear();
    c->col_begin.assign(c->nrep + 1, 0);
    size_t sp = 0, sz = 0;
    const int tk = col_tile<T>();
    for (int r = 0; r < c->nrep; ++r) {
        const RepDev &R = c->rd[r];
        const int *pl = &rep_plan[3 * r];
        for (int z = 0; z < R.n3; ++z)
            c->planes.push_back(PlaneWork{r, z, R.n1, R.n2, boff[pl[0]], blen[pl[0]], boff[pl[1]], blen[pl[1]], R.g0});
        c->col_begin[r] = (int)c->cols.size();
        for (int kx = 0; kx < R.n1h; ++kx)
            push_col_runs(c->cols, ColWork{r, kx, 0, 0, R.n1, R.n2, R.n3, R.bsp0, boff[pl[2]], blen[pl[2]], R.g0}, tk);
        sp = std::max(sp, plane_smem<T>(R.n1, R.n2));
        sz = std::max(sz, zconv_smem<T>(R.n3));
    }
    c->col_begin[c->nrep] = (int)c->cols.size();
    int dev_smem = 0;
    cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    if ((int)sp > dev_smem || (int)sz > dev_smem) {
        c->err = "PME grid plane does not fit in shared memory";
        return MOIL_NB_ERR_GRID;
    }
    c->smem_plane = sp;
    c->smem_zconv = sz;
    // the limit is per kernel, shared by every handle in the process: only ever raise it
    NB_CUDA_OK(c, raise_pme_limits<T>(sp, sz));
    NB_CUDA_OK(c, cudaMalloc(&c->d_planes, sizeof(PlaneWork) * c->planes.size()));
    NB_CUDA_OK(c, cudaMemcpy(c->d_planes, c->planes.data(), sizeof(PlaneWork) * c->planes.size(), cudaMemcpyHostToDevice));
    NB_CUDA_OK(c, cudaMalloc(&c->d_cols, sizeof(ColWork) * c->cols.size()));
    NB_CUDA_OK(c, cudaMemcpy(c->d_cols, c->cols.data(), sizeof(ColWork) * c->cols.size(), cudaMemcpyHostToDevice));
    NB_CUDA_OK(c, cudaMalloc(&c->d_col_begin, sizeof(int) * (c->nrep + 1)));
    NB_CUDA_OK(c, cudaMemcpy(c->d_col_begin, c->col_begin.data(), sizeof(int) * (c->nrep + 1), cudaMemcpyHostToDevice));
    NB_CUDA_OK(c, cudaMalloc(&c->d_e_col, sizeof(double) * c->cols.size()));
    // two spare elements: the FP32 gather's second aligned float4 of a row may reach 16 bytes
    // past the last plane
    NB_CUDA_OK(c, cudaMalloc(&c->d_grid, sizeof(C) * (c->grid_elems + 2)));
    NB_CUDA_OK(c, cudaMalloc(&c->d_fr, sizeof(typename vec4<T>::type) * c->nsite));
    NB_CUDA_OK(c, cudaMalloc(&c->d_part, sizeof(T) * 12 * c->nsite));
    NB_CUDA_OK(c, cudaMemset(c->d_part, 0, sizeof(T) * 12 * c->nsite));
    return MOIL_NB_OK;
}

}  // namespace

void nb_launch_pme(NbCtx *c)
{
    if (c->precision == MOIL_NB_FP64) pme_t<double>(c);
    else pme_t<float>(c);
}

// pressure analysis: the charge planes of the evaluation's sites spread and transformed
// again into grid (a copy beside the handle's own grid, whose potential planes stay valid),
// and the reciprocal virial per column work item into v_col (mixed path)
void nb_launch_pme_virial(NbCtx *c, cudaStream_t s, void *grid, double *v_col)
{
    const int np = (int)c->planes.size(), nc = (int)c->cols.size();
    if (c->precision == MOIL_NB_FP64) {
        k_plane_fwd<double><<<np, 256, c->smem_plane, s>>>(c->d_planes, c->d_reps, c->d_blob, (int)c->nW, c->d_zidx,
                                                               (const double4 *)c->d_fr, (double2 *)grid);
        k_press_zvir_d<<<nc, 256, c->smem_zconv, s>>>(c->d_cols, c->d_reps, c->d_blob, (const double *)c->d_bsp,
                                                      (const double2 *)grid, v_col);
        return;
    }
    k_plane_fwd<float><<<np, 256, c->smem_plane, s>>>(c->d_planes, c->d_reps, c->d_blob, (int)c->nW, c->d_zidx,
                                                          (const float4 *)c->d_fr, (float2 *)grid);
    k_press_zvir_f<<<nc, 256, c->smem_zconv, s>>>(c->d_cols, c->d_reps, c->d_blob, (const float *)c->d_bsp,
                                                  (const float2 *)grid, v_col);
}

// parameter derivatives on the plain path: the potential share of every plane at each site
// (4 slots per site) from the convolved grid the evaluation left in place
void nb_launch_pme_potential(NbCtx *c, double *phi4)
{
    k_plane_inv<double><<<(int)c->planes.size(), 256, c->smem_plane, c->stream>>>(
        c->d_planes, c->d_blob, (double2 *)c->d_grid, c->d_reps, (int)c->nW, c->d_zidx, (const double4 *)c->d_fr, phi4,
        1);
}

int nb_pme_configure(NbCtx *c)
{
    return c->precision == MOIL_NB_FP64 ? configure_t<double>(c) : configure_t<float>(c);
}

void nb_spread_scale(double qfc_max, RepDev *R)
{
    const int k = nb_spread_exp(qfc_max);
    R->spread_scale = (float)ldexp(1.0, k);
    R->spread_inv = (float)ldexp(1.0, -k);
    const double s216 = ldexp(1.0, k) / 216.0;
    R->spread216 = (float)s216;
    R->spread216_corr = s216 / (double)R->spread216;
}

void nb_pme_etab(const RepDev &R, const double *bsp, float *out)
{
    const int ns[3] = {R.n1, R.n2, R.n3};
    for (int d = 0, o = 0; d < 3; o += ns[d], ++d)
        for (int k = 0; k < ns[d]; ++k) {
            // MOIL's m folding (pot/ewald_receip.f:723-812): k > ceil(n/2) - 1 -> k - n
            const int m = k < (ns[d] + 1) / 2 ? k : k - ns[d];
            const double mh = m * R.invLd[d];
            out[o + k] = (float)(exp(-R.pme_fac * mh * mh) / bsp[o + k]);
        }
}

void nb_pme_fp32_consts(RepDev *R)
{
    const double fac2 = R->pme_fac * 1.4426950408889634;
    R->pme_fac2f = (float)fac2;
    R->fac2_lo = (float)(fac2 - (double)R->pme_fac2f);
    R->pivolf = (float)R->pivol;
    R->pivol_corr = (double)R->pivolf / R->pivol;
    for (int d = 0; d < 3; ++d) R->invL_lo[d] = (float)(R->invLd[d] - (double)R->invL[d]);
    for (int d = 0; d < 3; ++d) {
        const double c = R->invLd[d] * R->invLd[d];
        R->msq_c[d][0] = (float)c;
        R->msq_c[d][1] = (float)(c - (double)R->msq_c[d][0]);
    }
}

// ---------------------------------------------------------------------------------
// Allocation-free PME reciprocal sum (moil_nb_pme_noalloc).
//
// For callers that cannot allocate device memory: the same spread+FFT / convolution /
// FFT+gather kernels as the handle path (FP32), with every scratch buffer carved out of one
// file-scope device array.  The array is sized for at most NA_MAX_ATOMS atoms and PME
// grids of at most NA_MAX_N points per side; every GPU that loads this library holds it
// (about 5.6 MB) until the process exits.

namespace {

constexpr int NA_MAX_ATOMS = 65536;
constexpr int NA_MAX_N = 64;
constexpr int NA_MAX_COLS = (NA_MAX_N / 2 + 1) * ((NA_MAX_N + NB_TKF - 1) / NB_TKF);
struct alignas(16) NaParams {
    RepDev R;
    unsigned long long qmax;     // largest |charge| (bits of a non-negative double order as integers)
    unsigned done;               // blocks of k_na_load that have finished
};
constexpr size_t na_up(size_t x) { return (x + 255) & ~(size_t)255; }

// arena regions (byte offsets, 256-byte aligned)
constexpr size_t NA_REP = 0;
constexpr size_t NA_FR = NA_REP + na_up(sizeof(int) * NA_MAX_ATOMS);
constexpr size_t NA_ZIDX = NA_FR + na_up(sizeof(float4) * NA_MAX_ATOMS);
constexpr size_t NA_PART = NA_ZIDX + na_up(NA_MAX_ATOMS + 16);
constexpr size_t NA_GRID = NA_PART + na_up(sizeof(float) * 12 * NA_MAX_ATOMS);
constexpr size_t NA_ECOL = NA_GRID + na_up(sizeof(float2) * ((NA_MAX_N / 2 + 1) * NA_MAX_N * NA_MAX_N + 2));
constexpr size_t NA_ETAB = NA_ECOL + na_up(sizeof(double) * NA_MAX_COLS);
constexpr size_t NA_EOUT = NA_ETAB + na_up(sizeof(float) * 3 * NA_MAX_N);
// what the host lays out, one copy per call: constants (with the charge maximum and the block count
// of k_na_load, zero), planes, columns, tables
constexpr size_t NA_HOST = NA_EOUT + na_up(sizeof(double));
constexpr size_t NA_PLANES = sizeof(NaParams);
constexpr size_t NA_COLS = NA_PLANES + sizeof(PlaneWork) * NA_MAX_N;
constexpr size_t NA_BLOB = NA_COLS + sizeof(ColWork) * NA_MAX_COLS;
constexpr size_t NA_HOST_BYTES = NA_BLOB + 3 * (512 + sizeof(float2) * NA_MAX_N + sizeof(int2) * 8 * NA_MAX_N);
static_assert(sizeof(FftPlanDev) + 32 <= 512, "room of a plan in the tables");
constexpr size_t NA_BYTES = NA_HOST + na_up(NA_HOST_BYTES);

static __device__ __align__(256) unsigned char g_pme_scratch[NA_BYTES];

std::mutex g_na_mu;
constexpr int NA_MAX_DEVICES = 64;
unsigned char *g_na_base[NA_MAX_DEVICES] = {};

// Records of the atoms, and beside them the spread scale from the largest charge (same rule as the
// handle path), set by the last block to finish, and the influence function's tables (last
// block; order-4 B-spline moduli |1/6 + 2/3 w + 1/6 w^2|^2 = (2/3 + cos(2 pi k / n) / 3)^2,
// ewald_receip.f:413-481).  The charge maximum in a block of its own took 49 us for 23,556 atoms, and
// the moduli on the host 100.
__global__ void __launch_bounds__(256) k_na_load(int natom, NaParams *__restrict__ P, const double *__restrict__ coor,
                                                 const double *__restrict__ q, float4 *__restrict__ fr,
                                                 unsigned char *__restrict__ zidx, int *__restrict__ srep,
                                                 float *__restrict__ etab)
{
    __shared__ unsigned long long smax;
    RepDev &R = P->R;
    if (threadIdx.x == 0) smax = 0ull;
    __syncthreads();
    if (blockIdx.x == gridDim.x - 1) {
        const int n[3] = {R.n1, R.n2, R.n3};
        for (int t = threadIdx.x; t < n[0] + n[1] + n[2]; t += blockDim.x) {
            const int d = t < n[0] ? 0 : (t < n[0] + n[1] ? 1 : 2), k = t - (d > 0 ? n[0] : 0) - (d > 1 ? n[1] : 0);
            const int nd = d == 0 ? n[0] : (d == 1 ? n[1] : n[2]);
            const int m = k < (nd + 1) / 2 ? k : k - nd;
            const double b = 2.0 / 3.0 + cospi(2.0 * k / nd) / 3.0, mh = m * R.invLd[d];
            etab[t] = (float)(exp(-R.pme_fac * mh * mh) / (b * b));
        }
    } else {
        const int a = blockIdx.x * blockDim.x + threadIdx.x;
        double qa = 0.0;
        if (a < natom) {
            qa = q[a];
            const float x[3] = {(float)coor[3 * (size_t)a], (float)coor[3 * (size_t)a + 1], (float)coor[3 * (size_t)a + 2]};
            fr[a] = pme_site(R, x, (float)qa, zidx[a]);
            srep[a] = 0;
        }
        // (a NaN charge is left out, as fmax leaves it out)
        atomicMax(&smax, qa == qa ? (unsigned long long)__double_as_longlong(fabs(qa)) : 0ull);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&P->qmax, smax);
        __threadfence();
        if (atomicAdd(&P->done, 1u) == gridDim.x - 1) {
            const double m = __longlong_as_double((long long)atomicMax(&P->qmax, 0ull));
            const int k = nb_spread_exp(m * R.fcd);
            R.spread_scale = (float)ldexp(1.0, k);
            R.spread_inv = (float)ldexp(1.0, -k);
            const double s216 = ldexp(1.0, k) / 216.0;
            R.spread216 = (float)s216;
            const double c = s216 / (double)R.spread216;
            R.pme_qcorr = c * c;
        }
    }
}

// gradient (grad_sum, pot/ewald_receip.f:815-970), overwriting dpot, and in the last block the energy
__global__ void __launch_bounds__(256) k_na_grad(int natom, const RepDev *__restrict__ reps, const double *__restrict__ q,
                                                 const float *__restrict__ part, double *__restrict__ dpot, int ncol,
                                                 const double *__restrict__ e_col, double *__restrict__ out)
{
    __shared__ double sh[256];
    if (blockIdx.x == gridDim.x - 1) {
        double v = 0;
        for (int w = threadIdx.x; w < ncol; w += blockDim.x) v += e_col[w];
        sh[threadIdx.x] = v;
        __syncthreads();
        for (int o = blockDim.x / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) *out = 0.5 * sh[0];
        return;
    }
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= natom) return;
    const RepDev &R = reps[0];
    const float4 p = ((const float4 *)part)[a];   // k_pme_gather_f: one (x, y, z) per atom
    const double pg[3] = {(double)p.x, (double)p.y, (double)p.z};
    double qf = q[a] * R.fcd;
    dpot[3 * (size_t)a] = qf * R.n1 * R.invLd[0] * pg[0];
    dpot[3 * (size_t)a + 1] = qf * R.n2 * R.invLd[1] * pg[1];
    dpot[3 * (size_t)a + 2] = qf * R.n3 * R.invLd[2] * pg[2];
}

}  // namespace

extern "C" int moil_nb_pme_noalloc(const double *d_coor, const double *d_q, int natom, const double *box,
                                   const int *grid, double alpha, double eps, double *d_dpot, double *e_recip,
                                   void *stream_v)
{
    if (!d_coor || !d_q || !box || !grid || !d_dpot || !e_recip) return MOIL_NB_ERR_ARG;
    if (natom < 1 || natom > NA_MAX_ATOMS || !(alpha > 0) || !(eps > 0)) return MOIL_NB_ERR_ARG;
    for (int d = 0; d < 3; ++d) {
        FftPlanDev p;
        if (!(box[d] > 0) || grid[d] < 4 || grid[d] > NA_MAX_N || !make_plan(grid[d], &p, nullptr))
            return MOIL_NB_ERR_GRID;
    }
    cudaStream_t stream = (cudaStream_t)stream_v;
    // an error the caller's own earlier work left pending is reported and left in place
    if (cudaPeekAtLastError() != cudaSuccess) return MOIL_NB_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NA_MAX_DEVICES) return MOIL_NB_ERR_CUDA;
    unsigned char *base = nullptr;
    {
        // first call on this device: resolve the device address of the scratch array (the
        // symbol itself is only a host-side stand-in and must not be handed to a kernel)
        std::lock_guard<std::mutex> lk(g_na_mu);
        if (!g_na_base[dev]) {
            void *ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_pme_scratch) != cudaSuccess || !ptr) return MOIL_NB_ERR_CUDA;
            g_na_base[dev] = (unsigned char *)ptr;
        }
        base = g_na_base[dev];
    }
    const int n1 = grid[0], n2 = grid[1], n3 = grid[2];
    {
        // the planes of this grid must fit the device's shared memory per block
        int optin = 0;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            return MOIL_NB_ERR_CUDA;
        if (plane_smem<float>(n1, n2) > (size_t)optin || zconv_smem<float>(n3) > (size_t)optin)
            return MOIL_NB_ERR_GRID;
    }
    // shared-memory limits for this grid (raise only; other handles may need more)
    if (raise_pme_limits<float>(plane_smem<float>(n1, n2), zconv_smem<float>(n3)) != cudaSuccess)
        return MOIL_NB_ERR_CUDA;
    // one-replica constants, FFT plans and tables, work lists (host side)
    NaParams P;
    memset((void *)&P, 0, sizeof(P));
    RepDev &R = P.R;
    for (int d = 0; d < 3; ++d) {
        R.Ld[d] = box[d];
        R.L[d] = (float)box[d];
        R.invLd[d] = 1.0 / box[d];
        R.invL[d] = (float)(1.0 / box[d]);
        R.Llo[d] = (float)(box[d] - (double)R.L[d]);
    }
    R.n1 = n1; R.n2 = n2; R.n3 = n3; R.n1h = n1 / 2 + 1;
    R.epstmp = NB_KOFDIE / eps;
    R.fcd = sqrt(R.epstmp);
    R.fc = (float)R.fcd;
    R.alpha = (float)alpha;
    R.alphad = alpha;
    R.pme_fac = M_PI * M_PI / (alpha * alpha);
    R.pivol = M_PI * box[0] * box[1] * box[2];
    nb_pme_fp32_consts(&R);
    R.pme_qcorr = 1.0;    // the charges stay on the device: no rounding correction
    R.natom = R.noth = natom;   // every atom a non-water site
    std::vector<int4> blob;
    int boff[3], blen[3];
    for (int d = 0; d < 3; ++d) {
        FftPlanDev plan;
        std::vector<int2> tab;
        std::vector<float2> tw(grid[d]);
        make_plan(grid[d], &plan, &tab);
        for (int t = 0; t < grid[d]; ++t) {
            const double ang = -2.0 * M_PI * (double)t / (double)grid[d];
            tw[t] = make_float2((float)cos(ang), (float)sin(ang));
        }
        push_blob(blob, plan, tab, tw, &boff[d], &blen[d]);
    }
    NbCtx tmp;
    tmp.stream = stream;
    tmp.nrep = 1;
    tmp.nsite = natom;
    for (int z = 0; z < n3; ++z) tmp.planes.push_back(PlaneWork{0, z, n1, n2, boff[0], blen[0], boff[1], blen[1], 0});
    for (int kx = 0; kx < R.n1h; ++kx)
        push_col_runs(tmp.cols, ColWork{0, kx, 0, 0, n1, n2, n3, 0, boff[2], blen[2], 0}, NB_TKF);
    if (NA_BLOB + sizeof(int4) * blob.size() > NA_HOST_BYTES) return MOIL_NB_ERR_GRID;
    tmp.smem_plane = plane_smem<float>(n1, n2);
    tmp.smem_zconv = zconv_smem<float>(n3);
    tmp.d_site_rep = (int *)(base + NA_REP);
    tmp.d_fr = base + NA_FR;
    tmp.d_zidx = base + NA_ZIDX;
    tmp.d_part = base + NA_PART;
    tmp.d_grid = base + NA_GRID;
    tmp.d_e_col = (double *)(base + NA_ECOL);
    tmp.d_planes = (PlaneWork *)(base + NA_HOST + NA_PLANES);
    tmp.d_cols = (ColWork *)(base + NA_HOST + NA_COLS);
    tmp.d_blob = (int4 *)(base + NA_HOST + NA_BLOB);
    tmp.d_etab = (float *)(base + NA_ETAB);
    NaParams *d_P = (NaParams *)(base + NA_HOST);
    tmp.d_reps = &d_P->R;
    double *d_eout = (double *)(base + NA_EOUT);
    std::vector<unsigned char> host(NA_BLOB + sizeof(int4) * blob.size());
    memcpy(host.data(), &P, sizeof(P));
    memcpy(host.data() + NA_PLANES, tmp.planes.data(), sizeof(PlaneWork) * tmp.planes.size());
    memcpy(host.data() + NA_COLS, tmp.cols.data(), sizeof(ColWork) * tmp.cols.size());
    memcpy(host.data() + NA_BLOB, blob.data(), sizeof(int4) * blob.size());
    // (pageable memory: copied out before the call returns)
    if (cudaMemcpyAsync(d_P, host.data(), host.size(), cudaMemcpyHostToDevice, stream) != cudaSuccess)
        return MOIL_NB_ERR_CUDA;
    const int nb = (natom + 255) / 256 + 1;      // the last block: tables, energy
    k_na_load<<<nb, 256, 0, stream>>>(natom, d_P, d_coor, d_q, (float4 *)tmp.d_fr, tmp.d_zidx, tmp.d_site_rep, tmp.d_etab);
    pme_t<float>(&tmp);
    k_na_grad<<<nb, 256, 0, stream>>>(natom, tmp.d_reps, d_q, (const float *)tmp.d_part, d_dpot, (int)tmp.cols.size(),
                                      tmp.d_e_col, d_eout);
    // a launch that failed is reported before waiting for the stream (the error stays pending
    // for the caller to read)
    if (cudaPeekAtLastError() != cudaSuccess) return MOIL_NB_ERR_CUDA;
    if (cudaMemcpyAsync(e_recip, d_eout, sizeof(double), cudaMemcpyDeviceToHost, stream) != cudaSuccess)
        return MOIL_NB_ERR_CUDA;
    if (cudaStreamSynchronize(stream) != cudaSuccess || cudaPeekAtLastError() != cudaSuccess) return MOIL_NB_ERR_CUDA;
    return MOIL_NB_OK;
}
