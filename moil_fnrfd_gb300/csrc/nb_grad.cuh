// nb_grad.cuh -- the gradient of one caller atom from its parts, for the evaluation's last kernel and the
// MD integrator.
#pragma once
#include "nb_common.cuh"

namespace {

// one atom's gradient: fixed-point real space + FP64 corrections + PME; false if not finite.  fine (FP64
// path): the water sites' part at NB_FINE_SCALE, sites below nfine
template <typename T>
__device__ __forceinline__ bool final_grad(int a, const int *__restrict__ site_of, const int *__restrict__ atom_rep,
                                           const RepDev *__restrict__ reps, const long long *__restrict__ grad_site,
                                           const double *__restrict__ grad_ex, const T *__restrict__ part,
                                           const double *__restrict__ q, int nsw,
                                           const long long *__restrict__ fine, int nfine, double g[3])
{
    const RepDev &R = reps[atom_rep[a]];
    int s = site_of[a];
    bool bad = false;
    if constexpr (sizeof(T) == 4) {
        // FP32 path: the PME share (one float4 per site from k_pme_gather_f) is scaled in
        // FP32 (its own precision) and joins the fixed-point real-space and correction terms
        // as an integer; the double result is assembled with integer operations (no FP64
        // instruction).  Sites below nsw (waters whose corrections the water kernel added)
        // have no correction term.
        const long long *gx = (const long long *)grad_ex + 3 * (size_t)a;
        const bool ex = s >= nsw;
        const float qs = (float)q[a];
        const float4 p4 = ((const float4 *)part)[s];
        const float pg[3] = {p4.x, p4.y, p4.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const long long v = grad_site[3 * (size_t)s + d] + (ex ? gx[d] : 0LL) + nb_f2fix(qs * R.pme_gs[d] * pg[d]);
            bad |= (v > (1LL << 61)) | (v < -(1LL << 61));   // a saturated (non-finite) term
            g[d] = nb_fix2d(v);
        }
    } else {
        const T *p = part + 12 * (size_t)s;   // 4 plane slots per site (k_plane_inv)
        double pg[3] = {0, 0, 0};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            pg[0] += (double)p[3 * t];
            pg[1] += (double)p[3 * t + 1];
            pg[2] += (double)p[3 * t + 2];
        }
        double qf = q[a] * R.fcd;
        double sc[3] = {qf * R.n1 * R.invLd[0], qf * R.n2 * R.invLd[1], qf * R.n3 * R.invLd[2]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double v = (double)grad_site[3 * (size_t)s + d] * NB_FIX_INV;
            if (s < nfine) v += (double)fine[3 * (size_t)s + d] * (1.0 / NB_FINE_SCALE);
            v += grad_ex[3 * (size_t)a + d] + sc[d] * pg[d];
            bad |= !(v == v);
            g[d] = v;
        }
    }
    return !bad;
}

}  // namespace
