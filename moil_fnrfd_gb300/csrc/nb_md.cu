// nb_md.cu -- device-resident molecular dynamics around the nonbonded evaluation: leapfrog
// steps with rigid three-site waters, and the DCD trajectory writer.
//
// MOIL's integrator (dynamics/dyna.f:183-330) advances positions with leapfrog and holds
// water geometry with SHAKE (dynamics/shakept.f, matrix SHAKE dynamics/mshakpt.f); velocity
// constraints follow (dynamics/shakevl.f).  Here, after each evaluation,
//     v(t + dt/2) = v(t - dt/2) - dt * c * dpot / m          (c = 418.4: kcal/mol/Å/amu -> Å/ps^2)
//     x(t + dt)   = SETTLE(x(t), x(t) + dt * v(t + dt/2)),   v(t + dt/2) = (x(t + dt) - x(t)) / dt
// with SETTLE the analytic rigid-water solution of Miyamoto and Kollman (J. Comput. Chem. 13,
// 952 (1992)): the unconstrained molecule is expressed in a frame built from the previous
// molecule, the rotations phi, psi (out of plane) and theta (in plane) place the rigid
// molecule keeping the centre of mass and constraint forces along the old bonds.  Atoms
// outside waters move unconstrained (this library holds no bonded terms).  FP64 throughout.
// The trajectory writer follows dynamics/wdyncrd.f's binary branch: Fortran unformatted
// sequential records (4-byte length before and after each record).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>

#include "nb_grad.cuh"
#include "nb_internal.h"

namespace {

constexpr double kAccel = 418.4;

__device__ __forceinline__ double dot3(const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void cross3(const double *a, const double *b, double *c)
{
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ void unit3(double *a)
{
    const double s = rsqrt(dot3(a, a));
    a[0] *= s; a[1] *= s; a[2] *= s;
}

// rigid positions p1[3][3] (O, H, H) from the previous rigid p0 and the unconstrained p1;
// dhh the rigid H-H distance, h the height of O over it, mo, mh the masses
__device__ __forceinline__ void settle(const double p0[3][3], double p1[3][3], double dhh, double h, double mo, double mh)
{
    const double imt = 1.0 / (mo + 2.0 * mh), rc = 0.5 * dhh;
    const double ra = 2.0 * mh * h * imt, rb = h - ra;
    double com[3], a1[3], b1[3], c1[3], ab0[3], ac0[3], ex[3], ey[3], ez[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        com[d] = (mo * p1[0][d] + mh * (p1[1][d] + p1[2][d])) * imt;
        a1[d] = p1[0][d] - com[d];
        b1[d] = p1[1][d] - com[d];
        c1[d] = p1[2][d] - com[d];
        ab0[d] = p0[1][d] - p0[0][d];
        ac0[d] = p0[2][d] - p0[0][d];
    }
    // frame: z normal to the previous molecule, x normal to z and the new O offset
    cross3(ab0, ac0, ez);
    cross3(a1, ez, ex);
    unit3(ex); unit3(ez);
    cross3(ez, ex, ey);
    const double xb0 = dot3(ab0, ex), yb0 = dot3(ab0, ey), xc0 = dot3(ac0, ex), yc0 = dot3(ac0, ey);
    const double za1 = dot3(a1, ez);
    const double xb1 = dot3(b1, ex), yb1 = dot3(b1, ey), zb1 = dot3(b1, ez);
    const double xc1 = dot3(c1, ex), yc1 = dot3(c1, ey), zc1 = dot3(c1, ez);
    // phi and psi: the out-of-plane heights of O and of the H-H axis are kept
    const double sphi = za1 / ra, cphi = sqrt(fmax(1.0 - sphi * sphi, 0.0));
    const double spsi = (zb1 - zc1) / (2.0 * rc * cphi), cpsi = sqrt(fmax(1.0 - spsi * spsi, 0.0));
    const double ya2 = ra * cphi, xb2 = -rc * cpsi;
    const double yb2 = -rb * cphi - rc * spsi * sphi, yc2 = -rb * cphi + rc * spsi * sphi;
    // theta: the in-plane rotation for which the constraint forces lie along the old bonds
    const double al = xb2 * (xb0 - xc0) + yb0 * yb2 + yc0 * yc2;
    const double be = xb2 * (yc0 - yb0) + xb0 * yb2 + xc0 * yc2;
    const double ga = xb0 * yb1 - xb1 * yb0 + xc0 * yc1 - xc1 * yc0;
    const double ab2 = al * al + be * be;
    const double sth = (al * ga - be * sqrt(fmax(ab2 - ga * ga, 0.0))) / ab2, cth = sqrt(fmax(1.0 - sth * sth, 0.0));
    const double loc[3][3] = {{-ya2 * sth, ya2 * cth, za1},
                              {xb2 * cth - yb2 * sth, xb2 * sth + yb2 * cth, zb1},
                              {-xb2 * cth - yc2 * sth, -xb2 * sth + yc2 * cth, zc1}};
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int d = 0; d < 3; ++d) p1[m][d] = com[d] + loc[m][0] * ex[d] + loc[m][1] * ey[d] + loc[m][2] * ez[d];
}

// One water per thread: its caller atoms are consecutive (O, H, H).  Bound: the FP64 pipe (two lanes
// per clock and multiprocessor), so the work is cut into blocks of one warp that spread evenly over
// the multiprocessors: 28,800 waters in blocks of 128 left a third of them with half the work of the
// others, 30.6 us; blocks of 32, and the constants and unit vectors with fewer square roots and
// divisions, 19.7.
// In a step graph the gradient comes from its parts (StepGrad), not from an array that a kernel before
// has assembled.
#define NB_LF 32
struct ArrayGrad {
    const double *dpot;
    __device__ void operator()(size_t a, double g[3]) const
    {
#pragma unroll
        for (int d = 0; d < 3; ++d) g[d] = dpot[3 * a + d];
    }
};
template <typename T> struct StepGrad {
    const int *site_of, *atom_rep;
    const RepDev *reps;
    const long long *grad_site;
    const double *grad_ex;
    const T *part;
    const double *q;
    int nsw;
    const long long *fine;
    int nfine;
    int *nan_h, *ctl;
    __device__ void operator()(size_t a, double g[3]) const
    {
        if (!final_grad<T>((int)a, site_of, atom_rep, reps, grad_site, grad_ex, part, q, nsw, fine, nfine, g)) {
            *nan_h = 1;
            atomicOr(&ctl[2], NB_DEV_ERR_NAN);
        }
    }
};
template <typename G>
__global__ void __launch_bounds__(NB_LF) k_leapfrog_water(int nW, const int *__restrict__ unit_atom,
                                                          const double *__restrict__ mass, double dt, double inv_dt,
                                                          double dhh, double h, double *__restrict__ coor,
                                                          double *__restrict__ vel, G grad)
{
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nW) return;
    const size_t a = (size_t)unit_atom[w];
    const double ms[3] = {mass[a], mass[a + 1], mass[a + 2]};
    double p0[3][3], p1[3][3], f[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) f[m] = m == 2 && ms[2] == ms[1] ? f[1] : dt * kAccel / ms[m];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        double g[3];
        grad(a + m, g);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const size_t k = 3 * (a + m) + d;
            p0[m][d] = coor[k];
            p1[m][d] = p0[m][d] + dt * (vel[k] - f[m] * g[d]);
        }
    }
    settle(p0, p1, dhh, h, ms[0], ms[1]);
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const size_t k = 3 * (a + m) + d;
            vel[k] = (p1[m][d] - p0[m][d]) * inv_dt;
            coor[k] = p1[m][d];
        }
}

// every atom outside a water, unconstrained
template <typename G>
__global__ void k_leapfrog_free(int natom, const unsigned *__restrict__ aflags, const double *__restrict__ mass,
                                double dt, double *__restrict__ coor, double *__restrict__ vel, G grad)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= natom || (aflags[a] & SF_WATER)) return;
    const double f = dt * kAccel / mass[a];
    double g[3];
    grad(a, g);
    for (int d = 0; d < 3; ++d) {
        const size_t k = 3 * (size_t)a + d;
        vel[k] -= f * g[d];
        coor[k] += dt * vel[k];
    }
}

// kinetic energy partial sums per block (fixed order), summed on the host
__global__ void __launch_bounds__(256) k_kinetic(int natom, const double *__restrict__ mass,
                                                 const double *__restrict__ vel, double *__restrict__ part)
{
    __shared__ double sh[256];
    double s = 0.0;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < natom; a += gridDim.x * blockDim.x) {
        const double *v = vel + 3 * (size_t)a;
        s += 0.5 * mass[a] * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0] / kAccel;
}

// the integrator kernels of one (ungrouped) context over its caller-atom range
template <typename G>
int integrate(NbCtx *c, cudaStream_t s, double *coor, double *vel, const double *mass, G grad, double dt, double doh,
              double dhh)
{
    if (c->nW > 0)
        k_leapfrog_water<<<(int)((c->nW + NB_LF - 1) / NB_LF), NB_LF, 0, s>>>(
            (int)c->nW, c->d_unit_atom, mass, dt, 1.0 / dt, dhh, sqrt(doh * doh - 0.25 * dhh * dhh), coor, vel, grad);
    if (c->nA > 0)
        k_leapfrog_free<<<(int)((c->natom + 255) / 256), 256, 0, s>>>((int)c->natom, c->d_aflags, mass, dt, coor, vel,
                                                                      grad);
    NB_CUDA_OK(c, cudaGetLastError());
    return MOIL_NB_OK;
}

}  // namespace

int nb_launch_integrate(NbCtx *c, cudaStream_t s, double *coor, double *vel, const double *mass, double dt, double doh,
                        double dhh, int *ctl)
{
    auto with = [&](auto part, int nsw) {
        typedef std::remove_const_t<std::remove_pointer_t<decltype(part)>> T;
        return integrate(c, s, coor, vel, mass,
                         StepGrad<T>{c->d_site_of, c->d_atom_rep, c->d_reps, c->d_grad_site, c->d_grad_ex, part, c->d_q,
                                     nsw, c->d_grad_fine, c->d_grad_fine ? (int)(3 * c->nW) : 0, c->h_status + 23, ctl},
                         dt, doh, dhh);
    };
    if (c->precision == MOIL_NB_FP64) return with((const double *)c->d_part, 0);
    return with((const float *)c->d_part, c->water_excl_fast ? (int)(3 * c->nW) : 0);
}

namespace {

void put_record(FILE *f, const void *data, uint32_t bytes)
{
    fwrite(&bytes, 4, 1, f);
    fwrite(data, 1, bytes, f);
    fwrite(&bytes, 4, 1, f);
}

}  // namespace

extern "C" {

int moil_nb_md_step(moil_nb_ctx *h, double *d_coor, double *d_vel, const double *d_mass, double dt, int nsteps,
                    const double *water_geom, moil_energies *energies, double *ekin)
{
    if (!h || !d_coor || !d_vel || !d_mass || !(dt > 0.0) || nsteps < 0) return MOIL_NB_ERR_ARG;
    if (!h->inited || h->pending) return MOIL_NB_ERR_STATE;
    cudaSetDevice(h->device);
    // TIP3P: O-H 0.9572 Å, H-O-H 104.52 degrees
    const double doh = water_geom ? water_geom[0] : 0.9572;
    const double dhh = water_geom ? water_geom[1] : 2.0 * 0.9572 * sin(104.52 * M_PI / 360.0);
    const size_t n = (size_t)h->natom;
    if (!h->d_md_dpot) NB_CUDA_OK(h, cudaMalloc(&h->d_md_dpot, sizeof(double) * 3 * std::max<size_t>(n, 1)));
    // Device-side loop: every context replays graphs of whole steps with no host wait between them;
    // the error bits are read once at the end.  With a list period the host decides which steps
    // rebuild, in runs of at most 64 steps; a run whose lists were outrun before their time goes back
    // to its saved state and leaves the decision to the device, as do some of the next runs
    // (ListForesight).  Any other error (a list overflow to regrow, a
    // non-finite coordinate) sends the run back to the saved state and the rest of the call through
    // the per-step path below, which handles it as a single evaluation does.
    int first = 0;
    const bool loop = nsteps > 1 && h->use_graph && !h->timing;
    std::vector<NbCtx *> ctxs;
    if (h->grp.empty()) ctxs.push_back(h);
    else for (NbCtx *c : h->grp) ctxs.push_back(c);
    if (loop && !h->d_md_save) NB_CUDA_OK(h, cudaMalloc(&h->d_md_save, sizeof(double) * 6 * std::max<size_t>(n, 1)));
    // (a replica group's period is its own first replica's)
    bool periods = true;
    for (const NbCtx *c : ctxs) periods &= c->list_period > 0;
    while (loop && first < nsteps) {
        const bool host = h->md_lists.host(periods);
        const int run = host ? std::min(nsteps - first, 64) : nsteps - first;
        h->md_lists.begin();
        NB_CUDA_OK(h, cudaMemcpyAsync(h->d_md_save, d_coor, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
        NB_CUDA_OK(h, cudaMemcpyAsync(h->d_md_save + 3 * n, d_vel, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice,
                                      h->stream));
        int rc = MOIL_NB_OK;
        for (size_t g = 0; g < ctxs.size() && rc == MOIL_NB_OK; ++g) {
            NbCtx *c = ctxs[g];
            const int64_t a0 = h->grp.empty() ? 0 : h->grp_atom0[g];
            if (c != h) {
                NB_CUDA_OK(h, cudaEventRecord(h->ev[11], h->stream));            // the snapshot copies
                NB_CUDA_OK(h, cudaStreamWaitEvent(c->stream, h->ev[11], 0));
            }
            rc = nb_md_loop(c, d_coor + 3 * a0, d_vel + 3 * a0, d_mass + a0, dt, doh, dhh, run, host);
        }
        int err = 0;
        for (NbCtx *c : ctxs) {
            NB_CUDA_OK(h, cudaStreamSynchronize(c->stream));
            if (rc == MOIL_NB_OK) {
                err |= c->h_status[22];
                if (!c->h_status[22]) {
                    // the host's view of the list schedule, pair counts and energies
                    c->evals_since_build = c->h_status[20];
                    c->need_rebuild = 0;
                    read_energies_of(c, nullptr);
                }
            }
        }
        if (rc == MOIL_NB_OK && !err) {
            first += run;
            if (host) h->md_lists.kept();
            continue;
        }
        NB_CUDA_OK(h, cudaMemcpyAsync(d_coor, h->d_md_save, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
        NB_CUDA_OK(h, cudaMemcpyAsync(d_vel, h->d_md_save + 3 * n, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice,
                                      h->stream));
        NB_CUDA_OK(h, cudaStreamSynchronize(h->stream));
        for (NbCtx *c : ctxs) c->need_rebuild = 1;
        if (rc != MOIL_NB_OK) cudaGetLastError();
        if (rc != MOIL_NB_OK || err != NB_DEV_STALE) break;
        h->md_lists.outrun();
    }
    if (loop && first == nsteps) {
        if (!h->grp.empty()) {
            h->last_site_pairs = 0;
            for (NbCtx *c : ctxs) h->last_site_pairs += c->last_site_pairs;
        }
        if (energies) {
            for (size_t g = 0; g < ctxs.size(); ++g)
                read_energies_of(ctxs[g], energies + (h->grp.empty() ? 0 : h->grp_rep0[g]));
        }
    }
    for (int step = first; step < nsteps; ++step) {
        int rc = moil_nb_eval_device(h, d_coor, h->d_md_dpot, step + 1 == nsteps ? energies : nullptr);
        if (rc != MOIL_NB_OK) return rc;
        if (h->grp.empty()) {
            rc = integrate(h, h->stream, d_coor, d_vel, d_mass, ArrayGrad{h->d_md_dpot}, dt, doh, dhh);
        } else {
            // each group integrates its own atoms on its stream; the handle's stream waits
            for (size_t g = 0; g < h->grp.size() && rc == MOIL_NB_OK; ++g) {
                const int64_t a0 = h->grp_atom0[g];
                rc = integrate(h->grp[g], h->grp[g]->stream, d_coor + 3 * a0, d_vel + 3 * a0, d_mass + a0,
                               ArrayGrad{h->d_md_dpot + 3 * a0}, dt, doh, dhh);
            }
            for (NbCtx *c : h->grp) {
                NB_CUDA_OK(h, cudaEventRecord(c->ev[11], c->stream));
                NB_CUDA_OK(h, cudaStreamWaitEvent(h->stream, c->ev[11], 0));
            }
        }
        if (rc != MOIL_NB_OK) { if (h->err.empty() && !h->grp.empty()) h->err = h->grp[0]->err; return rc; }
    }
    if (ekin) {
        const int nb = (int)std::min<size_t>((n + 255) / 256, 1024);
        std::vector<double> part(std::max(nb, 1));
        double *d_part = nullptr;
        NB_CUDA_OK(h, cudaMallocAsync((void **)&d_part, sizeof(double) * part.size(), h->stream));
        k_kinetic<<<std::max(nb, 1), 256, 0, h->stream>>>((int)n, d_mass, d_vel, d_part);
        NB_CUDA_OK(h, cudaGetLastError());
        NB_CUDA_OK(h, cudaMemcpyAsync(part.data(), d_part, sizeof(double) * part.size(), cudaMemcpyDeviceToHost,
                                      h->stream));
        NB_CUDA_OK(h, cudaFreeAsync(d_part, h->stream));
        NB_CUDA_OK(h, cudaStreamSynchronize(h->stream));
        double k = 0.0;
        for (double v : part) k += v;
        *ekin = k;
    } else {
        NB_CUDA_OK(h, cudaStreamSynchronize(h->stream));
    }
    return MOIL_NB_OK;
}

int moil_nb_dcd_write(const char *path, int first, int nframes, int natom, const double *coor)
{
    if (!path || natom <= 0 || !coor) return MOIL_NB_ERR_ARG;
    FILE *f = fopen(path, first ? "wb" : "ab");
    if (!f) return MOIL_NB_ERR_ARG;
    if (first) {
        // header as dynamics/wdyncrd.f writes it: 'CORD' + 20 integers (1: frames,
        // 9: fixed atoms), a title record, the atom count
        unsigned char rec[84];
        int32_t vari[20] = {0};
        vari[0] = nframes;
        memcpy(rec, "CORD", 4);
        memcpy(rec + 4, vari, sizeof vari);
        put_record(f, rec, 84);
        unsigned char title[84];
        const int32_t one = 1;
        memcpy(title, &one, 4);
        char text[80];
        memset(text, ' ', 80);
        const char *t = "A dummy title to dynamics coordinates";
        memcpy(text, t, strlen(t));
        memcpy(title + 4, text, 80);
        put_record(f, title, 84);
        const int32_t n = natom;
        put_record(f, &n, 4);
    }
    std::vector<float> v(natom);
    for (int d = 0; d < 3; ++d) {
        for (int a = 0; a < natom; ++a) v[a] = (float)coor[3 * (size_t)a + d];
        put_record(f, v.data(), (uint32_t)(sizeof(float) * natom));
    }
    const int bad = ferror(f);
    fclose(f);
    return bad ? MOIL_NB_ERR_ARG : MOIL_NB_OK;
}

}  // extern "C"
