// negf_transmission.cu -- the FP64 transmission kernels whose block lives in
// global memory (negf.f90:115-174): F-mode streaming sweep + transmission
// epilogue, one CTA per (E,k) job, O(N^2) state per job.
#include "sweep_kernels.h"

namespace negf {
namespace {

// One F-mode sweep and the transmission trace for the job (E = e + i*eta,
// k-point ik) of problem g, in the workspace A0 (four ld x N blocks).  The
// basis must already be in s.nx / s.ny.  Returns tau in *tau (thread 0) and
// the LAPACK-style info.
template <int NB, int RPT, bool WIDE>
__device__ int transmission_job(const Geo &g, const Smem &s, double e, int ik, double2 *A0, double *tau) {
    const int N = g.N, ld = g.ld, Nz = g.Nz;
    double2 *A1 = A0 + (size_t)ld * N;
    double2 *P0 = A1 + (size_t)ld * N;
    double2 *P1 = P0 + (size_t)ld * N;
    const double2 E = make_double2(e, g.eta);
    job_vectors(g, s, E, e, ik);
    __syncthreads();
    open_rows(N, s);
    __syncthreads();
    const int nr = *s.nrows;
    double2 *cur = A0, *oth = A1, *P = P0, *Pn = P1;
    // generator_r(N_z-1) = inv(D_Nz)          math_kernel.f90:82
    form_block(cur, g, s, Nz - 1, E, ik, nullptr, nullptr);
    __syncthreads();
    int info = gj_invert<NB, RPT, WIDE>(cur, N, ld, s);
    unpermute_rows(P, ld, cur, ld, N, nr, s);
    __syncthreads();
    // generator_r(m) = inv(D_{m+1} - generator_r(m+1)), with the rows of the
    // running product P = gR(Nz-1) ... gR(m) of the first-column chain
    // G_{Nz,1} = (-1)^(Nz-1) gR(Nz-1) ... gR(1) G_11 (math_kernel.f90:83-90,120-128)
    // that the trace reads
    for (int m = Nz - 3; m >= 0; --m) {
        form_block(oth, g, s, m + 1, E, ik, cur, nullptr);
        __syncthreads();
        const int r = gj_invert<NB, RPT, WIDE>(oth, N, ld, s);
        if (r && !info) info = r;
        GemmArgs ga{Pn, ld, P, ld, s.iprow, oth, ld, s.iprow, nr, N, N, nullptr};
        cta_gemm(ga, s, GEMM_STORE, g.delta);
        __syncthreads();
        double2 *t = cur; cur = oth; oth = t;
        t = P; P = Pn; Pn = t;
    }
    // G_11 = inv(D_1 - generator_r(1))          math_kernel.f90:113-118
    form_block(oth, g, s, 0, E, ik, cur, nullptr);
    __syncthreads();
    const int r = gj_invert<NB, RPT, WIDE>(oth, N, ld, s);
    if (r && !info) info = r;
    // tau = sum_ij gamma_L,i gamma_R,j |2 dz^2 G_{Nz,1}(i,j)|^2   grid.f90:362-383
    GemmArgs ga{nullptr, 0, P, ld, s.iprow, oth, ld, s.iprow, nr, N, N, s.rows};
    double t = cta_gemm(ga, s, GEMM_TAU, g.delta);
    t = block_sum(t, s);
    *tau = t;
    return info;
}

template <int NB, int RPT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_transmission(Geo g, const double *__restrict__ energies, int nE, int njobs, double2 *ws,
                   size_t wstride, double *tau_jobs, int *info_jobs, Gate gate) {
    extern __shared__ __align__(256) unsigned char smem[];
    if (gate.shut()) return;
    Smem s = carve<NB>(smem, g.N);
    for (int i = threadIdx.x; i < g.N; i += NT) { s.nx[i] = g.nx[i]; s.ny[i] = g.ny[i]; }
    __syncthreads();
    double2 *A0 = ws + (size_t)blockIdx.x * wstride;
    for (int job = blockIdx.x; job < njobs; job += gridDim.x) {
        // job -> (energy, k-point), energy fastest: negf.f90:131-133
        const int ie = job % nE, ik = job / nE;
        double t = 0.0;
        const int info = transmission_job<NB, RPT, MINB == 1>(g, s, energies[ie], ik, A0, &t);
        if (threadIdx.x == 0) {
            tau_jobs[job] = t;
            if (info_jobs) info_jobs[job] = info;
        }
        __syncthreads();
    }
}

// Several problems (each its own basis, V table, slices and k-points) in one
// persistent launch: CTAs take jobs from a counter in the given order
// (largest first), so long and short sweeps balance across the SMs.
template <int NB, int RPT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_transmission_batch(const Geo *__restrict__ geos, const BatchJob *__restrict__ jobs, int njobs,
                         const double *__restrict__ energies, double2 *ws, size_t wstride, double *tau_jobs,
                         int *info_jobs, int *counter) {
    extern __shared__ __align__(256) unsigned char smem[];
    __shared__ int next;
    double2 *A0 = ws + (size_t)blockIdx.x * wstride;
    for (;;) {
        if (threadIdx.x == 0) next = atomicAdd(counter, 1);
        __syncthreads();
        const int q = next;
        __syncthreads();
        if (q >= njobs) break;
        const BatchJob jb = jobs[q];
        const Geo g = geos[jb.prob];
        Smem s = carve<NB>(smem, g.N);
        for (int i = threadIdx.x; i < g.N; i += NT) { s.nx[i] = g.nx[i]; s.ny[i] = g.ny[i]; }
        __syncthreads();
        double t = 0.0;
        const int info = transmission_job<NB, RPT, MINB == 1>(g, s, energies[jb.ie], jb.ik, A0, &t);
        if (threadIdx.x == 0) {
            tau_jobs[q] = t;
            info_jobs[q] = info;
        }
        __syncthreads();
    }
}

template <int NB, int RPT, int MINB>
SweepKernel make(int N) {
    return SweepKernel{(const void *)k_transmission<NB, RPT, MINB>, (const void *)k_transmission_batch<NB, RPT, MINB>,
                       NT, smem_bytes<NB, RPT, MINB == 1>(N), 4 * (size_t)round_up(N, 8) * N};
}

}  // namespace

SweepKernel sweep_kernel(Variant v, int N, int share, int open) {
    switch (v) {
        case V16x1: return make<16, 1, 2>(N);
        case V16x2: return make<16, 2, 1>(N);
        case V8x4: return make<8, 4, 1>(N);
        case VCHIP:
            if (N <= RNMAX) return register_kernel(N);
            if ((share >= 2 || N > NT) && open <= panel_channels(N) * (share >= 8 ? 2 : 1)) return panel_kernel(N);
            if (N > NT) return make<16, 2, 1>(N);
            return share >= 1 ? make<8, 1, 1>(N) : make<8, 1, 2>(N);
        default: return SweepKernel{};
    }
}

}  // namespace negf
