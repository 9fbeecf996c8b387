// negf_panel.cu -- the FP64 transmission kernels of 73 to 272 plane waves:
// panels in registers, one CTA or a team of CTAs per (E,k) job (rgf_panel.cuh).
#include "rgf_panel.cuh"

namespace negf {
namespace {

__device__ inline PanelTeam make_team(double2 *ws, size_t wstride, int N) {
    PanelTeam t;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(t.rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(t.size));
    t.ld = panel_rows(N);
    t.head = ws + (size_t)(blockIdx.x / t.size) * wstride;
    t.A = t.head + 2 * PHEAD;
    t.Vg = t.A + (size_t)t.ld * N;
    return t;
}

__global__ void __launch_bounds__(PT, 1)
    k_panel(Geo g, const double *__restrict__ energies, int nE, int njobs, double2 *ws, size_t wstride,
            double *tau_jobs, int *info_jobs, Gate gate) {
    extern __shared__ __align__(256) unsigned char smem[];
    if (gate.shut()) return;
    const PanelTeam t = make_team(ws, wstride, g.N);
    const PanelSmem s = carve_panel(smem, g.N, 0);
    for (int job = blockIdx.x / t.size; job < njobs; job += gridDim.x / t.size) {
        const int ie = job % nE, ik = job / nE;  // energy fastest: negf.f90:131-133
        int info;
        const double tau = panel_transmission_job(t, s, g, energies[ie], ik, &info);
        if (t.rank == 0 && threadIdx.x == 0) {
            tau_jobs[job] = tau;
            if (info_jobs) info_jobs[job] = info;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(PT, 1)
    k_panel_batch(const Geo *__restrict__ geos, const BatchJob *__restrict__ jobs, int njobs,
                  const double *__restrict__ energies, double2 *ws, size_t wstride, double *tau_jobs, int *info_jobs,
                  int *counter) {
    extern __shared__ __align__(256) unsigned char smem[];
    PanelTeam t = make_team(ws, wstride, 0);
    int *next = (int *)t.head + 4 * PHEAD - 1;  // (the header's last word)
    for (;;) {
        if (t.rank == 0 && threadIdx.x == 0) *next = atomicAdd(counter, 1);
        panel_sync(t);
        const int q = __ldcg(next);
        panel_sync(t);
        if (q >= njobs) break;
        const BatchJob jb = jobs[q];
        const Geo g = geos[jb.prob];
        t = make_team(ws, wstride, g.N);
        const PanelSmem s = carve_panel(smem, g.N, 0);
        int info;
        const double tau = panel_transmission_job(t, s, g, energies[jb.ie], jb.ik, &info);
        if (t.rank == 0 && threadIdx.x == 0) {
            tau_jobs[q] = tau;
            info_jobs[q] = info;
        }
        __syncthreads();
    }
}

}  // namespace

SweepKernel panel_kernel(int N) {
    SweepKernel k{(const void *)k_panel, (const void *)k_panel_batch, PT, panel_smem(N), panel_ws(N)};
    k.team = 8;
    return k;
}

}  // namespace negf
