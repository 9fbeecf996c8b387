// negf_register.cu -- the FP64 transmission kernels of up to 72 plane waves:
// one CTA per (E,k) job, the block in registers (rgf_register.cuh).
#include "rgf_register.cuh"

namespace negf {
namespace {

// CPW storage columns per warp, RPL row slots per lane (the block and
// its open channels), PR of them holding rows of the block.
template <int CPW, int RPL, int PR, int MINB>
__global__ void __launch_bounds__(RT, MINB)
    k_register(Geo g, const double *__restrict__ energies, int nE, int njobs, double2 *, size_t,
               double *tau_jobs, int *info_jobs, Gate) {
    __shared__ RegSmem<32 * RPL, CPW> s;
    for (int job = blockIdx.x; job < njobs; job += gridDim.x) {
        const int ie = job % nE, ik = job / nE;  // energy fastest: negf.f90:131-133
        int info;
        const double tau = reg_transmission_job<CPW, RPL, PR>(g, s, energies[ie], ik, &info);
        if (threadIdx.x == 0) {
            tau_jobs[job] = tau;
            if (info_jobs) info_jobs[job] = info;
        }
        __syncthreads();
    }
}

template <int CPW, int RPL, int PR, int MINB>
__global__ void __launch_bounds__(RT, MINB)
    k_register_batch(const Geo *__restrict__ geos, const BatchJob *__restrict__ jobs, int njobs,
                     const double *__restrict__ energies, double2 *, size_t, double *tau_jobs, int *info_jobs,
                     int *counter) {
    __shared__ RegSmem<32 * RPL, CPW> s;
    __shared__ int next;
    for (;;) {
        if (threadIdx.x == 0) next = atomicAdd(counter, 1);
        __syncthreads();
        const int q = next;
        __syncthreads();
        if (q >= njobs) break;
        const BatchJob jb = jobs[q];
        const Geo g = geos[jb.prob];
        int info;
        const double tau = reg_transmission_job<CPW, RPL, PR>(g, s, energies[jb.ie], jb.ik, &info);
        if (threadIdx.x == 0) {
            tau_jobs[q] = tau;
            info_jobs[q] = info;
        }
        __syncthreads();
    }
}

template <int CPW, int RPL, int PR, int MINB>
SweepKernel make() {
    return SweepKernel{(const void *)k_register<CPW, RPL, PR, MINB>, (const void *)k_register_batch<CPW, RPL, PR, MINB>,
                       RT, 0, 0};
}

}  // namespace

// 2, 4 or 6 columns a warp; the row slots hold 2 N rows, so that every channel
// may be open.  A narrower kernel leaves room for two or three CTAs per SM.
SweepKernel register_kernel(int N) {
    if (N <= 24) return make<2, 2, 1, 3>();
    if (N <= 48) return make<4, 3, 2, 2>();
    return make<6, 5, 3, 1>();
}

}  // namespace negf
