// sweep_kernels.h -- the sweep kernels as the host code sees them: what each
// launch needs, by kernel variant and basis size.  Private to the library.
#pragma once
#include "rgf_device.cuh"

namespace negf {

// One (problem, energy, k-point) job of a batch over several problems.
struct BatchJob {
    int prob, ie, ik, pad;
};

// A transmission kernel in its two forms, of one signature for every variant:
//   one    (Geo, const double *energies, int nE, int njobs, double2 *ws, size_t wstride,
//           double *tau_jobs, int *info_jobs): the nE * nk jobs of one problem, energy fastest
//   batch  (const Geo *, const BatchJob *, int njobs, const double *energies, double2 *ws,
//           size_t wstride, double *tau_jobs, int *info_jobs, int *counter): jobs of several
//           problems, taken in order from a counter
struct SweepKernel {
    const void *one = nullptr, *batch = nullptr;
    int threads = 0;
    size_t smem = 0;  // dynamic shared memory for a basis of N
    size_t ws = 0;    // workspace of one CTA (team) in double2 for a basis of N
    int team = 1;     // most CTAs (a thread-block cluster) that can share a job
};

// The variants of negf_set_variant.  0 .. 2 keep the block in global memory:
// (panel width NB, rows per thread RPT, CTAs per SM), two CTAs per SM up to 256
// plane waves.  3 is the family below, by basis size and number of jobs.
enum Variant { V16x1 = 0, V16x2 = 1, V8x4 = 2, VCHIP = 3, VNONE = 4 };

// The kernel of a variant for a basis of N.  Variant 3: the block in registers
// up to RNMAX; above, panels in registers and teams of CTAs if the jobs are
// few (at most one per two SMs: nine jobs of N = 221, N_z = 160, 175 -> 86 ms in
// teams of eight) or N > 256 (the next variant takes a whole SM as
// well, at two rows per thread); otherwise 8 x 1 x 2, whose two jobs per SM
// cover each other's pivots (N = 221: 840 us of an SM per slice and job, the
// panel kernel alone on an SM 1160).
SweepKernel sweep_kernel(Variant v, int N, bool few);  // negf_transmission.cu
SweepKernel register_kernel(int N);          // negf_register.cu, up to RNMAX
SweepKernel panel_kernel(int N);             // negf_panel.cu, up to PNMAX
constexpr int RNMAX = 72, PNMAX = 272;

struct RgfJob {
    double e_re, e_im;  // complex energy of the solve, E + i*eta already added
    double e_t;         // real energy of the transmission weights
    int ik;             // k-point
    int pad;
    // WANT_A only: slice k of the output is cd * G_kk + ca * G_k,s Gamma_s G_k,s^H
    // (s = the injecting lead's end slice, Gamma_s its open-channel widths)
    double cd_re, cd_im, ca_re, ca_im;
};

enum { WANT_D = 1, WANT_F = 2, WANT_L = 4, WANT_A = 8, WANT_MIRROR = 16 };

// k_rgf_slab's arguments: (Geo, const RgfJob *, int njobs, const double2 *Dexp, double2 *ws,
// size_t wstride, double2 *slabs, size_t sstride, int want, double2 *out_first, double2 *out_last,
// int *info_jobs); one CTA per job.
struct SlabKernel {
    const void *fn = nullptr;
    int threads = 0;
    size_t smem = 0;
    int blocks = 6;  // workspace of a job in blocks of round_up(N, 8) x N
};
SlabKernel slab_kernel(int N);                // negf_slab.cu
SlabKernel register_slab_kernel(int N);       // negf_register_slab.cu, up to RNMAX

}  // namespace negf
