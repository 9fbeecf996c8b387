// sweep_kernels.h -- the sweep kernels as the host code sees them: what each
// launch needs, by kernel variant and basis size.  Private to the library.
#pragma once
#include "rgf_device.cuh"

namespace negf {

// One (problem, energy, k-point) job of a batch over several problems.
struct BatchJob {
    int prob, ie, ik, pad;
};

// A kernel that has nothing to do unless lo <= *open < hi (open null: always runs).
struct Gate {
    const int *open = nullptr;
    int lo = 0, hi = 0;
    __device__ bool shut() const { return open && (*open < lo || *open >= hi); }
};

// A transmission kernel in its two forms, of one signature for every variant:
//   one    (Geo, const double *energies, int nE, int njobs, double2 *ws, size_t wstride,
//           double *tau_jobs, int *info_jobs, Gate): the nE * nk jobs of one problem, energy fastest
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
// plane waves.  3 is the family below, by basis size, jobs and open channels.
enum Variant { V16x1 = 0, V16x2 = 1, V8x4 = 2, VCHIP = 3, VNONE = 4 };

// The kernel of a variant for a basis of N, `share` SMs per job and at most
// `open` channels open in the left lead.  Variant 3: the block in registers up
// to RNMAX; above, panels in registers and teams of CTAs if the jobs are few
// (two SMs each, or more: nine jobs of N = 221, N_z = 160, 175 -> 86 ms in teams
// of eight) or N > 256 (148 jobs of N = 257, N_z = 6, 14.5 ms in 16 x 2 x 1, which
// takes a whole SM as well, 10.7 in panels; N = 272 15.2 and 12.8); otherwise
// 8 x 1 x 2, whose two jobs per SM cover each other's pivots (N = 221: 840 us of
// an SM per slice and job, the panel kernel alone on an SM 1000), or 8 x 1 x 1
// where every job has an SM to itself: the pipelined 64 x 64 tiles of the
// one-CTA variants (148 jobs of N = 128, 221, 256, N_z = 8, 2.76 -> 2.31, 9.3 -> 8.0,
// 13.6 -> 11.1 ms; 32 x 64 tiles alone on an SM were up to 4 % slower than unpipelined
// ones).
//
// A block of the panel kernel has room for panel_channels(N) channels; more
// take another sweep each time, where the other kernels only carry a wider
// product.  One pass always gains; a second one only in the largest teams
// (nine jobs of N = 257, 80 channels 12.3 -> 8.5 ms, 36 jobs 12.6 and 12.3, 148
// jobs 15.7 and 23.2; N = 272 with all open 16.6 and 29.1, 20.4 and 78.1), so
// that share >= 8 allows two passes, and every other call one.
SweepKernel sweep_kernel(Variant v, int N, int share, int open);  // negf_transmission.cu
SweepKernel register_kernel(int N);          // negf_register.cu, up to RNMAX
SweepKernel panel_kernel(int N);             // negf_panel.cu, up to PNMAX
// PNMAX: the block, its factor and one chunk of pivot rows in 227 KB of shared
// memory, 320 rows of it in registers.
constexpr int RNMAX = 72, PNMAX = 272;
__host__ __device__ inline int panel_rows(int N) { return 2 * N < 320 ? round_up(2 * N, 8) : 320; }
inline int panel_channels(int N) { return panel_rows(N) - N; }

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
