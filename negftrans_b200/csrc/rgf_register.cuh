// rgf_register.cuh -- the FP64 transmission sweep with the block held in registers
// (sm_100a, up to 72 plane waves).
//
// A block of at most 72 x 72 complex FP64 values fits the register file of one
// SM, so the whole sweep of a job runs without touching global memory for
// anything but the V table: D_k is generated into the registers that hold the
// previous inverse, the elimination updates them in place, and the result is
// the operand of the next slice.
//
// Layout: storage column c belongs to warp c % 12 (slot c / 12), storage row i
// to lane i % 32 (slot i / 32).  A column lies in one warp, so its pivot search
// is one warp reduction, and every warp reads its own part of the pivot row
// from one of its lanes.
//
// The chain product G_{Nz,1} = +- gR(Nz-1) ... gR(1) G_11 (math_kernel.f90:83-90,
// 120-128) is carried by the elimination itself: rows appended below the block
// take part in every step but are never pivots, and Gauss-Jordan turns
// [M; P] into [inv(M); -P inv(M)].  They start as the unit rows of the open
// channels, so no product is formed apart from the inverses.
//
// The rows and columns of the registers are never permuted.  Storage row i
// stands for basis row rho[i] and storage column c for basis column kappa[c];
// inv(M) of a block stored that way comes out at (i, c) = (rho'[i], kappa'[c])
// with rho'[prow[j]] = j and kappa'[cst[j]] = rho[prow[j]], where prow[j] is
// the pivot row of basis column j and cst[j] its storage column.  The next
// block is generated in exactly that order, element on element.
//
// Measured on a B200 against the global-memory kernel (8 x 1 x 2) it replaces
// for these sizes: N = 69, N_z = 200, one energy 28.6 -> 15.0 ms, 512 energies
// 80.2 -> 61.2 ms; N = 21, N_z = 60, one energy 1.91 -> 0.82 ms, 600 energies
// 6.2 -> 2.0 ms; N = 45, 400 energies 10.8 -> 5.5 ms.
#pragma once
#include "rgf_device.cuh"
#include "sweep_kernels.h"

namespace negf {

constexpr int RT = 384;       // threads per CTA
constexpr int RW = RT / 32;   // warps, which share the columns

// Shared state of one CTA: RMAX rows (basis rows and appended rows), CPW columns per warp.
template <int RMAX, int CPW>
struct RegSmem {
    double2 W[3][RMAX];        // multipliers of a step, by the step modulo 3
    double2 row[2][RW][CPW];   // each warp's part of a step's pivot row, by its parity
    double2 scale[2][RNMAX];   // 1 / pivot of each pivot row of a slice, by the slice's parity
    double2 sigL[RNMAX], sigR[RNMAX];
    double gL[RNMAX], gR[RNMAX], kin[RNMAX];
    double red[RW];
    int piv[3];                // pivot row of a step, by the step modulo 3
    int rho[2][RNMAX], kappa[2][RNMAX], cst[2][RNMAX];  // maps of a slice, by its parity
    int unit[RNMAX];           // of the last inverse: the row that was the pivot of each storage column
    int prow[RNMAX], lin[RNMAX], rows[RNMAX], nrows, info;
};

// Ends the body of one of several branches that differ in a register index
// only, so that the compiler does not merge them into one that indexes local
// memory.
template <int I>
__device__ __forceinline__ void reg_keep() { asm volatile("" ::"n"(I)); }

// f(0), ..., f(n - 1) with the index as a compile-time constant.
template <int I>
struct Slot { static constexpr int v = I; };
template <int n, int I = 0, typename F>
__device__ __forceinline__ void each_slot(F f) {
    if constexpr (I < n) {
        f(Slot<I>());
        each_slot<n, I + 1>(f);
    }
}

// The pivot of column k, held by one warp in v (row lane + 32 r in v[r]):
// the unused row with the largest |re|+|im| to 18 bits (the high word of the
// double with the slot in its low bits, one integer reduction; zgetf2's choice
// up to a relative 2^-17).  Each lane takes the reciprocal of its own best
// value while the reduction runs.  Publishes the step's multipliers W
// (W_i = -v_i / pivot, 0 in the pivot row), its row and 1 / pivot; v becomes
// the eliminated column, W (less the 1 of the pivot row: reg_eliminate).
template <int NRL, int PR, typename S>
__device__ __forceinline__ void reg_pivot(double2 (&v)[NRL], unsigned free_rows, int k, int slot, double2 *scale, S &s) {
    const int lane = threadIdx.x & 31;
    int key = -1;
#pragma unroll
    for (int r = 0; r < PR; ++r) {
        int h = __double2hiint(cabs1(v[r]));
        if ((unsigned)h >= 0x7ff80000u) h = 0;  // a NaN, of either sign, ranks as a zero pivot
        key = max(key, (free_rows >> r) & 1u ? (h & ~3) | r : -1);
    }
    // a lane without a candidate takes 1 / 1: no division by zero (slow path)
    double2 best = make_double2(1.0, 0.0);
    const unsigned hot = key < 0 ? 0u : 1u << (key & 3);
#pragma unroll
    for (int r = 0; r < PR; ++r) {
        const bool mine = (hot >> r) & 1u;  // as a bit: equality with r is turned into an indexed load
        best.x = mine ? v[r].x : best.x;
        best.y = mine ? v[r].y : best.y;
    }
    const int top = __reduce_max_sync(0xffffffffu, key);
    double2 d = zrcp(best);
    const int src = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
    d.x = __shfl_sync(0xffffffffu, d.x, src);
    d.y = __shfl_sync(0xffffffffu, d.y, src);
    const int p = src + 32 * (top & 3);
#pragma unroll
    for (int r = 0; r < NRL; ++r) {
        const double2 m = zmul(v[r], d);
        const bool piv = lane + 32 * r == p;
        v[r].x = piv ? 0.0 : -m.x;
        v[r].y = piv ? 0.0 : -m.y;
        s.W[slot][lane + 32 * r] = v[r];
    }
    if (lane == 0) {
        s.piv[slot] = p;
        s.prow[k] = p;
        scale[p] = d;
        if (top < 4 && s.info == 0) s.info = k + 1;
    }
}

// Gauss-Jordan elimination of the N columns of the register block a: row slots
// 0 .. NRL - 1 in use, the block's rows in the first PR of them, the appended
// rows after row N.  Column k of the basis is eliminated at step k, so the
// pivots and the reported info are those of the natural order; cst[k] = (slot
// << 8 | warp) of its storage column.
//
// A step is a += W a(p, :) with W_p = 0: a pivot row is left unscaled, its
// true values are scale[row] times the stored ones from its step on (scaling
// a row commutes with every later step), which the next block's formation
// applies.  The 1 that the pivot row leaves in its own column is left out as
// well: no later step reads it, it would cost the small terms that follow their
// low bits, and as the last term of scale * a + scale it costs no rounding
// (tri_solve of 40 blocks of N = 69: error against 64 bits 0.84 of that of
// scaled rows; with the 1 stored, 1.1 to 1.25 of it).  One barrier per step.  What bounds it is the chain from one pivot
// to the next (about 1900 cycles a step at N = 69, of which the FP64 pipes are
// busy for 470), so the warp that owns the next column brings that column up to
// date, publishes the next multipliers and goes straight to the next barrier;
// the rest of its update follows behind that.
template <int NRL, int PR, int CPW, int RPL, typename S>
__device__ __forceinline__ void reg_eliminate(double2 (&a)[CPW][RPL], int N, const int *cst, double2 *scale, S &s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned free_rows = 0;
#pragma unroll
    for (int r = 0; r < PR; ++r)
        if (lane + 32 * r < N) free_rows |= 1u << r;
    int q = cst[0], qn = N > 1 ? cst[1] : -1;
    auto pivot = [&](auto t, int k, int slot) {
        double2 v[NRL];
#pragma unroll
        for (int r = 0; r < NRL; ++r) v[r] = a[t.v][r];
        reg_pivot<NRL, PR>(v, free_rows, k, slot, scale, s);
#pragma unroll
        for (int r = 0; r < NRL; ++r) a[t.v][r] = v[r];
    };
    // a += W a(p, :) for the step in (slot, par)
    auto update = [&](int slot, int par) {
        double2 w[NRL];
#pragma unroll
        for (int r = 0; r < NRL; ++r) w[r] = s.W[slot][lane + 32 * r];
#pragma unroll
        for (int t = 0; t < CPW; ++t) {
            const double2 x = s.row[par][warp][t];
#pragma unroll
            for (int r = 0; r < NRL; ++r) a[t][r] = zfma(w[r], x, a[t][r]);
        }
    };
    if ((q & 255) == warp)
        each_slot<CPW>([&](auto t) {
            if (q >> 8 == t.v) {
                pivot(t, 0, 0);
                reg_keep<t.v>();
            }
        });
    bool behind = false;  // this warp has yet to apply the step before
    int slot = 0;
    for (int j = 0; j < N; ++j) {
        const int par = j & 1, after = slot == 2 ? 0 : slot + 1;
        const int q2 = j + 2 < N ? cst[j + 2] : -1;
        __syncthreads();
        if (behind) update(slot == 0 ? 2 : slot - 1, par ^ 1);
        behind = false;
        const int p = s.piv[slot], rp = p >> 5;
        double2 *row = s.row[par][warp];
        each_slot<PR>([&](auto r) {
            if (rp == r.v) {  // the same slot for the whole CTA
                if (lane == (p & 31)) {
#pragma unroll
                    for (int t = 0; t < CPW; ++t) row[t] = a[t][r.v];
                    free_rows &= ~(1u << r.v);
                }
                __syncwarp();  // (keeps this a branch: predicated, every slot's stores would issue)
                reg_keep<r.v>();
            }
        });
        if ((q & 255) == warp) {  // the eliminated column is final
            if (lane == 0) row[q >> 8] = make_double2(0.0, 0.0);
            __syncwarp();
        }
        if ((qn & 255) == warp) {
            each_slot<CPW>([&](auto t) {
                if (qn >> 8 == t.v) {
                    const double2 x = row[t.v];
#pragma unroll
                    for (int r = 0; r < NRL; ++r) a[t.v][r] = zfma(s.W[slot][lane + 32 * r], x, a[t.v][r]);
                    pivot(t, j + 1, after);
                    reg_keep<t.v>();
                }
            });
            __syncwarp();
            if (lane == 0) row[qn >> 8] = make_double2(0.0, 0.0);  // this column is done
            __syncwarp();
            behind = true;
        } else {
            update(slot, par);
        }
        q = qn;
        qn = q2;
        slot = after;
    }
}

// M = D_b - inv(previous block) in the registers, element on
// element (grid.f90:236-333), inv = scale a, + scale where a pivot was
// (reg_eliminate); the first block of a sweep is D_b alone.  D_b is
// generated, or read from the explicit blocks Dexp.  One column at a time: its
// PR gathers in flight, few registers beside a.
template <int PR, int CPW, int RPL, typename S>
__device__ __forceinline__ void reg_form(double2 (&a)[CPW][RPL], const Geo &g, const S &s, const int *rho,
                                         const int *kappa, const double2 *scale, int b, double2 E, bool first,
                                         const double2 *Dexp = nullptr) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int N = g.N, Nz = g.Nz;
    const double2 *vs = g.vhat + (size_t)g.W * g.H * b + g.ngx + g.W * g.ngy;
    const double2 *Dk = Dexp + (size_t)N * N * b;
#pragma unroll
    for (int t = 0; t < CPW; ++t) {
        const int c = warp + RW * t;
        if (c < N) {
            const int kc = kappa[c], one = first ? -1 : s.unit[c];
            double2 d[PR];
#pragma unroll
            for (int r = 0; r < PR; ++r) {
                const int m = lane + 32 * r < N ? rho[lane + 32 * r] : -1;
                d[r] = m < 0 ? make_double2(0.0, 0.0) : Dexp ? Dk[m + (size_t)N * kc] : __ldg(vs + (s.lin[m] - s.lin[kc]));
            }
#pragma unroll
            for (int r = 0; r < PR; ++r)
                if (lane + 32 * r < N) {
                    const int m = rho[lane + 32 * r];
                    double2 x = d[r];
                    if (!Dexp) {
                        if (m != kc) x = make_double2(-d[r].x * g.c2, -d[r].y * g.c2);
                        else {  // the diagonal and the lead terms of the end blocks
                            x = make_double2((-(d[r].x + s.kin[m]) + E.x) * g.c2 - 2.0, (-d[r].y + E.y) * g.c2);
                            if (b == 0) x = zadd(x, s.sigL[m]);
                            if (b == Nz - 1) x = zadd(x, s.sigR[m]);
                        }
                    }
                    if (!first) {
                        const double2 sc = scale[lane + 32 * r];
                        if (lane + 32 * r == one) x = zsub(x, sc);
                        x = zfms(sc, a[t][r], x);
                    }
                    a[t][r] = x;
                }
        }
    }
}

// The maps of the inverse, from those of the block (parity sp): the CTA's
// threads together, before the next block is formed.
template <typename S>
__device__ __forceinline__ void reg_remap(S &s, int N, int sp) {
    if (threadIdx.x < N) {
        const int j = threadIdx.x, p = s.prow[j], c = s.cst[sp][j], m = s.rho[sp][p];
        s.rho[sp ^ 1][p] = j;
        s.kappa[sp ^ 1][(c >> 8) * RW + (c & 255)] = m;
        s.unit[(c >> 8) * RW + (c & 255)] = p;
        s.cst[sp ^ 1][m] = c;
    }
    __syncthreads();
}

// One F-mode sweep and its transmission trace (math_kernel.f90:81-128,
// grid.f90:335-385); returns tau (every thread) and the info of the first
// block with a zero pivot.
template <int CPW, int RPL, int PR, typename S>
__device__ double reg_transmission_job(const Geo &g, S &s, double e, int ik, int *info) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = g.N, Nz = g.Nz;
    const double2 E = make_double2(e, g.eta);
    Smem v{};
    v.sigL = s.sigL; v.sigR = s.sigR; v.gL = s.gL; v.gR = s.gR; v.rows = s.rows; v.nrows = &s.nrows;
    job_vectors(g, v, E, e, ik);
    for (int i = tid; i < N; i += RT) {
        const double ax = g.ax[ik * N + i], ay = g.ay[ik * N + i];
        s.kin[i] = (ax * ax + ay * ay) / 2;
        s.lin[i] = g.nx[i] + g.W * g.ny[i];
        s.rho[0][i] = s.kappa[0][i] = i;
        s.cst[0][i] = (i / RW) << 8 | i % RW;
    }
    if (tid == 0) s.info = 0;
    __syncthreads();
    open_rows(N, v);
    __syncthreads();
    const int nr = s.nrows, nrl = (N + nr + 31) / 32;
    double2 a[CPW][RPL];
#pragma unroll
    for (int t = 0; t < CPW; ++t)
#pragma unroll
        for (int r = 0; r < RPL; ++r) {
            const int c = warp + RW * t, i = lane + 32 * r - N;
            a[t][r] = make_double2((i >= 0 && i < nr && c < N && s.rows[i] == c) ? 1.0 : 0.0, 0.0);
        }
    int sp = 0;
    for (int b = Nz - 1; b >= 0; --b) {
        reg_form<PR>(a, g, s, s.rho[sp], s.kappa[sp], s.scale[sp ^ 1], b, E, b == Nz - 1);
        // the code of this job's row count: no tests of slots inside the steps
        each_slot<RPL - PR + 1>([&](auto x) {
            if (nrl == PR + x.v || (x.v == 0 && nrl < PR)) {
                reg_eliminate<PR + x.v, PR>(a, N, s.cst[sp], s.scale[sp], s);
                reg_keep<x.v>();
            }
        });
        reg_remap(s, N, sp);
        sp ^= 1;
    }
    // tau = sum_ij gamma_L,i gamma_R,j |2 dz^2 G_{Nz,1}(i,j)|^2   grid.f90:362-383
    double tau = 0.0;
#pragma unroll
    for (int t = 0; t < CPW; ++t)
#pragma unroll
        for (int r = 0; r < RPL; ++r) {
            const int c = warp + RW * t, i = lane + 32 * r - N;
            if (c < N && i >= 0 && i < nr) {
                const double gx = a[t][r].x * 2.0 * (g.delta * g.delta), gy = a[t][r].y * 2.0 * (g.delta * g.delta);
                tau += s.gL[s.rows[i]] * s.gR[s.kappa[sp][c]] * (gx * gx + gy * gy);
            }
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tau += __shfl_xor_sync(0xffffffffu, tau, o);
    if (lane == 0) s.red[warp] = tau;
    __syncthreads();
    tau = 0.0;
#pragma unroll
    for (int w = 0; w < RW; ++w) tau += s.red[w];
    *info = s.info;
    return tau;
}

}  // namespace negf
