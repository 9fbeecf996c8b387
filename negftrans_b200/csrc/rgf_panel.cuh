// rgf_panel.cuh -- the FP64 sweep with panels in registers and teams of CTAs
// (sm_100a, up to 272 plane waves).
//
// The block lives in global memory (it stays in L2 when one job runs per SM)
// and never moves: storage row i stands for basis row rho[i] and storage
// column c for basis column kappa[c], the next block is formed element on
// element, and the elimination changes the maps only (as in rgf_register.cuh,
// which also explains the appended rows that carry the chain product and the
// unscaled pivot rows).
//
// One inverse = panels of 32 columns.  A panel is eliminated in registers (16
// warps, two columns each, the rows across the lanes, so that a search is one
// warp reduction).  Its steps together are A += V A_old(P, :), P the panel's
// pivot rows, so every other column gets one rank-32 update.  The update keeps
// V in shared memory for the whole pass, stages the pivot rows of 64 columns
// at a time, and every warp runs its own 16 x 16 tiles on the FP64 tensor cores
// with the next tile's old values already on their way into registers: no
// barrier and no exposed load inside a chunk of columns.
//
// Teams: T CTAs (a thread-block cluster) share a job.  While one of them
// brings the next panel up to date and eliminates it, the others update the
// rest of the columns; one cluster barrier per panel.  With fewer jobs than
// SMs this puts the idle SMs to work, and the time of a slice falls to that of
// its panels.
//
// Measured on a B200, N = 221 with 28 channels open: a panel takes 95 thousand
// cycles (a step's chain 3000, its FP64 work 500; 149 thousand from panel to
// panel in a team, with the columns it needs and the cluster barrier), the update of the other 189
// columns 126 thousand alone on the chip (94 thousand at the DMMA rate).  Nine
// jobs of 160 slices 175 -> 86 ms.
#pragma once
#include "rgf_register.cuh"

namespace negf {

constexpr int PT = 512;               // threads per CTA
constexpr int PW = PT / 32;           // warps
constexpr int PB = 32;                // panel columns
constexpr int PCN = 64;               // columns whose pivot rows are staged at once
constexpr int PCP = PCN + 2;          // their pitch: k rows 8 banks apart
constexpr int PROWS = 320;            // most rows (basis and appended) of a block

struct PanelSmem {
    double2 *V;            // [PB][ldv] the panel's factor, k-major
    double2 *B;            // [PB][PCP] pivot rows of a chunk of columns
    // in B's place while a panel is eliminated:
    double2 *mul;          // [3][PROWS] multipliers of a step, by the step modulo 3
    double2 *row;          // [2][PW][2] pivot row of a step, each warp's part
    double2 *scale;        // [2][N] 1 / pivot of each pivot row, by the slice's parity
    double2 *sigL, *sigR;  // [N]
    double *gL, *gR, *kin; // [N]
    double *red;           // [PW]
    int *rho, *kappa, *cst;       // [N] maps of the slice
    int *prow, *lin, *rows, *used;  // [N]
    int *rest;             // [N] columns that a panel updates; between two inverses the pivot row of each storage column
    int *nrows, *info;
    int *piv;              // [3] pivot row of a step, by the step modulo 3
    int ldv;
};

__host__ __device__ inline size_t panel_smem(int N) {
    const size_t n = round_up(N, 4);
    static_assert(3 * PROWS + 4 * PW <= PB * PCP, "the exchange buffers fit in B");
    size_t b = ((size_t)PB * (panel_rows(N) + 2) + (size_t)PB * PCP) * sizeof(double2);
    b += 4 * n * sizeof(double2) + 3 * n * sizeof(double) + PW * sizeof(double) + (8 * n + 8) * sizeof(int);
    return b;
}
// Workspace of a team in double2: the block, two panels' factors and a header.
constexpr int PHEAD = 64;  // double2: next job, then per panel parity info, prow[32], and 1 / pivot[32]
__host__ __device__ inline size_t panel_ws(int N) {
    return (size_t)panel_rows(N) * N + 2 * (size_t)PB * (panel_rows(N) + 2) + 2 * PHEAD;
}

__device__ inline PanelSmem carve_panel(unsigned char *base, int N, int ldv) {
    const int n = round_up(N, 4);
    PanelSmem s;
    s.ldv = ldv;
    s.V = (double2 *)base;
    s.B = s.V + (size_t)PB * (panel_rows(N) + 2);
    s.mul = s.B;
    s.row = s.mul + 3 * PROWS;
    s.scale = s.B + PB * PCP;
    s.sigL = s.scale + 2 * n;
    s.sigR = s.sigL + n;
    s.gL = (double *)(s.sigR + n);
    s.gR = s.gL + n;
    s.kin = s.gR + n;
    s.red = s.kin + n;
    s.rho = (int *)(s.red + PW);
    s.kappa = s.rho + n;
    s.cst = s.kappa + n;
    s.prow = s.cst + n;
    s.lin = s.prow + n;
    s.rows = s.lin + n;
    s.rest = s.rows + n;
    s.used = s.rest + n;
    s.nrows = s.used + n;
    s.info = s.nrows + 1;
    s.piv = s.nrows + 2;
    return s;
}

// The CTAs of a job and the global memory they share.
struct PanelTeam {
    int rank, size;
    double2 *A;     // [N][ld] the block, appended rows from row N
    double2 *Vg;    // [2][PB][ld + 2] published factors
    double2 *head;  // [2][PHEAD]
    int ld;
};

__device__ __forceinline__ void panel_sync(const PanelTeam &t) {
    if (t.size > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    } else {
        __syncthreads();
    }
}

// ------------------------------------------------------------ panel in registers
// The pivot of column k of the basis, held by one warp in v (row lane + 32 r):
// the scheme of reg_pivot, to 16 bits of the magnitude; v becomes the
// multipliers, 0 in the pivot row.
template <int NRL>
__device__ __forceinline__ void panel_pivot(double2 (&v)[NRL], unsigned free_rows, int k, int slot, double2 *scale,
                                            const PanelSmem &s) {
    constexpr int PR = NRL < 9 ? NRL : 9;
    const int lane = threadIdx.x & 31;
    int key = -1;
#pragma unroll
    for (int r = 0; r < PR; ++r) {
        int h = __double2hiint(cabs1(v[r]));
        if ((unsigned)h >= 0x7ff80000u) h = 0;  // a NaN, of either sign, ranks as a zero pivot
        key = max(key, (free_rows >> r) & 1u ? (h & ~15) | r : -1);
    }
    // a lane without a candidate takes 1 / 1: no division by zero (slow path)
    double2 best = make_double2(1.0, 0.0);
    const unsigned hot = key < 0 ? 0u : 1u << (key & 15);
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
    const int p = src + 32 * (top & 15);
#pragma unroll
    for (int r = 0; r < NRL; ++r) {
        const double2 m = zmul(v[r], d);
        const bool piv = lane + 32 * r == p;
        v[r].x = piv ? 0.0 : -m.x;
        v[r].y = piv ? 0.0 : -m.y;
        s.mul[slot * PROWS + lane + 32 * r] = v[r];
    }
    if (lane == 0) {
        s.piv[slot] = p;
        s.prow[k] = p;
        scale[p] = d;
        if (top < 16 && *s.info == 0) *s.info = k + 1;
    }
}

// Eliminates the nb columns of the panel at basis column k0, a[t][r] = (storage
// row lane + 32 r, panel column 16 t + warp).  On return a = V; the pivot rows
// are in s.prow[k0 ..], 1 / pivot in scale.  The scheme is that of
// reg_eliminate: one barrier per step, the owner of the next column first, the
// rest of its update behind the next barrier.
template <int NRL>
__device__ __forceinline__ void panel_factor(double2 (&a)[2][NRL], int N, int k0, int nb, double2 *scale, const PanelSmem &s) {
    constexpr int PR = NRL < 9 ? NRL : 9;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned free_rows = 0;
#pragma unroll
    for (int r = 0; r < PR; ++r)
        if (lane + 32 * r < N && !s.used[lane + 32 * r]) free_rows |= 1u << r;
    auto update = [&](int slot, const double2 *row) {
        const double2 x0 = row[0], x1 = row[1];
#pragma unroll
        for (int r = 0; r < NRL; ++r) {
            const double2 w = s.mul[slot * PROWS + lane + 32 * r];
            a[0][r] = zfma(w, x0, a[0][r]);
            a[1][r] = zfma(w, x1, a[1][r]);
        }
    };
    if (warp == 0) panel_pivot<NRL>(a[0], free_rows, k0, 0, scale, s);
    bool behind = false;
    int slot = 0;
    for (int j = 0; j < nb; ++j) {
        const int par = j & 1, after = slot == 2 ? 0 : slot + 1;
        __syncthreads();
        if (behind) update(slot == 0 ? 2 : slot - 1, s.row + (par ^ 1) * 2 * PW + 2 * warp);
        behind = false;
        const int p = s.piv[slot], rp = p >> 5;
        double2 *row = s.row + par * 2 * PW + 2 * warp;
        each_slot<PR>([&](auto r) {
            if (rp == r.v) {  // the same slot for the whole CTA
                if (lane == (p & 31)) {
                    row[0] = a[0][r.v];
                    row[1] = a[1][r.v];
                    free_rows &= ~(1u << r.v);
                }
                __syncwarp();  // (keeps this a branch: predicated, every slot's stores would issue)
                reg_keep<r.v>();
            }
        });
        if ((j & 15) == warp) {  // the eliminated column is final
            if (lane == 0) row[j >> 4] = make_double2(0.0, 0.0);
            __syncwarp();
        }
        if (j + 1 < nb && ((j + 1) & 15) == warp) {
            each_slot<2>([&](auto t) {
                if ((j + 1) >> 4 == t.v) {
                    const double2 x = row[t.v];
#pragma unroll
                    for (int r = 0; r < NRL; ++r) a[t.v][r] = zfma(s.mul[slot * PROWS + lane + 32 * r], x, a[t.v][r]);
                    panel_pivot<NRL>(a[t.v], free_rows, k0 + j + 1, after, scale, s);
                    reg_keep<t.v>();
                }
            });
            __syncwarp();
            if (lane == 0) row[(j + 1) >> 4] = make_double2(0.0, 0.0);  // this column is done
            __syncwarp();
            behind = true;
        } else {
            update(slot, row);
        }
        slot = after;
    }
    __syncthreads();
}

// Loads, eliminates and publishes the panel at k0: V into shared memory (a
// team of one) or Vg[par] with its pivots (a larger team), the panel's own
// columns V into the block (V + e_p less the 1: reg_eliminate).
template <int NRL>
__device__ __noinline__ void panel_rows_run(const PanelTeam &t, const PanelSmem &s, int N, int R, int k0, double2 *scale,
                                            int par) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = min(PB, N - k0);
    double2 a[2][NRL];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int k = 16 * c + warp;
        const double2 *col = t.A + (size_t)t.ld * (k < nb ? s.cst[k0 + k] : 0);
#pragma unroll
        for (int r = 0; r < NRL; ++r) {
            const int i = lane + 32 * r;
            a[c][r] = (k < nb && i < R) ? __ldcg(col + i) : make_double2(0.0, 0.0);
        }
    }
    __syncthreads();  // B is free: the steps' exchange buffers take its place
    panel_factor<NRL>(a, N, k0, nb, scale, s);
    double2 *V = t.size > 1 ? t.Vg + (size_t)par * PB * (t.ld + 2) : s.V;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int k = 16 * c + warp;
        double2 *col = t.A + (size_t)t.ld * (k < nb ? s.cst[k0 + k] : 0);
#pragma unroll
        for (int r = 0; r < NRL; ++r) {
            const int i = lane + 32 * r;
            if (i < s.ldv - 2) V[(size_t)k * s.ldv + i] = a[c][r];
            if (k < nb && i < R) col[i] = a[c][r];
        }
    }
    if (t.size > 1) {
        double2 *h = t.head + par * PHEAD;
        if (threadIdx.x < nb) {
            const int p = s.prow[k0 + threadIdx.x];
            ((int *)h)[4 + threadIdx.x] = p;
            h[16 + threadIdx.x] = scale[p];
        }
        if (threadIdx.x == 0) ((int *)h)[0] = *s.info;
    }
}

__device__ inline void panel_run(const PanelTeam &t, const PanelSmem &s, int N, int R, int k0, double2 *scale, int par) {
    if (R <= 128) panel_rows_run<4>(t, s, N, R, k0, scale, par);
    else if (R <= 192) panel_rows_run<6>(t, s, N, R, k0, scale, par);
    else if (R <= 256) panel_rows_run<8>(t, s, N, R, k0, scale, par);
    else if (R <= 288) panel_rows_run<9>(t, s, N, R, k0, scale, par);
    else panel_rows_run<10>(t, s, N, R, k0, scale, par);
}

// ------------------------------------------------------------ rank-32 update
// A(:, c) += V A(prow, c) for the storage columns cols[0 .. n): 16 x 16 warp
// tiles on DMMA, V in shared memory.
__device__ __noinline__ void panel_update(const PanelTeam &t, const PanelSmem &s, const int *cols, int n, int R,
                                          const int *prow, int nb) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int nrt = (R + 15) / 16, ksteps = (nb + 3) / 4;
    double2 *A = t.A;
    const int ld = t.ld;
    // pivot row kk (of this thread) of columns tid / 32 + 16 u of a chunk
    const int kk = tid & 31;
    const int pk = kk < nb ? prow[kk] : -1;
    double2 br[PCN / PW];
    auto fetch = [&](int c0) {
#pragma unroll
        for (int u = 0; u < PCN / PW; ++u) {
            const int c = c0 + warp + PW * u;
            br[u] = (pk >= 0 && c < n) ? __ldcg(A + pk + (size_t)ld * cols[c]) : make_double2(0.0, 0.0);
        }
    };
    fetch(0);
    for (int c0 = 0; c0 < n; c0 += PCN) {
        __syncthreads();  // the chunk before is done with B, V is complete
#pragma unroll
        for (int u = 0; u < PCN / PW; ++u) s.B[kk * PCP + warp + PW * u] = br[u];
        __syncthreads();
        if (c0 + PCN < n) fetch(c0 + PCN);
        const int nct = min(PCN / 16, (n - c0 + 15) / 16), items = nrt * nct;
        double2 cn[2][2][2];
        auto load = [&](int item) {
            const int i0 = item / nct * 16 + g, j0 = c0 + item % nct * 16 + 2 * q;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int i = i0 + 8 * m, j = j0 + 8 * x + e;
                        cn[m][x][e] = (i < R && j < n) ? __ldcg(A + i + (size_t)ld * cols[j]) : make_double2(0.0, 0.0);
                    }
        };
        if (warp < items) load(warp);
        for (int item = warp; item < items; item += PW) {
            double re[2][2][2], im[2][2][2];
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        re[m][x][e] = cn[m][x][e].x;
                        im[m][x][e] = cn[m][x][e].y;
                    }
            if (item + PW < items) load(item + PW);  // in flight while this tile runs
            const double2 *sa = s.V + (size_t)q * s.ldv + item / nct * 16 + g;
            const double2 *sb = s.B + q * PCP + item % nct * 16 + g;
#pragma unroll 2
            for (int k = 0; k < ksteps; ++k) {
                double2 a[2], b[2];
#pragma unroll
                for (int m = 0; m < 2; ++m) a[m] = sa[8 * m];
#pragma unroll
                for (int x = 0; x < 2; ++x) b[x] = sb[8 * x];
                sa += 4 * s.ldv;
                sb += 4 * PCP;
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        dmma(re[m][x][0], re[m][x][1], a[m].x, b[x].x);
                        dmma(im[m][x][0], im[m][x][1], a[m].x, b[x].y);
                    }
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const double na = -a[m].y;
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        dmma(re[m][x][0], re[m][x][1], na, b[x].y);
                        dmma(im[m][x][0], im[m][x][1], a[m].y, b[x].x);
                    }
                }
            }
            const int i0 = item / nct * 16 + g, j0 = c0 + item % nct * 16 + 2 * q;
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = j0 + 8 * x + e;
                    if (j < n) {
                        double2 *col = A + (size_t)ld * cols[j];
#pragma unroll
                        for (int m = 0; m < 2; ++m)
                            if (i0 + 8 * m < R) col[i0 + 8 * m] = make_double2(re[m][x][e], im[m][x][e]);
                    }
                }
        }
    }
    __syncthreads();
}

// In-place Gauss-Jordan inverse of the block (rows N .. R - 1 appended): maps,
// pivots and scales in s.  Every CTA of the team calls it; the block must be
// complete (panel_sync) before.
__device__ inline void panel_invert(const PanelTeam &t, const PanelSmem &s, int N, int R, double2 *scale) {
    const int tid = threadIdx.x;
    for (int i = tid; i < N; i += PT) s.used[i] = 0;
    __syncthreads();
    if (t.rank == 0) panel_run(t, s, N, R, 0, scale, 0);
    panel_sync(t);
    for (int k0 = 0, m = 0; k0 < N; k0 += PB, ++m) {
        const int nb = min(PB, N - k0), par = m & 1;
        if (t.size > 1) {  // take over the published panel
            const double2 *h = t.head + par * PHEAD, *V = t.Vg + (size_t)par * PB * (t.ld + 2);
            if (tid < nb) {
                const int p = __ldcg((const int *)h + 4 + tid);
                s.prow[k0 + tid] = p;
                scale[p] = __ldcg(h + 16 + tid);
            }
            if (tid == 0) *s.info = __ldcg((const int *)h);
            for (int e = tid; e < PB * s.ldv; e += PT) cp_async16(s.V + e, V + e, true);
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
        }
        if (tid < nb) s.used[s.prow[k0 + tid]] = 1;
        // columns to update: the next panel's first, then all others
        const int next = min(PB, N - k0 - nb);
        for (int j = tid; j < N - nb; j += PT) {
            const int b = j < next ? k0 + nb + j : j - next < k0 ? j - next : j + nb;
            s.rest[j] = s.cst[b];
        }
        __syncthreads();
        const int owner = next > 0 ? (m + 1) % t.size : -1;
        int c0, c1;  // this CTA's share
        if (t.size == 1) {
            c0 = 0;
            c1 = N - nb;
        } else if (t.rank == owner) {
            c0 = 0;
            c1 = next;
        } else {
            // the others share the rest in units of 16 columns
            const int lo = owner >= 0 ? next : 0, parts = t.size - (owner >= 0 ? 1 : 0);
            const int me = owner >= 0 && t.rank > owner ? t.rank - 1 : t.rank;
            const int units = (N - nb - lo + 15) / 16;
            c0 = min(N - nb, lo + units * me / parts * 16);
            c1 = min(N - nb, lo + units * (me + 1) / parts * 16);
        }
        if (c1 > c0) panel_update(t, s, s.rest + c0, c1 - c0, R, s.prow + k0, nb);
        if (t.size == 1) {
            if (next > 0) panel_run(t, s, N, R, k0 + nb, scale, 0);
        } else if (t.rank == owner) {
            panel_run(t, s, N, R, k0 + nb, scale, par ^ 1);
        }
        panel_sync(t);
    }
    // the maps of the inverse
    int p = 0, c = 0, b = 0;
    if (tid < N) {
        p = s.prow[tid];
        c = s.cst[tid];
        b = s.rho[p];
    }
    __syncthreads();
    if (tid < N) {
        s.rho[p] = tid;
        s.kappa[c] = b;
        s.cst[b] = c;
        s.rest[c] = p;
    }
    __syncthreads();
}

// ------------------------------------------------------------ the sweep
__device__ inline void panel_vectors(const Geo &g, const PanelSmem &s, double2 E, double e_t, int ik) {
    Smem v{};
    v.sigL = s.sigL; v.sigR = s.sigR; v.gL = s.gL; v.gR = s.gR; v.rows = s.rows; v.nrows = s.nrows;
    job_vectors(g, v, E, e_t, ik);
    for (int i = threadIdx.x; i < g.N; i += PT) {
        const double ax = g.ax[ik * g.N + i], ay = g.ay[ik * g.N + i];
        s.kin[i] = (ax * ax + ay * ay) / 2;
        s.lin[i] = g.nx[i] + g.W * g.ny[i];
    }
    if (threadIdx.x == 0) *s.info = 0;
    __syncthreads();
    open_rows(g.N, v);
    __syncthreads();
}

// The block of slice b, D_b - inv(previous block) in place (grid.f90:236-333);
// first: D_b alone, with the unit rows of `nr` open channels appended.  Columns
// are dealt to the team's warps; a lane's eight rows are in flight together.
__device__ inline void panel_form(const PanelTeam &t, const PanelSmem &s, const Geo &g, int b, double2 E, bool first,
                                  const double2 *scale, const int *rows, int nr) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int N = g.N;
    const double2 *vs = g.vhat + (size_t)g.W * g.H * b + g.ngx + g.W * g.ngy;
    for (int c = warp * t.size + t.rank; c < N; c += PW * t.size) {
        double2 *col = t.A + (size_t)t.ld * c;
        const int kc = s.kappa[c], one = first ? -1 : s.rest[c];
        const double2 *vc = vs - s.lin[kc];
        for (int i0 = 0; i0 < N; i0 += 32 * 8) {
            double2 d[8], x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + lane + 32 * u;
                const bool ok = i < N;
                d[u] = ok ? __ldg(vc + s.lin[s.rho[i]]) : make_double2(0.0, 0.0);
                x[u] = ok && !first ? __ldcg(col + i) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + lane + 32 * u;
                if (i < N) {
                    const int m = s.rho[i];
                    double2 y = make_double2(-d[u].x * g.c2, -d[u].y * g.c2);
                    if (m == kc) {
                        y = make_double2((-(d[u].x + s.kin[m]) + E.x) * g.c2 - 2.0, (-d[u].y + E.y) * g.c2);
                        if (b == 0) y = zadd(y, s.sigL[m]);
                        if (b == g.Nz - 1) y = zadd(y, s.sigR[m]);
                    }
                    if (!first) {
                        const double2 sc = scale[i];
                        if (i == one) y = zsub(y, sc);
                        y = zfms(sc, x[u], y);
                    }
                    col[i] = y;
                }
            }
        }
        if (first)
            for (int i = lane; i < nr; i += 32) col[N + i] = make_double2(rows[i] == c ? 1.0 : 0.0, 0.0);
    }
}

// One F-mode sweep and its transmission trace (math_kernel.f90:81-128,
// grid.f90:335-385), by a team; tau and the info are those of rank 0.  Open
// channels beyond the rows of a block take another pass over the slices.
__device__ inline double panel_transmission_job(const PanelTeam &t, const PanelSmem &s0, const Geo &g, double e, int ik,
                                                int *info) {
    PanelSmem s = s0;
    const int tid = threadIdx.x, N = g.N;
    const double2 E = make_double2(e, g.eta);
    const int n4 = round_up(N, 4);
    panel_vectors(g, s, E, e, ik);
    const int open = *s.nrows;
    double tau = 0.0;
    for (int first = 0; first == 0 || first < open; first += t.ld - N) {
        const int nr = min(open - first, t.ld - N), R = N + nr;
        s.ldv = round_up(R, 8) + 2;
        for (int i = tid; i < N; i += PT) s.rho[i] = s.kappa[i] = s.cst[i] = i;
        __syncthreads();
        int sp = 0;
        for (int b = g.Nz - 1; b >= 0; --b, sp ^= 1) {
            panel_form(t, s, g, b, E, b == g.Nz - 1, s.scale + (sp ^ 1) * n4, s.rows + first, nr);
            panel_sync(t);
            panel_invert(t, s, N, R, s.scale + sp * n4);
        }
        // tau = sum_ij gamma_L,i gamma_R,j |2 dz^2 G_{Nz,1}(i,j)|^2   grid.f90:362-383
        if (t.rank == 0)
            for (int x = tid; x < nr * N; x += PT) {
                const int i = x % nr, c = x / nr;
                const double2 v = __ldcg(t.A + N + i + (size_t)t.ld * c);
                const double gx = v.x * 2.0 * (g.delta * g.delta), gy = v.y * 2.0 * (g.delta * g.delta);
                tau += s.gL[s.rows[first + i]] * s.gR[s.kappa[c]] * (gx * gx + gy * gy);
            }
        panel_sync(t);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tau += __shfl_xor_sync(0xffffffffu, tau, o);
    if ((tid & 31) == 0) s.red[tid >> 5] = tau;
    __syncthreads();
    tau = 0.0;
#pragma unroll
    for (int w = 0; w < PW; ++w) tau += s.red[w];
    *info = *s.info;
    return tau;
}

}  // namespace negf
