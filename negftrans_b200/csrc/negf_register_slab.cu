// negf_register_slab.cu -- the sweeps that keep every generator block, up to 72
// plane waves: inverses in registers (rgf_register.cuh), the products of the
// diagonal and column recursions on the FP64 tensor cores from shared memory.
// The modes, the slab's layout and the recursions are those of k_rgf_slab
// (negf_slab.cu).
//
// What bounds it: the pivot chain of the inverse (about two thirds of a
// slice), then the two products, which run at the DMMA rate from shared memory
// (both operands of a 72 x 72 product fit, so no tile is staged twice).
// Measured on a B200 against k_rgf_slab<16, 1, 2>, N = 69, whole calls: biased
// density of 120 points, N_z = 100, 33.6 -> 20.0 ms; LDOS of 300 energies,
// N_z = 200, 145.6 -> 83.2 ms; D, F and L of 40 explicit blocks 24.0 -> 14.0 ms.
// There a product alone on its SM took 89 thousand cycles (20.5 thousand at the
// DMMA rate): 64 x 64 tiles left most of the 69 rows' second tile empty.
#include "rgf_register.cuh"

namespace negf {
namespace {

constexpr int SP = 74;  // pitch of a shared block: k columns 8 banks apart for the A fragments
constexpr int SC = 72;  // its columns

// The block's inverse in natural order, to out (leading dimension ldo): scale a,
// + scale where a pivot was (reg_eliminate).
template <int PR, int CPW, int RPL, typename S>
__device__ __forceinline__ void reg_store(const double2 (&a)[CPW][RPL], int N, const S &s, const int *rho, const int *kappa,
                                          const double2 *scale, double2 *out, int ldo) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < CPW; ++t) {
        const int c = warp + RW * t;
        if (c < N) {
            double2 *col = out + (size_t)ldo * kappa[c];
            const int one = s.unit[c];
#pragma unroll
            for (int r = 0; r < PR; ++r) {
                const int i = lane + 32 * r;
                if (i < N) {
                    const double2 sc = scale[i];
                    col[rho[i]] = i == one ? zfma(sc, a[t][r], sc) : zmul(sc, a[t][r]);
                }
            }
        }
    }
}

// dst (pitch SP) = the N x nc block src; asynchronous: wait and synchronise after it.
__device__ __forceinline__ void slab_load(double2 *dst, const double2 *src, int ld, int N, int nc) {
    for (int c = threadIdx.x >> 5; c < nc; c += RW)
        for (int i = threadIdx.x & 31; i < N; i += 32) cp_async16(dst + c * SP + i, src + i + (size_t)ld * c, true);
    cp_async_commit();
}

// The 8 x 8 output tiles of a product, dealt to the warps: at most 7 each.
struct SlabAcc {
    double re[7][2], im[7][2];
};

// acc = A B over N x N shared blocks (rows and columns N .. 71 zero); nt = tiles per side.
__device__ __forceinline__ void slab_mma(SlabAcc &acc, const double2 *A, const double2 *B, int nt, int ksteps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    int oa[7], ob[7];
#pragma unroll
    for (int u = 0; u < 7; ++u) {
        const int t = min(warp + RW * u, nt * nt - 1);  // (the tiles past the end repeat the last)
        oa[u] = t % nt * 8 + g + q * SP;
        ob[u] = (t / nt * 8 + g) * SP + q;
        acc.re[u][0] = acc.re[u][1] = acc.im[u][0] = acc.im[u][1] = 0.0;
    }
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (warp + RW * u < nt * nt) {
                const double2 a = A[oa[u] + 4 * k * SP], b = B[ob[u] + 4 * k];
                dmma(acc.re[u][0], acc.re[u][1], a.x, b.x);
                dmma(acc.im[u][0], acc.im[u][1], a.x, b.y);
                dmma(acc.re[u][0], acc.re[u][1], -a.y, b.y);
                dmma(acc.im[u][0], acc.im[u][1], a.y, b.x);
            }
    }
}

// f(row, column, value) over the calling thread's elements of the product.
template <typename F>
__device__ __forceinline__ void slab_each(const SlabAcc &acc, int N, int nt, F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < 7; ++u) {
        const int t = warp + RW * u;
        if (t < nt * nt) {
            const int i = t % nt * 8 + (lane >> 2), j0 = t / nt * 8 + 2 * (lane & 3);
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (i < N && j0 + e < N) f(i, j0 + e, make_double2(acc.re[u][e], acc.im[u][e]));
        }
    }
}

template <int CPW, int RPL>
__global__ void __launch_bounds__(RT, 1)
    k_register_slab(Geo g, const RgfJob *__restrict__ jobs, int njobs, const double2 *__restrict__ Dexp, double2 *ws,
                    size_t wstride, double2 *slabs, size_t sstride, int want, double2 *out_first, double2 *out_last,
                    int *info_jobs) {
    extern __shared__ __align__(256) unsigned char smem[];
    typedef RegSmem<32 * RPL, CPW> S;
    S &s = *(S *)smem;
    double2 *bufA = (double2 *)(smem + (sizeof(S) + 255) / 256 * 256), *bufB = bufA + SP * SC;
    const int job = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (job >= njobs) return;
    const int N = g.N, ld = g.ld, Nz = g.Nz, nt = (N + 7) / 8, ksteps = (N + 3) / 4;
    const size_t NB2 = (size_t)ld * N, NN = (size_t)N * N;
    double2 *Ya = ws + (size_t)job * wstride, *Yb = Ya + NB2;
    double2 *slab = slabs + (size_t)job * sstride;
    const bool mirror = (want & WANT_MIRROR) != 0;
    auto sl = [&](int x) { return mirror ? Nz - 1 - x : x; };
    auto blk = [&](int x) { return slab + NB2 * sl(x); };
    const RgfJob jb = jobs[job];
    const double2 E = make_double2(jb.e_re, jb.e_im);
    Smem v{};
    v.sigL = s.sigL; v.sigR = s.sigR; v.gL = s.gL; v.gR = s.gR; v.rows = s.rows; v.nrows = &s.nrows;
    if (!Dexp) {
        job_vectors(g, v, E, jb.e_t, jb.ik);
        for (int i = tid; i < N; i += RT) {
            const double ax = g.ax[jb.ik * N + i], ay = g.ay[jb.ik * N + i];
            s.kin[i] = (ax * ax + ay * ay) / 2;
            s.lin[i] = g.nx[i] + g.W * g.ny[i];
        }
    }
    for (int e = tid; e < 2 * SP * SC; e += RT) bufA[e] = make_double2(0.0, 0.0);  // the padding stays zero
    if (tid == 0) s.info = 0;

    // The inverses of a sweep over the slices of steps x0, x0 + dx, ... (n of
    // them), each block minus the inverse before; store(x, ...) writes them.
    auto sweep = [&](int x0, int dx, int n, auto target) {
        double2 a[CPW][RPL];
        __syncthreads();
        for (int i = tid; i < N; i += RT) {
            s.rho[0][i] = s.kappa[0][i] = i;
            s.cst[0][i] = (i / RW) << 8 | i % RW;
        }
        __syncthreads();
        for (int y = 0, sp = 0; y < n; ++y, sp ^= 1) {
            const int x = x0 + dx * y;
            reg_form<RPL>(a, g, s, s.rho[sp], s.kappa[sp], s.scale[sp ^ 1], sl(x), E, y == 0, Dexp);
            reg_eliminate<RPL, RPL>(a, N, s.cst[sp], s.scale[sp], s);
            reg_remap(s, N, sp);
            int ldo = ld;
            double2 *out = target(x, ldo);
            reg_store<RPL>(a, N, s, s.rho[sp ^ 1], s.kappa[sp ^ 1], s.scale[sp], out, ldo);
        }
        __syncthreads();
    };
    // dst[k] (blocks of leading dimension N) = -gen(k) dst of the step before
    auto chain = [&](double2 *out, int k0, int dk, auto gen) {
        slab_load(bufB, out + NN * k0, N, N, N);
        for (int y = 1, k = k0 + dk; y < Nz; ++y, k += dk) {
            slab_load(bufA, gen(k), ld, N, N);
            cp_async_wait<0>();
            __syncthreads();
            SlabAcc acc;
            slab_mma(acc, bufA, bufB, nt, ksteps);
            __syncthreads();
            slab_each(acc, N, nt, [&](int i, int j, double2 z) {
                z = make_double2(-z.x, -z.y);
                bufB[j * SP + i] = z;
                out[NN * k + i + (size_t)N * j] = z;
            });
        }
        __syncthreads();
    };

    if (want & (WANT_D | WANT_F)) {
        // generator_r(m) = the inverse at slice m + 1 into block m, G_11 into Yb;
        // math_kernel.f90:81-91
        sweep(Nz - 1, -1, Nz, [&](int x, int &) { return x > 0 ? blk(x - 1) : Yb; });
        if ((want & WANT_F) && out_first) {
            for (int e = tid; e < N * N; e += RT) out_first[e] = Yb[e % N + (size_t)ld * (e / N)];
            __syncthreads();
            // G_k1 = -gR(k-1) G_{k-1,1}, math_kernel.f90:112-129
            chain(out_first, 0, 1, [&](int k) { return slab + NB2 * (k - 1); });
        }
        if (want & WANT_D) {
            // G_kk = gR(k-1) (I + G_{k-1,k-1} gR(k-1)), math_kernel.f90:94-109; block
            // k-1 is replaced by G_{k-1,k-1} once gR(k-1) has been read
            const bool wa = (want & WANT_A) != 0;
            const double2 cd = wa ? make_double2(jb.cd_re, jb.cd_im) : make_double2(1.0, 0.0);
            const double2 ca = make_double2(jb.ca_re, jb.ca_im);
            slab_load(bufA, Yb, ld, N, N);  // G_11
            cp_async_wait<0>();
            int nA = 0;
            if (wa && (ca.x != 0.0 || ca.y != 0.0)) {
                const double *gam = mirror ? s.gR : s.gL;
                __syncthreads();
                open_cols(N, v, gam);
                __syncthreads();
                nA = s.nrows;
                for (int e = tid; e < N * nA; e += RT) {
                    const int i = e % N, j = s.rows[e / N];
                    const double sg = sqrt(gam[j]);
                    const double2 z = bufA[j * SP + i];
                    Ya[e] = make_double2(z.x * sg, z.y * sg);
                }
            }
            __syncthreads();
            double2 *Y = Ya, *Yn = Yb;
            for (int k = 1; k <= Nz; ++k) {
                double2 *out = blk(k - 1);
                SlabAcc acc;
                if (k < Nz) {
                    slab_load(bufB, out, ld, N, N);  // gR(k-1)
                    cp_async_wait<0>();
                }
                __syncthreads();
                // block k-1 of the result: cd G + ca Y Y^H
                for (int c = warp; c < N; c += RW)
                    for (int i = lane; i < N; i += 32) {
                        double2 z = zmul(cd, bufA[c * SP + i]);
                        if (nA) {
                            double2 y = make_double2(0.0, 0.0);
                            for (int m = 0; m < nA; ++m) {
                                const double2 p = Y[i + m * N], q = Y[c + m * N];
                                y = zfma(p, make_double2(q.x, -q.y), y);
                            }
                            z = zfma(ca, y, z);
                        }
                        out[i + (size_t)ld * c] = z;
                    }
                if (k == Nz) break;
                for (int c = warp; c < nA; c += RW)  // Y_k = -gR(k-1) Y_{k-1}
                    for (int i = lane; i < N; i += 32) {
                        double2 z = make_double2(0.0, 0.0);
                        for (int m = 0; m < N; ++m) z = zfms(bufB[m * SP + i], Y[m + c * N], z);
                        Yn[i + c * N] = z;
                    }
                slab_mma(acc, bufA, bufB, nt, ksteps);
                __syncthreads();
                slab_each(acc, N, nt, [&](int i, int j, double2 z) {
                    if (i == j) z.x += 1.0;
                    bufA[j * SP + i] = z;
                });
                __syncthreads();
                slab_mma(acc, bufB, bufA, nt, ksteps);
                __syncthreads();
                slab_each(acc, N, nt, [&](int i, int j, double2 z) { bufA[j * SP + i] = z; });
                double2 *t = Y; Y = Yn; Yn = t;
            }
        }
    }
    if ((want & WANT_L) && out_last) {
        // generator_l and the last column, math_kernel.f90:132-162; the
        // generator_l blocks reuse slab blocks 0..Nz-2 (D/F are done with it)
        sweep(0, 1, Nz, [&](int x, int &ldo) {
            if (x < Nz - 1) return slab + NB2 * x;
            ldo = N;
            return out_last + NN * (Nz - 1);
        });
        chain(out_last, Nz - 1, -1, [&](int k) { return slab + NB2 * k; });
    }
    if (tid == 0 && info_jobs) info_jobs[job] = s.info;
}

template <int CPW, int RPL>
SlabKernel make() {
    return SlabKernel{(const void *)k_register_slab<CPW, RPL>, RT,
                      (sizeof(RegSmem<32 * RPL, CPW>) + 255) / 256 * 256 + 2 * SP * SC * sizeof(double2), 2};
}

}  // namespace

SlabKernel register_slab_kernel(int N) {
    if (N <= 24) return make<2, 1>();
    if (N <= 48) return make<4, 2>();
    return make<6, 3>();
}

}  // namespace negf
