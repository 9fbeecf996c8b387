// negf_slab.cu -- the sweeps that keep every generator block, for the diagonal
// (density, LDOS) and first / last column (tri_solve) blocks (negf.f90:9-113,
// 176-236; math_kernel.f90:44-165).
#include "sweep_kernels.h"

namespace negf {
namespace {

// One job per CTA.  slab (Nz blocks, leading dimension ld) first receives
// the generator_r blocks; with WANT_D it ends up holding G_kk in block k.
// out_first / out_last (leading dimension N) receive G_k1 / G_kNz.
// WANT_A (with WANT_D): block k becomes cd * G_kk + ca * A_k, where
// A_k = G_k1 Gamma_L G_k1^H is the spectral function injected by the left
// lead, restricted to its open channels: Y_1 = G_11(:, open) sqrt(gamma_L),
// Y_k = -gR(k-1) Y_{k-1}, A_k = Y_k Y_k^H (8 n_open N^2 flop per product).
// WANT_MIRROR runs the same recursions with the slices numbered from the
// right end (left-connected generators; the injecting lead is the right
// one), writing every block at its own slice index.  Workspace: 6 blocks.
template <int NB, int RPT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_rgf_slab(Geo g, const RgfJob *__restrict__ jobs, int njobs, const double2 *__restrict__ Dexp,
               double2 *ws, size_t wstride, double2 *slabs, size_t sstride, int want,
               double2 *out_first, double2 *out_last, int *info_jobs) {
    extern __shared__ __align__(256) unsigned char smem[];
    Smem s = carve<NB>(smem, g.N);
    const int N = g.N, ld = g.ld, Nz = g.Nz;
    const size_t NB2 = (size_t)ld * N;  // one workspace block
    const size_t NN = (size_t)N * N;    // one output block
    for (int i = threadIdx.x; i < N; i += NT) { s.nx[i] = g.nx[i]; s.ny[i] = g.ny[i]; }
    __syncthreads();
    const int job = blockIdx.x;
    if (job >= njobs) return;
    double2 *A0 = ws + (size_t)blockIdx.x * wstride;
    double2 *A1 = A0 + NB2, *T0 = A1 + NB2, *T1 = T0 + NB2, *T2 = T1 + NB2, *Zt = T2 + NB2;
    double2 *slab = slabs + (size_t)blockIdx.x * sstride;
    const bool mirror = (want & WANT_MIRROR) != 0;
    // slice of step x, and the slab block that holds it
    auto sl = [&](int x) { return mirror ? Nz - 1 - x : x; };
    auto blk = [&](int x) { return slab + NB2 * sl(x); };
    const RgfJob jb = jobs[job];
    const double2 E = make_double2(jb.e_re, jb.e_im);
    const int ik = jb.ik;
    if (!Dexp) job_vectors(g, s, E, jb.e_t, ik);
    __syncthreads();
    int info = 0, r;
    double2 *cur = A0, *oth = A1;

    if (want & (WANT_D | WANT_F)) {
        // generator_r, math_kernel.f90:81-91
        form_block(cur, g, s, sl(Nz - 1), E, ik, nullptr, Dexp);
        __syncthreads();
        info = gj_invert<NB, RPT>(cur, N, ld, s);
        unpermute(blk(Nz - 2), ld, cur, ld, N, s, 1.0);
        __syncthreads();
        for (int m = Nz - 3; m >= 0; --m) {
            form_block(oth, g, s, sl(m + 1), E, ik, cur, Dexp);
            __syncthreads();
            r = gj_invert<NB, RPT>(oth, N, ld, s);
            if (r && !info) info = r;
            unpermute(blk(m), ld, oth, ld, N, s, 1.0);
            __syncthreads();
            double2 *t = cur; cur = oth; oth = t;
        }
        form_block(oth, g, s, sl(0), E, ik, cur, Dexp);
        __syncthreads();
        r = gj_invert<NB, RPT>(oth, N, ld, s);
        if (r && !info) info = r;
        unpermute(T0, ld, oth, ld, N, s, 1.0);  // T0 = G_11
        __syncthreads();
        if ((want & WANT_F) && out_first) {
            // G_k1 = -gR(k-1) G_{k-1,1}, math_kernel.f90:112-129
            for (int e = threadIdx.x; e < N * N; e += NT) {
                const int i = e % N, j = e / N;
                out_first[e] = T0[i + (size_t)ld * j];
            }
            __syncthreads();
            for (int k = 1; k < Nz; ++k) {
                GemmArgs ga{out_first + NN * k, N, slab + NB2 * (k - 1), ld, nullptr,
                            out_first + NN * (k - 1), N, nullptr, N, N, N, nullptr};
                cta_gemm(ga, s, GEMM_STORE_NEG, g.delta);
                __syncthreads();
            }
        }
        if (want & WANT_D) {
            // G_kk = gR(k-1) (I + G_{k-1,k-1} gR(k-1)), math_kernel.f90:94-109.
            // Block k-1 of the slab is replaced by G_{k-1,k-1} once gR(k-1)
            // has been used for the last time.
            const bool wa = (want & WANT_A) != 0;
            const double2 cd = wa ? make_double2(jb.cd_re, jb.cd_im) : make_double2(1.0, 0.0);
            const double2 ca = make_double2(jb.ca_re, jb.ca_im);
            int nA = 0;
            double2 *Ya = A0, *Yb = A1;  // A0, A1 are free once the sweep is done
            if (wa && (ca.x != 0.0 || ca.y != 0.0)) {
                const double *gam = mirror ? s.gR : s.gL;
                open_cols(N, s, gam);
                __syncthreads();
                nA = *s.nrows;
                for (int e = threadIdx.x; e < N * nA; e += NT) {
                    const int i = e % N, c = e / N, j = s.rows[c];
                    const double sg = sqrt(gam[j]);
                    const double2 v = T0[i + (size_t)ld * j];
                    Ya[e] = make_double2(v.x * sg, v.y * sg);
                }
                __syncthreads();
            }
            // block += ca * Y Y^H, through Zt = Y^H (nA x N)
            auto add_spectral = [&](double2 *dst, const double2 *Y) {
                for (int e = threadIdx.x; e < N * nA; e += NT) {
                    const int i = e % N, c = e / N;
                    Zt[c + (size_t)nA * i] = make_double2(Y[e].x, -Y[e].y);
                }
                __syncthreads();
                GemmArgs ga{dst, ld, Y, N, nullptr, Zt, nA, nullptr, N, N, nA, nullptr, ca};
                cta_gemm(ga, s, GEMM_ADD_SCALED, g.delta);
                __syncthreads();
            };
            double2 *Gc = T0, *Gn = T2;
            for (int k = 1; k < Nz; ++k) {
                double2 *gRk = blk(k - 1);
                if (nA) {
                    GemmArgs gy{Yb, N, gRk, ld, nullptr, Ya, N, nullptr, N, nA, N, nullptr};
                    cta_gemm(gy, s, GEMM_STORE_NEG, g.delta);
                    __syncthreads();
                }
                GemmArgs g1{T1, ld, Gc, ld, nullptr, gRk, ld, nullptr, N, N, N, nullptr};
                cta_gemm(g1, s, GEMM_STORE_ADD_EYE, g.delta);
                __syncthreads();
                GemmArgs g2{Gn, ld, gRk, ld, nullptr, T1, ld, nullptr, N, N, N, nullptr};
                cta_gemm(g2, s, GEMM_STORE, g.delta);
                __syncthreads();
                for (int e = threadIdx.x; e < N * N; e += NT) {
                    const int i = e % N, j = e / N;
                    gRk[i + (size_t)ld * j] = zmul(cd, Gc[i + (size_t)ld * j]);
                }
                __syncthreads();
                if (nA) {
                    add_spectral(gRk, Ya);
                    double2 *t = Ya; Ya = Yb; Yb = t;
                }
                double2 *t = Gc; Gc = Gn; Gn = t;
            }
            double2 *last = blk(Nz - 1);
            for (int e = threadIdx.x; e < N * N; e += NT) {
                const int i = e % N, j = e / N;
                last[i + (size_t)ld * j] = zmul(cd, Gc[i + (size_t)ld * j]);
            }
            __syncthreads();
            if (nA) add_spectral(last, Ya);
        }
    }
    if ((want & WANT_L) && out_last) {
        // generator_l and the last column, math_kernel.f90:132-162; the
        // generator_l blocks reuse slab blocks 0..Nz-2 (D/F are done with it).
        cur = A0; oth = A1;
        form_block(cur, g, s, 0, E, ik, nullptr, Dexp);
        __syncthreads();
        r = gj_invert<NB, RPT>(cur, N, ld, s);
        if (r && !info) info = r;
        unpermute(slab, ld, cur, ld, N, s, 1.0);
        __syncthreads();
        for (int m = 1; m <= Nz - 2; ++m) {
            form_block(oth, g, s, m, E, ik, cur, Dexp);
            __syncthreads();
            r = gj_invert<NB, RPT>(oth, N, ld, s);
            if (r && !info) info = r;
            unpermute(slab + NB2 * m, ld, oth, ld, N, s, 1.0);
            __syncthreads();
            double2 *t = cur; cur = oth; oth = t;
        }
        form_block(oth, g, s, Nz - 1, E, ik, cur, Dexp);
        __syncthreads();
        r = gj_invert<NB, RPT>(oth, N, ld, s);
        if (r && !info) info = r;
        unpermute(out_last + NN * (Nz - 1), N, oth, ld, N, s, 1.0);
        __syncthreads();
        for (int k = 1; k < Nz; ++k) {
            GemmArgs ga{out_last + NN * (Nz - 1 - k), N, slab + NB2 * (Nz - 1 - k), ld, nullptr,
                        out_last + NN * (Nz - k), N, nullptr, N, N, N, nullptr};
            cta_gemm(ga, s, GEMM_STORE_NEG, g.delta);
            __syncthreads();
        }
    }
    if (threadIdx.x == 0 && info_jobs) info_jobs[job] = info;
}

template <int NB, int RPT, int MINB>
SlabKernel make(int N) {
    return SlabKernel{(const void *)k_rgf_slab<NB, RPT, MINB>, NT, smem_bytes<NB, RPT>(N)};
}

}  // namespace

SlabKernel slab_kernel(int N) {
    if (N <= RNMAX) return register_slab_kernel(N);
    if (N <= NT) return make<16, 1, 2>(N);
    if (N <= 2 * NT) return make<16, 2, 1>(N);
    if (N <= 4 * NT) return make<8, 4, 1>(N);
    return SlabKernel{};
}

}  // namespace negf
