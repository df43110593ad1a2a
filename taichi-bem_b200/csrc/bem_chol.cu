// Blocked Cholesky factorisation N = L L^H of a Hermitian positive definite
// matrix (the column-equilibrated normal matrix of the transmission least
// squares), left in the tile-LU format of bem_lu_factor_tiled so that the
// persistent triangular solve (bem_lu_solve_tiled) and the refinement calls
// take it unchanged.
//
// Right-looking, panels of 1024 columns by default (BEM_TUNE_CHOL_NB), each
// factored in sub-blocks of 64 in FP64:
//   chol64_kernel     the 64 x 64 diagonal block and the inverse of its factor,
//                     both in registers;
//   dmma_gemm_kernel  L21 = A21 L11^{-H} (a product with that inverse) and the
//                     update of the panel's remaining columns, on the FP64
//                     tensor cores (DMMA);
// then the trailing Hermitian rank-1024 update A22 -= L21 L21^H of the lower
// triangle, the step that carries the O(n^3) work:
//   BEM_PREC_FP64   DMMA products (dmma_gemm_kernel, lower tiles only);
//   BEM_PREC_MIXED  tcgen05 products of FP16 hi/lo splits of the panel (the
//                   normal-matrix kernel of bem_lstsq.cu in its update mode),
//                   summed in FP64 and subtracted from the FP64 Schur
//                   complement.  The panels and the Schur complement stay in
//                   FP64; only the products are split, so the factor's error
//                   is that of the ~22-bit products (about 4e-7 of the
//                   update, measured on the normal matrix), not an FP32
//                   accumulation over the n / 256 updates.
// The reference solves this system with torch.linalg.lstsq
// (BEM_manager.py:1049); the factor here preconditions the FP64 iteration of
// bem_lstsq_refine.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "bem_internal.cuh"

namespace {

constexpr int CH_IB = 64;   // diagonal sub-block
constexpr int CH_SP = 256;  // sub-panel width of the panel factorisation
constexpr int CH_NB_DEFAULT = 1024;  // panel width (columns per trailing update; measured 510 / 410 / 384 ms for 256 / 512 / 1024 on the 30722-unknown normal matrix)

struct cd {
    double re, im;
};

template <bool C>
__device__ __forceinline__ cd ld_c(const double* A, int64_t idx) {
    return C ? cd{A[2 * idx], A[2 * idx + 1]} : cd{A[idx], 0.0};
}
template <bool C>
__device__ __forceinline__ void st_c(double* A, int64_t idx, cd v) {
    if (C) {
        A[2 * idx] = v.re;
        A[2 * idx + 1] = v.im;
    } else {
        A[idx] = v.re;
    }
}

// Cholesky of the nb x nb (nb <= 64) diagonal block at A (lower triangle
// read and written), and Linv = L^{-1} (64 x 64, identity beyond nb) into
// inv.  A non-positive or non-finite pivot sets *info to 1 + its global
// column (the first one wins) and is replaced by 1 so the kernel finishes.
//
// One CTA on the factorisation's serial chain, so what counts is the latency
// of a column.  Both triangles live in registers (thread (ty, tx) of a 16 x 16
// grid holds the entries (ty + 16 a, tx + 16 b) of the block and of the
// inverse) and one elimination runs on both: with the unscaled column m_i =
// M[i][j], pivot d and the unscaled row x_c = X[j][c],
//   M[i][c] -= m_i conj(m_c) / d  (i >= c > j),   X[i][c] -= m_i x_c / d  (i > j),
// so the square roots stay off the chain (L[i][j] = m_i / sqrt(d_j), X[i][c]
// / sqrt(d_i), taken at the end) and a column costs one CTA barrier: its
// owners publish the column and the row in one of two shared buffers, the
// others read them while those of the next column are filled.  Blocks that
// the column does not reach are skipped (whole 16 x 16 blocks, so a warp does
// not diverge on it).  Measured (64 x 64 complex, B200): 26 us a block in a factorisation
// against 110 us with the block and the inverse in shared memory, three
// barriers a column, and the inverse built by rows afterwards.
template <bool C>
__global__ void __launch_bounds__(256) chol64_kernel(double* A, int64_t lda, int nb, double* inv, int32_t* info,
                                                     int col0) {
    __shared__ cd s_col[2][CH_IB];
    __shared__ cd s_row[2][CH_IB];
    __shared__ double s_piv[CH_IB];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    cd M[4][4], X[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            X[a][b] = cd{r == c ? 1.0 : 0.0, 0.0};
            M[a][b] = X[a][b];
            if (r < nb && c <= r) M[a][b] = ld_c<C>(A, (int64_t)r * lda + c);
        }
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
        for (int jj = 0; jj < 16; ++jj) {
            const int j = 16 * jb + jj;
            cd* col = s_col[j & 1];
            cd* row = s_row[j & 1];
            if (tx == jj) {
#pragma unroll
                for (int a = jb; a < 4; ++a) col[ty + 16 * a] = M[a][jb];
            }
            if (ty == jj) {
#pragma unroll
                for (int b = 0; b <= jb; ++b) row[tx + 16 * b] = X[jb][b];
            }
            __syncthreads();
            double d = col[j].re;
            if (!(d > 0.0) || !isfinite(d)) {
                if (tid == 0 && j < nb) atomicCAS(info, 0, col0 + j + 1);
                d = 1.0;
            }
            if (tid == 0) s_piv[j] = d;
            const double rd = 1.0 / d;
            cd mi[4];  // m_i / d of this thread's rows below j (0 elsewhere)
#pragma unroll
            for (int a = jb; a < 4; ++a) {
                const bool below = ty + 16 * a > j;
                const cd v = col[ty + 16 * a];
                mi[a] = cd{below ? v.re * rd : 0.0, C && below ? v.im * rd : 0.0};
            }
#pragma unroll
            for (int b = jb; b < 4; ++b) {
                const bool right = tx + 16 * b > j;
                cd v = col[tx + 16 * b];
                if (!right) v = cd{0.0, 0.0};
#pragma unroll
                for (int a = b; a < 4; ++a) {
                    // M -= (m_i / d) conj(m_c)
                    M[a][b].re -= mi[a].re * v.re;
                    if (C) {
                        M[a][b].re -= mi[a].im * v.im;
                        M[a][b].im -= mi[a].im * v.re;
                        M[a][b].im += mi[a].re * v.im;
                    }
                }
            }
#pragma unroll
            for (int b = 0; b <= jb; ++b) {
                const cd v = row[tx + 16 * b];  // zero right of the diagonal
#pragma unroll
                for (int a = jb; a < 4; ++a) {
                    X[a][b].re -= mi[a].re * v.re;
                    if (C) {
                        X[a][b].re += mi[a].im * v.im;
                        X[a][b].im -= mi[a].re * v.im;
                        X[a][b].im -= mi[a].im * v.re;
                    }
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int c = tx + 16 * b;
        const double sc = sqrt(s_piv[c]), rc = 1.0 / sc;
#pragma unroll
        for (int a = b; a < 4; ++a) {
            const int r = ty + 16 * a;
            if (r < nb && c <= r)
                st_c<C>(A, (int64_t)r * lda + c, r == c ? cd{sc, 0.0} : cd{M[a][b].re * rc, M[a][b].im * rc});
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a;
        const double rc = 1.0 / sqrt(s_piv[r]);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int c = tx + 16 * b;
            st_c<C>(inv, r * CH_IB + c, cd{X[a][b].re * rc, X[a][b].im * rc});
        }
    }
}

// C (m x n, ldc) += alpha op(A) op(B) on the FP64 tensor cores (DMMA,
// mma.sync m8n8k4).  op(A) = A (m x k) or A^H (A stored k x m, CONJA); op(B) =
// B (k x n) or B^H (B stored n x k, CONJT).  LOWER skips the tiles strictly
// above the diagonal shifted by `diag`.  blockIdx.z takes the K range [z
// kchunk, (z + 1) kchunk); with more than one range the tiles are added with
// FP64 atomics (split K for thin products).  tri & 1: op(A) is lower
// triangular, tri & 2: op(B) is upper triangular; the K range of a tile then
// ends at its diagonal.
//
// BM x 64 entries per CTA (BM = 64 or 32), eight warps of BM / 2 x 16 (4 or 2 x
// 2 fragments of 8 x 8; complex: four real products per complex one), K in stages of DG_BK that cp.async
// brings straight into shared memory, four (DG_BK = 8) or three (16) deep, one CTA barrier a stage.
// The factorisations call this with K = 64 and 256, so a CTA lives for 8 to 32
// stages: depth, two CTAs per SM and C on its way into L2 are what keep the
// tensor pipe fed.  Long products have half the barriers with DG_BK = 16.  Shared rows are k, entries interleaved; the row strides put the
// fragments' 8-lane (16-byte) or 16-lane (8-byte) phases on distinct banks.
// The fragment layouts of m8n8k4: A[row = lane / 4][k = lane % 4], B[k = lane %
// 4][col = lane / 4], C[row = lane / 4][col = 2 (lane % 4) + {0, 1}].
// Measured (B200, against one stage prefetched in registers and two barriers a
// stage): the trailing updates of a 2999 complex LU (K = 64) 3.3 against 4.0 ms
// (22 against 18 TFLOP/s), those inside the panels of a 7682 complex Cholesky
// (K = 64 and 256) 6.0 against 6.9 ms (5.7 with 32-row tiles where few).
// Long products, against that form: A B of 1500 complex 930 and 932 us (958 in
// stages of 8), A^H B 874 and 1006, A B^H 1015 and 985 us; A^H B of 2500 real 1122 and
// 1149 us (1248 in stages of 8).
constexpr int DG_BM = 64;
constexpr int DG_OVERWRITE = 4;  // flag beside the triangular ones; C may then be A where n <= 64 (a CTA reads only its rows)
template <bool CPLX, int BK>
struct DgTile {
    static constexpr int W = CPLX ? 2 : 1;
    static constexpr int STAGES = BK == 8 ? 4 : 3;
    static constexpr int LD = CPLX ? DG_BM + 2 : DG_BM + 4;  // entries per k row
    static constexpr int OPERAND = BK * LD * W;              // doubles per operand and stage
    static constexpr size_t SMEM = sizeof(double) * 2 * OPERAND * STAGES;
};

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// one entry (complex: aligned 16-byte copy or two of 8) into shared memory, zero when !ok
template <bool CPLX>
__device__ __forceinline__ void cp_entry(double* dst, const double* src, bool ok, bool al) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (CPLX && al) {
        const int bytes = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
        return;
    }
    const int bytes = ok ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    if (CPLX) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + 8), "l"(src + 1), "r"(bytes) : "memory");
}

template <bool CPLX, bool CONJA, bool CONJT, bool LOWER, int BM, int DG_BK>
__global__ void __launch_bounds__(256, 2) dmma_gemm_kernel(double* Cm, int64_t ldc,
                                                            const double* Am, int64_t lda,
                                                            const double* __restrict__ Bm, int64_t ldb, int64_t m,
                                                            int64_t n, int k, double alpha, int64_t diag, int kchunk,
                                                            int tri, int al) {
    using Tile = DgTile<CPLX, DG_BK>;
    constexpr int DG_STAGES = Tile::STAGES;
    constexpr int W = Tile::W, LD = Tile::LD, NP = CPLX ? 2 : 1;
    constexpr int FA = BM / 16;  // fragments of a warp along the rows
    extern __shared__ __align__(16) double dg_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)blockIdx.x * DG_BM;
    if (LOWER && n0 > m0 + BM - 1 + diag) return;
    const int wr = warp & 1, wc = warp >> 1;
    const bool overwrite = (tri & DG_OVERWRITE) != 0;  // C = alpha op(A) op(B)
    const bool vec_c = CPLX && (reinterpret_cast<uintptr_t>(Cm) & 15) == 0;
    double acc[FA][2][NP][2];
    auto c_entry = [&](int a, int b, int e, bool& ok) -> double* {
        const int64_t gr = m0 + BM / 2 * wr + 8 * a + (lane >> 2), gc = n0 + 16 * wc + 8 * b + 2 * (lane & 3) + e;
        ok = gr < m && gc < n;
        return Cm + W * (gr * ldc + gc);
    };
    const int kbeg = (int)blockIdx.z * kchunk;
    int kend = min(k, kbeg + kchunk);
    if (tri & 1) kend = (int)min((int64_t)kend, m0 + BM);
    if (tri & 2) kend = (int)min((int64_t)kend, n0 + DG_BM);
    // an operand's 64 (A: BM) entries x 8 k, two (one) copies per thread, along its rows in memory:
    // stored with k contiguous (A, B^H): eight k of an entry side by side (real: 4 k of 4 entries in 16 lanes,
    // which the row stride puts on distinct banks), and the entry 32 further; otherwise 64 entries of a k, and k + 4
    const int kc = CPLX ? tid & 7 : (tid & 3) | ((tid >> 2) & 4), ec = CPLX ? tid >> 3 : ((tid >> 2) & 3) | ((tid >> 5) << 2);
    const int ks = tid >> 6, es = tid & 63;  // entries contiguous
    const int ka = !CONJA ? kc : (BM == 64 ? ks : tid >> 5), ea = !CONJA ? ec : (BM == 64 ? es : tid & 31);
    const int kb = CONJT ? kc : ks, eb = CONJT ? ec : es;
    // this thread's first entry of the next stage, and the steps to the other ones and along K
    const double* pa = Am + W * (CONJA ? (int64_t)(kbeg + ka) * lda + m0 + ea : (m0 + ea) * lda + kbeg + ka);
    const double* pb = Bm + W * (CONJT ? (n0 + eb) * ldb + kbeg + kb : (int64_t)(kbeg + kb) * ldb + n0 + eb);
    const int64_t ha = W * (CONJA ? 4 : 32) * lda, hb = W * (CONJT ? 32 : 4) * ldb;
    const int64_t ga = CONJA ? 8 * W * lda : 8 * W, gb = CONJT ? 8 * W : 8 * W * ldb;
    int kleft = kend - kbeg;
    auto stage = [&](int slot) {
        double* sA = dg_smem + (size_t)slot * 2 * Tile::OPERAND;
        double* sB = sA + Tile::OPERAND;
#pragma unroll
        for (int g = 0; g < DG_BK; g += 8) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (32 * h < BM) {
                    const int kk = ka + g + (CONJA ? 4 * h : 0), e = ea + (CONJA ? 0 : 32 * h);
                    const bool ok = m0 + e < m && kk < kleft;
                    cp_entry<CPLX>(sA + W * (kk * LD + e), ok ? pa + h * ha : Am, ok, al != 0);
                }
                {
                    const int kk = kb + g + (CONJT ? 0 : 4 * h), e = eb + (CONJT ? 32 * h : 0);
                    const bool ok = n0 + e < n && kk < kleft;
                    cp_entry<CPLX>(sB + W * (kk * LD + e), ok ? pb + h * hb : Bm, ok, al != 0);
                }
            }
            pa += ga;
            pb += gb;
        }
        kleft -= DG_BK;
    };
    const int nk = kend > kbeg ? (kend - kbeg + DG_BK - 1) / DG_BK : 0;
#pragma unroll
    for (int s = 0; s < DG_STAGES - 1; ++s) {
        if (s < nk) stage(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int a = 0; a < FA; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[a][b][p][0] = acc[a][b][p][1] = 0.0;
            // C is added to at the end (not summed onto: its rounding would enter with every
            // product); bring it into L2 meanwhile
            bool ok;
            const double* c = c_entry(a, b, 0, ok);
            if (ok && !overwrite) asm volatile("prefetch.global.L2 [%0];" ::"l"(c));
        }
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DG_STAGES - 2) : "memory");
        __syncthreads();  // stage kt is in; the slot of stage kt - 1 is free
        if (kt + DG_STAGES - 1 < nk) stage((kt + DG_STAGES - 1) % DG_STAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double* sA = dg_smem + (size_t)(kt % DG_STAGES) * 2 * Tile::OPERAND;
        const double* sB = sA + Tile::OPERAND;
#pragma unroll
        for (int k4 = 0; k4 < DG_BK; k4 += 4) {
            const int kr = k4 + (lane & 3);
            double fa[FA][NP], fb[2][NP];
#pragma unroll
            for (int a = 0; a < FA; ++a) {
                const double* e = sA + W * (kr * LD + BM / 2 * wr + 8 * a + (lane >> 2));
                if (CPLX) {
                    const double2 v = *reinterpret_cast<const double2*>(e);
                    fa[a][0] = v.x;
                    fa[a][NP - 1] = CONJA ? -v.y : v.y;
                } else {
                    fa[a][0] = e[0];
                }
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const double* e = sB + W * (kr * LD + 16 * wc + 8 * b + (lane >> 2));
                if (CPLX) {
                    const double2 v = *reinterpret_cast<const double2*>(e);
                    fb[b][0] = v.x;
                    fb[b][NP - 1] = CONJT ? -v.y : v.y;
                } else {
                    fb[b][0] = e[0];
                }
            }
#pragma unroll
            for (int a = 0; a < FA; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    dmma(acc[a][b][0][0], acc[a][b][0][1], fa[a][0], fb[b][0]);
                    if (CPLX) {
                        dmma(acc[a][b][1][0], acc[a][b][1][1], fa[a][0], fb[b][1]);
                        dmma(acc[a][b][0][0], acc[a][b][0][1], -fa[a][1], fb[b][1]);
                        dmma(acc[a][b][1][0], acc[a][b][1][1], fa[a][1], fb[b][0]);
                    }
                }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const bool add = gridDim.z == 1 && !overwrite;
#pragma unroll
    for (int a = 0; a < FA; ++a) {
        double old[2][2][NP];  // one row of fragments: its loads together
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                bool ok;
                const double* c = c_entry(a, b, e, ok);
                if (CPLX && vec_c) {
                    const double2 v = ok && add ? *reinterpret_cast<const double2*>(c) : make_double2(0.0, 0.0);
                    old[b][e][0] = v.x;
                    old[b][e][NP - 1] = v.y;
                } else {
#pragma unroll
                    for (int p = 0; p < NP; ++p) old[b][e][p] = ok && add ? c[p] : 0.0;
                }
            }
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                bool ok;
                double* c = c_entry(a, b, e, ok);
                if (!ok) continue;
                if (gridDim.z > 1) {
#pragma unroll
                    for (int p = 0; p < NP; ++p) atomicAdd(c + p, alpha * acc[a][b][p][e]);
                } else if (CPLX && vec_c) {
                    *reinterpret_cast<double2*>(c) = make_double2(old[b][e][0] + alpha * acc[a][b][0][e],
                                                                  old[b][e][NP - 1] + alpha * acc[a][b][NP - 1][e]);
                } else {
#pragma unroll
                    for (int p = 0; p < NP; ++p) c[p] = old[b][e][p] + alpha * acc[a][b][p][e];
                }
            }
    }
}

// Tile-LU form of L L^H: with D = diag(L) (real, positive),
//   L' = L D^{-1} (unit lower, strictly lower part stored),  U = D L^H,
// so L' U = L L^H.  The diagonal of L is read from dg (copied beforehand);
// each thread takes one strictly lower entry (i, j) and writes both (i, j)
// and (j, i); the diagonal becomes U[j][j] = D_j^2.
template <bool C>
__global__ void chol_to_lu_kernel(double* A, int64_t lda, int n, const double* dg) {
    const int j = blockIdx.y * 16 + (threadIdx.x >> 4);
    const int64_t i0 = (int64_t)blockIdx.x * 16 + (threadIdx.x & 15);
    if (j >= n || i0 >= n) return;
    const int i = (int)i0;
    if (i == j) {
        st_c<C>(A, (int64_t)j * lda + j, cd{dg[j] * dg[j], 0.0});
        return;
    }
    if (i < j) return;
    const cd l = ld_c<C>(A, (int64_t)i * lda + j);
    const double dj = dg[j];
    st_c<C>(A, (int64_t)i * lda + j, cd{l.re / dj, l.im / dj});
    st_c<C>(A, (int64_t)j * lda + i, cd{dj * l.re, -dj * l.im});
}

template <bool C>
__global__ void diag_copy_kernel(const double* A, int64_t lda, int n, double* dg) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) dg[j] = C ? A[2 * ((int64_t)j * lda + j)] : A[(int64_t)j * lda + j];
}

__global__ void iota_kernel(int32_t* piv, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) piv[i] = i;
}

// One launch of dmma_gemm_kernel with tiles of BM x 64; `splits` ranges of K.
template <bool C, bool CONJA, bool CONJT, bool LOWER, int BM, int DG_BK>
int gemm64_launch(bem_ctx* ctx, double* Cm, int64_t ldc, const double* A, int64_t lda, const double* B, int64_t ldb,
                  int64_t m, int64_t n, int k, double alpha, int64_t diag, int tri, int splits, cudaStream_t s) {
    dim3 grid((unsigned)((n + DG_BM - 1) / DG_BM), (unsigned)((m + BM - 1) / BM));
    const int kchunk = (int)(((int64_t)k + splits - 1) / splits + DG_BK - 1) / DG_BK * DG_BK;
    grid.z = (unsigned)(((int64_t)k + kchunk - 1) / kchunk);
    constexpr size_t smem = DgTile<C, DG_BK>::SMEM;
    if (int rc = bem_check_cuda(ctx, cudaFuncSetAttribute(dmma_gemm_kernel<C, CONJA, CONJT, LOWER, BM, DG_BK>,
                                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                "dmma_gemm_kernel smem"))
        return rc;
    // 16-byte copies of complex entries need 16-byte aligned operands
    const int al = ((uintptr_t)A | (uintptr_t)B) % 16 == 0 ? 1 : 0;
    dmma_gemm_kernel<C, CONJA, CONJT, LOWER, BM, DG_BK>
        <<<grid, 256, smem, s>>>(Cm, ldc, A, lda, B, ldb, m, n, k, alpha, diag, kchunk, tri, al);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "dmma_gemm_kernel");
}

// C += alpha op(A) op(B) (see dmma_gemm_kernel); products with fewer tiles
// than two waves of CTAs split K into ranges of at least 512.  Tiles are 64
// rows, or 32 where the 64-row tiles would not fill the SMs once: such a
// product takes one tile's time, and half a tile's is shorter (K = 64
// complex: L21 of the Cholesky 17.0 -> 10.6 us).
template <bool C, bool CONJA, bool CONJT, bool LOWER>
int gemm64x(bem_ctx* ctx, double* Cm, int64_t ldc, const double* A, int64_t lda, const double* B, int64_t ldb,
            int64_t m, int64_t n, int k, double alpha, int64_t diag, cudaStream_t s, int tri = 0) {
    if (m <= 0 || n <= 0 || k <= 0) return BEM_OK;
    if ((m + DG_BM - 1) / DG_BM > 65535) return bem_fail(ctx, BEM_ERR_INVALID, "dmma_gemm_kernel: m too large");
    const int64_t tiles = ((n + DG_BM - 1) / DG_BM) * ((m + DG_BM - 1) / DG_BM);
    int splits = 1;
    if (!LOWER && !(tri & DG_OVERWRITE) && tiles < 2 * (int64_t)ctx->num_sms)
        splits = (int)std::max<int64_t>(1, std::min<int64_t>((2 * ctx->num_sms) / tiles, k / 512));
    if (tiles <= ctx->num_sms && splits == 1)
        return gemm64_launch<C, CONJA, CONJT, LOWER, 32, 8>(ctx, Cm, ldc, A, lda, B, ldb, m, n, k, alpha, diag, tri, 1, s);
    // stages of 16 where the ranges of K are long and B comes in rows (with B^H, 8 is the faster)
    if constexpr (!CONJT && !LOWER)
        if (k / splits >= 512)
            return gemm64_launch<C, CONJA, CONJT, LOWER, 64, 16>(ctx, Cm, ldc, A, lda, B, ldb, m, n, k, alpha, diag, tri,
                                                                 splits, s);
    return gemm64_launch<C, CONJA, CONJT, LOWER, 64, 8>(ctx, Cm, ldc, A, lda, B, ldb, m, n, k, alpha, diag, tri, splits, s);
}

template <bool C, bool CONJT, bool LOWER>
int gemm64(bem_ctx* ctx, double* Cm, int64_t ldc, const double* A, int64_t lda, const double* B, int64_t ldb,
           int64_t m, int64_t n, int k, double alpha, int64_t diag, cudaStream_t s) {
    return gemm64x<C, false, CONJT, LOWER>(ctx, Cm, ldc, A, lda, B, ldb, m, n, k, alpha, diag, s);
}

// The blocked Cholesky.  With X == nullptr the factor is left in tile-LU
// form (piv, dinv); otherwise L stays in the lower triangle and each diagonal
// tile's inverse L_jj^{-1} is written into X's diagonal tile (X, ldx: the
// start of bem_chol_inverse's triangular inverse).
template <bool C>
int chol_t(bem_ctx* ctx, double* A, int64_t n, int64_t lda, bool tensor_cores, int32_t* piv, double* dinv,
           int32_t* info, cudaStream_t s, double* X = nullptr, int64_t ldx = 0) {
    const int W = C ? 2 : 1;
    const int ni = (int)n;
    // workspace: the inverse of the current 64 x 64 factor, the diagonal
    const size_t inv_d = (size_t)W * CH_IB * CH_IB;
    if (int rc = bem_ws_reserve(ctx, sizeof(double) * (inv_d + n))) return rc;
    double* inv = static_cast<double*>(ctx->ws);
    double* dg = inv + inv_d;
    if (int rc = bem_check_cuda(ctx, cudaMemsetAsync(info, 0, sizeof(int32_t), s), "chol info")) return rc;
    auto at = [&](int64_t r, int64_t c) { return A + W * (r * lda + c); };
    const int nbw = ctx->tune[BEM_TUNE_CHOL_NB] > 0 ? ctx->tune[BEM_TUNE_CHOL_NB] : CH_NB_DEFAULT;
    for (int64_t k0 = 0; k0 < n; k0 += nbw) {
        const int64_t kb = std::min<int64_t>(nbw, n - k0);
        // the panel in sub-panels of CH_SP columns: 64-wide steps update only
        // their sub-panel's remaining columns (K = 64); the sub-panel then
        // updates the rest of the panel in one product (K = CH_SP)
        for (int64_t s0 = k0; s0 < k0 + kb; s0 += CH_SP) {
        const int64_t sb = std::min<int64_t>(CH_SP, k0 + kb - s0);
        for (int64_t j0 = s0; j0 < s0 + sb; j0 += CH_IB) {
            const int jb = (int)std::min<int64_t>(CH_IB, s0 + sb - j0);
            chol64_kernel<C><<<1, 256, 0, s>>>(at(j0, j0), lda, jb, inv, info, (int)j0);
            ctx->launches++;
            if (int rc = bem_check_cuda(ctx, cudaGetLastError(), "chol64_kernel")) return rc;
            if (X)
                if (int rc = bem_check_cuda(ctx, cudaMemcpy2DAsync(X + W * (j0 * ldx + j0), sizeof(double) * W * ldx,
                                                                   inv, sizeof(double) * W * CH_IB,
                                                                   sizeof(double) * W * jb, jb,
                                                                   cudaMemcpyDeviceToDevice, s),
                                            "diagonal inverse copy"))
                    return rc;
            const int64_t r1 = j0 + jb, m1 = n - r1;
            if (m1 <= 0) continue;
            // L21 = A21 L11^{-H}, in place: a CTA's 64 rows depend on themselves only
            if (int rc = gemm64x<C, false, true, false>(ctx, at(r1, j0), lda, at(r1, j0), lda, inv, CH_IB, m1, jb, jb, 1.0,
                                                        0, s, DG_OVERWRITE))
                return rc;
            // the sub-panel's remaining columns: A[r1:, r1:s0+sb] -= L21 L21[0:w]^H (lower part)
            const int64_t w = s0 + sb - r1;
            if (w > 0)
                if (int rc = gemm64<C, true, true>(ctx, at(r1, r1), lda, at(r1, j0), lda, at(r1, j0), lda, m1, w, jb,
                                                   -1.0, 0, s))
                    return rc;
        }
        // the rest of the panel: A[r3:, r3:k0+kb] -= L_sub L_sub[0:w3]^H (lower part, K = sb)
        const int64_t r3 = s0 + sb, w3 = k0 + kb - r3, m3 = n - r3;
        if (w3 > 0 && m3 > 0)
            if (int rc = gemm64<C, true, true>(ctx, at(r3, r3), lda, at(r3, s0), lda, at(r3, s0), lda, m3, w3,
                                               (int)sb, -1.0, 0, s))
                return rc;
        }
        // trailing Hermitian update of the lower triangle
        const int64_t r2 = k0 + kb, m2 = n - r2;
        if (m2 <= 0) continue;
        if (tensor_cores) {
            if (int rc = bem_herk_tc_update(ctx, C, at(r2, k0), lda, (int)m2, (int)kb, at(r2, r2), lda, s)) return rc;
        } else {
            if (int rc = gemm64<C, true, true>(ctx, at(r2, r2), lda, at(r2, k0), lda, at(r2, k0), lda, m2, m2, (int)kb,
                                               -1.0, 0, s))
                return rc;
        }
    }
    if (X) return BEM_OK;
    // the factor in tile-LU form, identity tile pivots, inverses of the diagonal tiles
    diag_copy_kernel<C><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A, lda, ni, dg);
    const unsigned nb16 = (unsigned)((n + 15) / 16);
    chol_to_lu_kernel<C><<<dim3(nb16, nb16), 256, 0, s>>>(A, lda, ni, dg);
    iota_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(piv, ni);
    ctx->launches += 3;
    if (int rc = bem_check_cuda(ctx, cudaGetLastError(), "chol_to_lu")) return rc;
    return bem_tile_inverses(ctx, C, A, n, lda, dinv, s);
}

// X = L^{-1} for the lower triangle of L (n x n, lda) whose diagonal tiles'
// inverses are already in X's diagonal tiles (the rest of X zero), by the
// recursion on halves (rounded to 64 rows)
//   L = [L11 0; L21 L22],  L^{-1} = [X11 0; -X22 L21 X11  X22],
// the two products on the FP64 tensor cores; ws holds L21 X11.
template <bool C>
int tri_inv_rec(bem_ctx* ctx, const double* L, int64_t lda, double* X, int64_t ldx, int64_t lo, int64_t hi,
                double* ws, cudaStream_t s) {
    const int W = C ? 2 : 1;
    if (hi - lo <= CH_IB) return BEM_OK;
    const int64_t mid = lo + ((hi - lo) / 2 + CH_IB - 1) / CH_IB * CH_IB;
    if (int rc = tri_inv_rec<C>(ctx, L, lda, X, ldx, lo, mid, ws, s)) return rc;
    if (int rc = tri_inv_rec<C>(ctx, L, lda, X, ldx, mid, hi, ws, s)) return rc;
    const int64_t m1 = mid - lo, m2 = hi - mid;
    if (int rc = bem_check_cuda(ctx, cudaMemsetAsync(ws, 0, sizeof(double) * W * m2 * m1, s), "tri_inv ws")) return rc;
    // ws = L21 X11 (X11 lower triangular: the product's K range is all of it)
    if (int rc = gemm64x<C, false, false, false>(ctx, ws, m1, L + W * (mid * lda + lo), lda, X + W * (lo * ldx + lo),
                                                 ldx, m2, m1, (int)m1, 1.0, 0, s))
        return rc;
    // X21 = -X22 ws
    return gemm64x<C, false, false, false>(ctx, X + W * (mid * ldx + lo), ldx, X + W * (mid * ldx + mid), ldx, ws,
                                           m1, m2, m1, (int)m2, -1.0, 0, s);
}

}  // namespace

int bem_dmma_sub(bem_ctx* ctx, bool cplx, double* Cm, const double* A, const double* B, int64_t m, int64_t n, int k,
                 int64_t lda, cudaStream_t s) {
    return cplx ? gemm64x<true, false, false, false>(ctx, Cm, lda, A, lda, B, lda, m, n, k, -1.0, 0, s)
                : gemm64x<false, false, false, false>(ctx, Cm, lda, A, lda, B, lda, m, n, k, -1.0, 0, s);
}

extern "C" int bem_gemm(bem_ctx* ctx, int dtype, int conj_a, int conj_b, int tri, int64_t m, int64_t n, int64_t k,
                        double alpha, const void* A, int64_t lda, const void* B, int64_t ldb, void* Cm, int64_t ldc,
                        void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (m < 0 || n < 0 || k < 0 || k > (1 << 30) || !Cm || ldc < n || (m > 0 && n > 0 && k > 0 && (!A || !B)))
        return bem_fail(ctx, BEM_ERR_INVALID, "gemm: bad arguments");
    if (lda < (conj_a ? m : k) || ldb < (conj_b ? k : n)) return bem_fail(ctx, BEM_ERR_INVALID, "gemm: bad leading dimension");
    if (dtype != BEM_C128 && dtype != BEM_F64) return bem_fail(ctx, BEM_ERR_INVALID, "gemm: dtype must be F64 or C128");
    cudaStream_t s = (cudaStream_t)stream;
    const double* a = (const double*)A;
    const double* b = (const double*)B;
    double* c = (double*)Cm;
    const int kk = (int)k;
    if (tri < 0 || tri > 3) return bem_fail(ctx, BEM_ERR_INVALID, "gemm: tri must be 0..3");
#define BEM_GEMM_CASE(CX, CA, CB) \
    return gemm64x<CX, CA, CB, false>(ctx, c, ldc, a, lda, b, ldb, m, n, kk, alpha, 0, s, tri)
    if (dtype == BEM_C128) {
        if (conj_a) {
            if (conj_b) BEM_GEMM_CASE(true, true, true);
            BEM_GEMM_CASE(true, true, false);
        }
        if (conj_b) BEM_GEMM_CASE(true, false, true);
        BEM_GEMM_CASE(true, false, false);
    }
    if (conj_a) {
        if (conj_b) BEM_GEMM_CASE(false, true, true);
        BEM_GEMM_CASE(false, true, false);
    }
    if (conj_b) BEM_GEMM_CASE(false, false, true);
    BEM_GEMM_CASE(false, false, false);
#undef BEM_GEMM_CASE
}

extern "C" int bem_chol_inverse(bem_ctx* ctx, int dtype, void* A, int64_t n, int64_t lda, void* X, int64_t ldx,
                                int32_t* info, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A || !X || !info || n <= 0 || lda < n || ldx < n || n > (1 << 28))
        return bem_fail(ctx, BEM_ERR_INVALID, "chol_inverse: bad arguments");
    if (dtype != BEM_C128 && dtype != BEM_F64)
        return bem_fail(ctx, BEM_ERR_INVALID, "chol_inverse: A must be F64 or C128");
    cudaStream_t s = (cudaStream_t)stream;
    const bool C = dtype == BEM_C128;
    const int W = C ? 2 : 1;
    if (int rc = bem_check_cuda(ctx, cudaMemset2DAsync(X, sizeof(double) * W * ldx, 0, sizeof(double) * W * n, n, s),
                                "chol_inverse zero"))
        return rc;
    double* a = (double*)A;
    double* x = (double*)X;
    int rc = C ? chol_t<true>(ctx, a, n, lda, false, nullptr, nullptr, info, s, x, ldx)
               : chol_t<false>(ctx, a, n, lda, false, nullptr, nullptr, info, s, x, ldx);
    if (rc) return rc;
    // the recursion's scratch: L21 X11 of the top level, at most (n/2 + 64)^2
    const int64_t h = n / 2 + CH_IB;
    void* ws = nullptr;
    if (int e = bem_big_ws(ctx, sizeof(double) * W * h * h, &ws)) return e;
    return C ? tri_inv_rec<true>(ctx, a, lda, x, ldx, 0, n, (double*)ws, s)
             : tri_inv_rec<false>(ctx, a, lda, x, ldx, 0, n, (double*)ws, s);
}

extern "C" int bem_chol_factor(bem_ctx* ctx, int dtype, void* A, int64_t n, int64_t lda, int method, int32_t* piv,
                               void* dinv, int32_t* info, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A || !piv || !dinv || !info || n <= 0 || lda < n || n > (1 << 28))
        return bem_fail(ctx, BEM_ERR_INVALID, "chol_factor: bad arguments");
    if (dtype != BEM_C128 && dtype != BEM_F64) return bem_fail(ctx, BEM_ERR_INVALID, "chol_factor: A must be F64 or C128");
    if (method != BEM_PREC_MIXED && method != BEM_PREC_FP64)
        return bem_fail(ctx, BEM_ERR_INVALID, "chol_factor: method must be BEM_PREC_MIXED or BEM_PREC_FP64");
    cudaStream_t s = (cudaStream_t)stream;
    const bool tc = method == BEM_PREC_MIXED;
    return dtype == BEM_C128 ? chol_t<true>(ctx, (double*)A, n, lda, tc, piv, (double*)dinv, info, s)
                             : chol_t<false>(ctx, (double*)A, n, lda, tc, piv, (double*)dinv, info, s);
}
