// Tile-pivoted LU and barrier-free triangular solves (the low-precision factor
// of the mixed path).
//
// Factorisation, per diagonal block k (LU_T = 64 columns):
//   diag   : one CTA factors the 64x64 diagonal block with partial pivoting
//            restricted to the block's rows;
//   laswp  : the block's row swaps applied to the other columns;
//   U12 = L11^{-1} A12 and L21 = A21 U11^{-1}: one CTA per 64-wide tile,
//            substitution against the factored diagonal block, the tile in
//            registers (one CTA barrier per row or column);
//   update : A22 -= L21 U12 (the trailing GEMM of bem_gemm.cuh).
// After the last block, one launch forms the explicit inverses Linv_k (unit
// lower) and Uinv_k (upper) of every diagonal block (`dinv`, used by the
// solves), one CTA per block, off the factorisation's dependency chain.
// No grid-wide synchronisation is needed.  Pivoting within the diagonal tile
// is weaker than full partial pivoting; the FP64 iterative refinement that
// consumes this factor corrects the difference (and reports non-convergence).
//
// Solve: a persistent kernel in which CTA b owns block rows b, b+P, b+2P...;
// block row k accumulates L_kj x_j for every finished j < k (each value is its
// own ready flag; bounded waits), applies Linv_k and publishes x_k.  Each CTA
// handles its block rows in increasing order and all CTAs are co-resident
// (cooperative launch), so every wait ends.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "bem_gemm.cuh"
#include "bem_internal.cuh"

namespace {

constexpr int LU_T = 64;
constexpr unsigned FLAG_SPIN_CAP = 1u << 22;

template <typename T>
struct CE {
    T re, im;
};

template <typename T, bool C>
__device__ __forceinline__ CE<T> ldE(const T* A, int64_t i) {
    CE<T> e;
    e.re = C ? A[2 * i] : A[i];
    e.im = C ? A[2 * i + 1] : T(0);
    return e;
}
template <typename T, bool C>
__device__ __forceinline__ void stE(T* A, int64_t i, CE<T> e) {
    if (C) {
        A[2 * i] = e.re;
        A[2 * i + 1] = e.im;
    } else {
        A[i] = e.re;
    }
}
template <typename T>
__device__ __forceinline__ CE<T> cmul(CE<T> a, CE<T> b) {
    return CE<T>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
// 1 / a; 0 for zero and NaN (a preconditioner's factor stays finite)
template <bool C, typename T>
__device__ __forceinline__ CE<T> cinv(CE<T> a) {
    if (!C) return CE<T>{fabs(a.re) > T(0) ? T(1) / a.re : T(0), T(0)};
    T d = a.re * a.re + a.im * a.im;
    if (d > T(1e-30) && d < T(1e30)) return CE<T>{a.re / d, -a.im / d};  // the scale off the pivot chain
    const T s = bem_unit_scale(a.re, a.im);
    a = CE<T>{a.re * s, a.im * s};
    d = a.re * a.re + a.im * a.im;
    return d > T(0) ? CE<T>{a.re / d * s, -a.im / d * s} : CE<T>{T(0), T(0)};
}
// x / a over the whole range; a = 0 gives infinities and NaN
template <bool C>
__device__ __forceinline__ CE<double> cdiv(CE<double> x, CE<double> a) {
    if (!C) return CE<double>{x.re / a.re, 0.0};
    const double s = bem_unit_scale(a.re, a.im);
    a = CE<double>{a.re * s, a.im * s};
    const double d = a.re * a.re + a.im * a.im;
    return CE<double>{(x.re * a.re + x.im * a.im) / d * s, (x.im * a.re - x.re * a.im) / d * s};
}

// --------------------------------------------------------------------------
// diagonal tile: GEPP inside the tile; explicit inverses of the factored tiles
// --------------------------------------------------------------------------
// Pivot key of a candidate: |re| + |im| as float bits (monotonic for
// non-negative floats), plus one so that 0 means "no candidate".  NaN counts
// as 0.
template <typename T>
__device__ __forceinline__ unsigned pivot_key(CE<T> v) {
    float a = (float)(fabs(v.re) + fabs(v.im));
    if (!(a == a)) a = 0.0f;
    return __float_as_uint(a) + 1u;
}

constexpr int DIAG_LD = LU_T + 1;  // padded row stride: column reads hit distinct banks
constexpr int DIAG_PW = 8;         // row blocks of tile_inv_kernel
// tile_inv_kernel: the factored block and the inverse being built
constexpr size_t inv_smem_bytes(size_t elem) { return elem * (LU_T * DIAG_LD + LU_T * LU_T); }

// One CTA of 256 threads factors the 64x64 diagonal tile (GEPP restricted to
// the tile's rows).  The tile is on the factorisation's serial chain, so the
// latency of a column is what it costs.  It stays in registers: thread (ty,
// tx) of a 16 x 16 grid holds the entries (ty + 16 a, tx + 16 b).  Per column
// two barriers: its owners publish the column; every warp finds the pivot
// itself (lane l looks at rows l and l + 32; two warp reductions, largest |re|
// + |im|, first position on ties); the pivot row's owners publish that row;
// every thread updates its entries.  Rows do not move: a row carries its
// position and is written to it at the end (the pivots are those of moved
// rows).  Measured (complex FP32, B200): 34 us a tile alone on the GPU against
// 48 us with the tile in shared memory, 8-column panels in registers and three
// barriers a column.  The explicit inverses are formed later, by
// tile_inv_kernel.
template <typename T, bool C>
__global__ void __launch_bounds__(256) tile_diag_kernel(T* A, int64_t lda, int n, int k0, int32_t* piv,
                                                        int32_t* info) {
    __shared__ CE<T> s_col[2][LU_T];
    __shared__ CE<T> s_row[LU_T];
    __shared__ int s_pos[LU_T];
    const int m = min(LU_T, n - k0);
    const int tid = threadIdx.x, lane = tid & 31;
    const int tx = tid & 15, ty = tid >> 4;
    CE<T> M[4][4];
    int done = 0;  // bit a: row ty + 16 a is a pivot row already, or outside the matrix
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (ty + 16 * a >= m) done |= 1 << a;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            M[a][b] = r < m && c < m ? ldE<T, C>(A, (int64_t)(k0 + r) * lda + k0 + c) : CE<T>{T(0), T(0)};
        }
    }
    // positions of rows lane and lane + 32, in every warp; LU_T = not a candidate any more
    int pos0 = lane, pos1 = lane + 32;
    bool free0 = lane < m, free1 = lane + 32 < m;
    int zero = 0;  // 1 + first column whose pivot is zero
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
        const int je = min(16, m - 16 * jb);
        for (int jj = 0; jj < je; ++jj) {
            const int j = 16 * jb + jj;
            CE<T>* col = s_col[j & 1];
            if (tx == jj) {
#pragma unroll
                for (int a = 0; a < 4; ++a) col[ty + 16 * a] = M[a][jb];
            }
            __syncthreads();
            const unsigned key0 = free0 ? pivot_key(col[lane]) : 0u, key1 = free1 ? pivot_key(col[lane + 32]) : 0u;
            const unsigned best = __reduce_max_sync(0xffffffffu, key0 > key1 ? key0 : key1);
            // first position, with the row it belongs to in the low bits
            int cand = 0x7fffffff;
            if (key0 == best && free0) cand = (pos0 << 6) | lane;
            if (key1 == best && free1) cand = min(cand, (pos1 << 6) | (lane + 32));
            cand = __reduce_min_sync(0xffffffffu, cand);
            const int p = cand & 63, pp = cand >> 6;  // pivot row and its position
            if (pos0 == j) pos0 = pp;
            if (pos1 == j) pos1 = pp;
            if (p == lane) {
                pos0 = j;
                free0 = false;
            }
            if (p == lane + 32) {
                pos1 = j;
                free1 = false;
            }
            if (ty == (p & 15)) {
                // selects, not an index: the entries stay in registers
                const int pa = p >> 4;
                done |= 1 << pa;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const CE<T> lo = (pa & 1) ? M[1][b] : M[0][b], hi = (pa & 1) ? M[3][b] : M[2][b];
                    s_row[tx + 16 * b] = (pa & 2) ? hi : lo;
                }
            }
            if (tid == 0) piv[k0 + j] = k0 + pp;
            __syncthreads();
            const CE<T> pv = s_row[j];
            if (!(pv.re != T(0) || pv.im != T(0)) && zero == 0) zero = k0 + j + 1;
            const CE<T> inv = cinv<C>(pv);
            CE<T> l[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                l[a] = cmul(col[ty + 16 * a], inv);
                if ((done >> a) & 1) l[a] = CE<T>{T(0), T(0)};
            }
            // no branches: l = 0 on finished rows, u = 0 left of and on the column
#pragma unroll
            for (int b = jb; b < 4; ++b) {
                CE<T> u = s_row[tx + 16 * b];
                if (b == jb && tx <= jj) u = CE<T>{T(0), T(0)};
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    M[a][b].re -= l[a].re * u.re - (C ? l[a].im * u.im : T(0));
                    if (C) M[a][b].im -= l[a].re * u.im + l[a].im * u.re;
                }
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const bool own = tx == jj && !((done >> a) & 1);
                M[a][jb].re = own ? l[a].re : M[a][jb].re;
                M[a][jb].im = own ? l[a].im : M[a][jb].im;
            }
        }
    }
    if (tid < 32) {
        s_pos[lane] = pos0;
        s_pos[lane + 32] = pos1;
    }
    __syncthreads();
    if (tid == 0 && zero != 0 && *info == 0) *info = zero;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a;
        if (r >= m) continue;
        const int64_t row = (int64_t)(k0 + s_pos[r]) * lda + k0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (tx + 16 * b < m) stE<T, C>(A, row + tx + 16 * b, M[a][b]);
    }
}

// Explicit inverses Linv (unit lower) and Uinv (upper) of every factored
// diagonal block, one CTA per block (blockIdx.x = block), by block
// substitution over DIAG_PW-row blocks against the identity.  Runs once the
// factorisation is complete: later row swaps never touch a diagonal block.
// The inverses are formed and held in D: the factor's own type for the
// preconditioners (a zero pivot's reciprocal is 0, so that they stay finite),
// FP64 for bem_lu_solve.  EXACT: an inverse X that one correction of the solve
// does not bring to the accuracy of substitution is written as NaN, which the
// solve looks for.  The correction squares the relative residual of the first
// product, a few eps |T||X|: up to 2^24 that leaves (4 * 1.1e-16 * 2^24)^2 =
// 5e-17.  A zero pivot, or an inverse that overflows, fails the same test.
constexpr double INV_COND_MAX = 16777216.0;
template <typename T, bool C, typename D, bool EXACT>
__global__ void __launch_bounds__(256) tile_inv_kernel(const T* A, int64_t lda, int n, CE<D>* dinv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CE<D>* S = reinterpret_cast<CE<D>*>(smem_raw);  // [LU_T][DIAG_LD] factored block
    CE<D>* X = S + LU_T * DIAG_LD;                  // [LU_T][LU_T] inverse being built
    const int k0 = blockIdx.x * LU_T;
    const int m = min(LU_T, n - k0);
    const int tid = threadIdx.x;
    for (int e = tid; e < LU_T * LU_T; e += blockDim.x) {
        const int r = e / LU_T, c = e - r * LU_T;
        CE<D> v = CE<D>{D(0), D(0)};
        if (r < m && c < m) {
            const CE<T> t = ldE<T, C>(A, (int64_t)(k0 + r) * lda + k0 + c);
            v = CE<D>{(D)t.re, (D)t.im};
        }
        S[r * DIAG_LD + c] = v;
    }
    __syncthreads();
    CE<D>* out = dinv + (size_t)blockIdx.x * 2 * LU_T * LU_T;
    // ---- explicit inverses by block substitution against the identity ----
    // Linv: for row block i: X_i = L_ii^{-1} (E_i - sum_{k<i} L_ik X_k)
    // Uinv: for row block i (descending): X_i = U_ii^{-1} (E_i - sum_{k>i} U_ik X_k)
    // thread: column c = tid & 63, rows (tid >> 6) * 2 + {0, 1} of the block
    __shared__ CE<D> s_rdiag[LU_T];  // 1 / U[r][r], formed in parallel off the substitution chain
    __shared__ D s_sum[EXACT ? LU_T : 1];
    if (tid < LU_T) {
        CE<D> v{D(1), D(0)};
        if (tid < m) {
            if constexpr (EXACT)
                v = cdiv<C>(v, S[tid * DIAG_LD + tid]);
            else
                v = cinv<C>(S[tid * DIAG_LD + tid]);
        }
        s_rdiag[tid] = v;
    }
    const int c = tid & 63, rq = (tid >> 6) * 2;
    for (int which = 0; which < 2; ++which) {
        for (int bs = 0; bs < LU_T / DIAG_PW; ++bs) {
            const int ib = which == 0 ? bs : LU_T / DIAG_PW - 1 - bs;
            const int r0 = ib * DIAG_PW;
            // T = E_i - sum over finished blocks, two rows per thread
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + rq + h;
                CE<D> v = CE<D>{r == c ? D(1) : D(0), D(0)};
                if (r < m) {
                    if (which == 0) {
                        for (int q = 0; q < r0; ++q) {
                            const CE<D> l = S[r * DIAG_LD + q], x = X[q * LU_T + c];
                            v.re -= l.re * x.re - l.im * x.im;
                            v.im -= l.re * x.im + l.im * x.re;
                        }
                    } else {
                        for (int q = r0 + DIAG_PW; q < m; ++q) {
                            const CE<D> uu = S[r * DIAG_LD + q], x = X[q * LU_T + c];
                            v.re -= uu.re * x.re - uu.im * x.im;
                            v.im -= uu.re * x.im + uu.im * x.re;
                        }
                    }
                }
                X[r * LU_T + c] = v;
            }
            __syncthreads();
            // diagonal block: substitution down (Linv) or up (Uinv) the 8 rows, one thread per column
            if (tid < LU_T) {
                CE<D> y[DIAG_PW];
#pragma unroll
                for (int i = 0; i < DIAG_PW; ++i) y[i] = X[(r0 + i) * LU_T + c];
                if (which == 0) {
#pragma unroll
                    for (int i = 0; i < DIAG_PW; ++i) {
                        const int r = r0 + i;
                        if (r >= m) {
                            y[i] = CE<D>{r == c ? D(1) : D(0), D(0)};  // identity padding of a short last tile
                            continue;
                        }
#pragma unroll
                        for (int q = 0; q < i; ++q) {
                            const CE<D> l = S[r * DIAG_LD + r0 + q];
                            y[i].re -= l.re * y[q].re - l.im * y[q].im;
                            y[i].im -= l.re * y[q].im + l.im * y[q].re;
                        }
                    }
                } else {
#pragma unroll
                    for (int i = DIAG_PW - 1; i >= 0; --i) {
                        const int r = r0 + i;
                        if (r >= m) {
                            y[i] = CE<D>{r == c ? D(1) : D(0), D(0)};
                            continue;
                        }
                        if (c >= m) {
                            y[i] = CE<D>{D(0), D(0)};
                            continue;
                        }
#pragma unroll
                        for (int q = i + 1; q < DIAG_PW; ++q) {
                            if (r0 + q >= m) continue;
                            const CE<D> uu = S[r * DIAG_LD + r0 + q];
                            y[i].re -= uu.re * y[q].re - uu.im * y[q].im;
                            y[i].im -= uu.re * y[q].im + uu.im * y[q].re;
                        }
                        y[i] = cmul(y[i], s_rdiag[r]);
                    }
                }
#pragma unroll
                for (int i = 0; i < DIAG_PW; ++i) X[(r0 + i) * LU_T + c] = y[i];
            }
            __syncthreads();
        }
        bool good = true;
        if constexpr (EXACT) {
            // the largest row sum of |T| |X| (thread: row tid / 4, every fourth column)
            const int r = tid >> 2, p = tid & 3;
            D sum = D(0);
            for (int q = p; q < LU_T; q += 4) sum += fabs(X[r * LU_T + q].re) + fabs(X[r * LU_T + q].im);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (p == 0) s_sum[r] = sum;
            __syncthreads();
            sum = p == 0 && which == 0 ? s_sum[r] : D(0);  // L's unit diagonal
            for (int q = p; q < LU_T; q += 4) {
                const CE<D> t = S[r * DIAG_LD + q];
                if (which == 0 ? q < r : q >= r) sum += (fabs(t.re) + fabs(t.im)) * s_sum[q];
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            good = !__syncthreads_or(!(sum <= D(INV_COND_MAX)));
        }
        for (int e = tid; e < LU_T * LU_T; e += blockDim.x)
            out[which * LU_T * LU_T + e] = good ? X[e] : CE<D>{D(NAN), D(NAN)};
        __syncthreads();
    }
}

template <typename T, bool C>
__global__ void tile_laswp_kernel(T* A, int64_t lda, int n, int k0, int m, const int32_t* piv) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n || (c >= k0 && c < k0 + m)) return;
    for (int j = 0; j < m; ++j) {
        int r1 = k0 + j, r2 = piv[k0 + j];
        if (r1 == r2) continue;
        CE<T> a = ldE<T, C>(A, (int64_t)r1 * lda + c);
        CE<T> b = ldE<T, C>(A, (int64_t)r2 * lda + c);
        stE<T, C>(A, (int64_t)r1 * lda + c, b);
        stE<T, C>(A, (int64_t)r2 * lda + c, a);
    }
}

// blockIdx.y = 0: U12 tile (rows k0.., 64 columns) <- L11^{-1} tile (unit lower)
// blockIdx.y = 1: L21 tile (64 rows, columns k0..) <- tile U11^{-1} (upper)
// Both run in one launch (they touch disjoint parts of A).  The factored
// diagonal block is in shared memory, the tile in registers (thread (ty, tx) of
// a 16 x 16 grid holds the entries (ty + 16 a, tx + 16 b)); the substitution
// goes row by row (mode 0) or column by column (mode 1): the owners publish
// the finished row (column) in one of two buffers, one barrier, and every
// thread takes it off its entries below (right of) it.  Measured (complex FP32,
// B200): 22 us a launch against 26 us in blocks of eight out of shared
// memory, a block's triangle solved by one thread per column.
constexpr int APPLY_LD = LU_T + 1;
constexpr size_t apply_smem_bytes(size_t elem) { return elem * LU_T * APPLY_LD; }

template <typename T, bool C>
__global__ void __launch_bounds__(256) tile_apply_kernel(T* A, int64_t lda, int n, int k0, int m) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CE<T>* D = reinterpret_cast<CE<T>*>(smem_raw);  // [LU_T][APPLY_LD] factored diagonal block
    __shared__ CE<T> s_rdiag[LU_T];
    __shared__ CE<T> s_vec[2][LU_T];
    const int mode = blockIdx.y;
    const int base = k0 + m + blockIdx.x * LU_T;  // first column (mode 0) / row (mode 1) of the tile
    const int cnt = min(LU_T, n - base);
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int rows = mode == 0 ? m : cnt, cols = mode == 0 ? cnt : m;
    T* tile = A + (C ? 2 : 1) * (mode == 0 ? (int64_t)k0 * lda + base : (int64_t)base * lda + k0);
    CE<T> X[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            X[a][b] = r < rows && c < cols ? ldE<T, C>(tile, (int64_t)r * lda + c) : CE<T>{T(0), T(0)};
        }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            const CE<T> d = r < m && c < m ? ldE<T, C>(A, (int64_t)(k0 + r) * lda + k0 + c) : CE<T>{T(0), T(0)};
            D[r * APPLY_LD + c] = d;
            if (r == c) s_rdiag[r] = r < m ? cinv<C>(d) : CE<T>{T(0), T(0)};
        }
    __syncthreads();
    if (mode == 0) {
#pragma unroll
        for (int jb = 0; jb < 4; ++jb) {
            const int je = min(16, m - 16 * jb);
            for (int jj = 0; jj < je; ++jj) {
                const int j = 16 * jb + jj;
                CE<T>* v = s_vec[j & 1];
                if (ty == jj) {
#pragma unroll
                    for (int b = 0; b < 4; ++b) v[tx + 16 * b] = X[jb][b];
                }
                __syncthreads();
#pragma unroll
                for (int a = jb; a < 4; ++a) {
                    const int r = ty + 16 * a;
                    if (r <= j) continue;
                    const CE<T> l = D[r * APPLY_LD + j];
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const CE<T> u = v[tx + 16 * b];
                        X[a][b].re -= l.re * u.re - (C ? l.im * u.im : T(0));
                        if (C) X[a][b].im -= l.re * u.im + l.im * u.re;
                    }
                }
            }
        }
    } else {
#pragma unroll
        for (int jb = 0; jb < 4; ++jb) {
            const int je = min(16, m - 16 * jb);
            for (int jj = 0; jj < je; ++jj) {
                const int j = 16 * jb + jj;
                CE<T>* v = s_vec[j & 1];
                if (tx == jj) {
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        X[a][jb] = cmul(X[a][jb], s_rdiag[j]);
                        v[ty + 16 * a] = X[a][jb];
                    }
                }
                __syncthreads();
#pragma unroll
                for (int b = jb; b < 4; ++b) {
                    const int c = tx + 16 * b;
                    if (c <= j) continue;
                    const CE<T> u = D[j * APPLY_LD + c];
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const CE<T> l = v[ty + 16 * a];
                        X[a][b].re -= l.re * u.re - (C ? l.im * u.im : T(0));
                        if (C) X[a][b].im -= l.re * u.im + l.im * u.re;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            if (r < rows && c < cols) stE<T, C>(tile, (int64_t)r * lda + c, X[a][b]);
        }
}

// --------------------------------------------------------------------------
// barrier-free triangular solves
// --------------------------------------------------------------------------
// The solution vectors start out as BEM_PENDING (pending_kernel); a value is its
// own ready flag.
__device__ __forceinline__ double ld_vol(const double* p) {
    double v;
    asm volatile("ld.volatile.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_vol(double* p, double v) {
    asm volatile("st.volatile.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// x = U^{-1} L^{-1} b for NR right-hand sides (FP64, real or complex
// interleaved, vs doubles apart; b already permuted), y the intermediate;
// y and x are BEM_PENDING on entry.  Persistent: CTA b owns block rows b, b + P,
// ... of each pass (forward with L into y, backward with U into x), all CTAs
// are co-resident (cooperative launch) and wait only for rows earlier in the
// pass's order, so every wait ends; the waits are bounded all the same.
//
// What bounds it is the chain of 2 n / 64 block rows, each waiting for the one
// before; the factor's bytes stream beside it.  So per hop there is one trip
// through L2 and nothing else: the consumer polls the 64 values themselves (no
// fence, flag and second read), the block of that last dependency, the
// diagonal inverse (and, REF, the diagonal block) are already in shared
// memory, and the blocks of the earlier dependencies are loaded into registers
// before their values are waited for.  Measured (B200, one right-hand side,
// against a ready flag per block row and the loads after it): complex FP64
// 2999 rows 228 against 505 us, 7682 rows 612 against 1510 us; complex FP32
// 5120 rows 334 against 543 us.  With REF, against one CTA solving each
// diagonal block between grid barriers: 2999 complex, three right-hand sides,
// 0.84 against 5.2 ms.
//
// Sums over the streamed blocks are held in ACC: the factor's own type for the
// preconditioners (as the products of an FP32 factor are), FP64 with REF.  REF
// (the solves of a partial-pivoting factor): the explicit inverse, in FP64
// whatever the factor's type, is corrected once against the diagonal block
// itself, y0 = D a, y = y0 + D (a - T y0), which brings its backward error to
// that of substitution.  Where that is not finite (an inverse that
// tile_inv_kernel did not accept, infinities and NaN of the right-hand side)
// the block is solved by substitution instead, so the solve has the range of
// substitution too.
constexpr int SOLVE_LD = LU_T + 4;  // padded row stride of the staged blocks
constexpr int SMALL_LD = LU_T + 1;  // of small_solve_kernel's tile
// elem, inv: bytes of an element of the factor and of the diagonal inverses
constexpr size_t solve_smem_bytes(size_t elem, size_t inv, bool ref) {
    return ((ref ? 2 : 1) * elem + inv) * LU_T * SOLVE_LD;
}

// type of the diagonal inverses of a solve
template <typename T, bool REF>
struct SolveInv {
    using type = typename std::conditional<REF, double, T>::type;
};

template <typename T, bool C, int NR, bool REF>
__global__ void __launch_bounds__(256) tri_solve_kernel(const T* LU, int64_t lda, int n,
                                                        const CE<typename SolveInv<T, REF>::type>* dinv,
                                                        const double* b, double* y, double* x, int64_t vs,
                                                        int vec, int32_t* err, const int* skip) {
    // skip != NULL: a device word set by the asynchronous refinement once it
    // has converged; the later, already queued solves return at once
    if (skip != nullptr && *skip != 0) return;
    using ACC = typename SolveInv<T, REF>::type;
    constexpr int RW = LU_T / 8;  // rows per warp in the streamed part
    constexpr int W = C ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CE<ACC>* sD = reinterpret_cast<CE<ACC>*>(smem_raw);              // [LU_T][SOLVE_LD] diagonal inverse
    CE<T>* sB = reinterpret_cast<CE<T>*>(sD + LU_T * SOLVE_LD);      // [LU_T][SOLVE_LD] last dependency block
    CE<T>* sT = sB + LU_T * SOLVE_LD;                                // REF: [LU_T][SOLVE_LD] diagonal block
    __shared__ double s_acc[LU_T][NR][2];
    __shared__ double s_x[LU_T][NR][2];
    __shared__ double s_r[REF ? LU_T : 1][NR][2];
    __shared__ int s_abort;
    const int nbk = (n + LU_T - 1) / LU_T;
    const int P = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int gr = tid >> 2, gq = tid & 3;  // GEMV mapping: row gr, columns gq + 4i
    if (tid == 0) s_abort = 0;
    __syncthreads();
    // element i of the row at p (aligned: one access per complex element)
    auto elem = [&](const T* p, int i) -> CE<T> {
        if (C && vec) {
            if constexpr (sizeof(T) == 8) {
                const double2 v = *reinterpret_cast<const double2*>(p + 2 * i);
                return CE<T>{(T)v.x, (T)v.y};
            } else {
                const float2 v = *reinterpret_cast<const float2*>(p + 2 * i);
                return CE<T>{(T)v.x, (T)v.y};
            }
        }
        return ldE<T, C>(p, i);
    };
    // One warp: value c of every right-hand side of v into (re, im), 0 for c >= lim;
    // waits (bounded) until all of the warp's are written.
    auto fetch = [&](const double* v, int base, int c0_, int lim, double (*re)[NR], double (*im)[NR], int cols) -> bool {
        unsigned it = 0;
        for (;;) {
            bool ready = true;
            for (int h = 0; h < cols; ++h) {
                const int c = c0_ + 32 * h;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    double a = 0.0, d = 0.0;
                    if (c < lim) {
                        a = ld_vol(v + r * vs + (int64_t)W * (base + c));
                        if (C) d = ld_vol(v + r * vs + (int64_t)W * (base + c) + 1);
                        ready = ready && !bem_pending(a) && !bem_pending(d);
                    }
                    re[h][r] = a;
                    im[h][r] = d;
                }
            }
            if (__all_sync(0xffffffffu, ready)) return true;
            // lane 0 polls one value; the others wait for it
            int ok = 1;
            if (lane == 0) {
                while (bem_pending(ld_vol(v + (int64_t)W * base))) {
                    if (++it > FLAG_SPIN_CAP) {
                        atomicExch(err, BEM_ERR_TIMEOUT);
                        ok = 0;
                        break;
                    }
                    if ((it & 63u) == 0u && *(volatile int32_t*)err != 0) {
                        ok = 0;
                        break;
                    }
                    if (it > 256u) __nanosleep(32);
                }
                if (++it > FLAG_SPIN_CAP) {
                    atomicExch(err, BEM_ERR_TIMEOUT);
                    ok = 0;
                }
            }
            if (!__shfl_sync(0xffffffffu, ok, 0)) return false;
        }
    };
    for (int pass = 0; pass < 2; ++pass) {
        const bool fwd = pass == 0;
        const double* src = fwd ? b : y;
        double* dst = fwd ? y : x;
        for (int t = blockIdx.x; t < nbk; t += P) {
            const int k = fwd ? t : nbk - 1 - t;
            const int r0 = k * LU_T, m = min(LU_T, n - r0);
            const int ndep = fwd ? k : nbk - 1 - k;
            const int jc = ndep > 0 ? (fwd ? k - 1 : k + 1) : -1;  // critical (last) dependency
            const int nstream = ndep > 0 ? ndep - 1 : 0;           // the others
            auto block = [&](int d) { return fwd ? d : nbk - 1 - d; };
            // the streamed block d: row wid + 8i, columns lane and lane + 32 of each warp
            CE<T> la[RW], lb[RW];
            auto load = [&](int d) {
                const int c0 = block(d) * LU_T, mj = min(LU_T, n - c0);
#pragma unroll
                for (int i = 0; i < RW; ++i) {
                    const int r = wid + 8 * i;
                    const T* row = LU + W * ((int64_t)(r0 + r) * lda + c0);
                    la[i] = (r < m && lane < mj) ? elem(row, lane) : CE<T>{T(0), T(0)};
                    lb[i] = (r < m && lane + 32 < mj) ? elem(row, lane + 32) : CE<T>{T(0), T(0)};
                }
            };
            if (nstream > 0) load(0);
            // stage the diagonal inverse, the critical block and the diagonal block
            const CE<ACC>* Dk = dinv + (size_t)k * 2 * LU_T * LU_T + (fwd ? 0 : LU_T * LU_T);
            for (int e = tid; e < LU_T * LU_T; e += blockDim.x) {
                const int r = e / LU_T, c = e - r * LU_T;
                sD[r * SOLVE_LD + c] = Dk[e];
                const T* row = LU + W * ((int64_t)(r0 + r) * lda);
                CE<T> v = CE<T>{T(0), T(0)};
                if (jc >= 0) {
                    const int c0 = jc * LU_T;
                    if (r < m && c0 + c < n) v = elem(row + (int64_t)W * c0, c);
                }
                sB[r * SOLVE_LD + c] = v;
                if constexpr (REF) {
                    CE<T> d = CE<T>{r == c ? T(1) : T(0), T(0)};
                    if (r < m && c < m && (fwd ? c < r : c >= r)) d = elem(row + (int64_t)W * r0, c);
                    sT[r * SOLVE_LD + c] = d;
                }
            }
            ACC acc_re[RW][NR], acc_im[RW][NR];
#pragma unroll
            for (int i = 0; i < RW; ++i)
#pragma unroll
                for (int r = 0; r < NR; ++r) acc_re[i][r] = acc_im[i][r] = ACC(0);
            bool ok = true;
            for (int d = 0; d < nstream && ok; ++d) {
                const int c0 = block(d) * LU_T;
                double xr[2][NR], xi[2][NR];
                ok = fetch(dst, c0, lane, min(LU_T, n - c0), xr, xi, 2);
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < RW; ++i)
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const ACC x0 = (ACC)xr[0][r], z0 = (ACC)xi[0][r], x1 = (ACC)xr[1][r], z1 = (ACC)xi[1][r];
                        acc_re[i][r] += (ACC)la[i].re * x0;
                        acc_re[i][r] += (ACC)lb[i].re * x1;
                        if (C) {
                            acc_re[i][r] -= (ACC)la[i].im * z0;
                            acc_im[i][r] += (ACC)la[i].re * z0;
                            acc_im[i][r] += (ACC)la[i].im * x0;
                            acc_re[i][r] -= (ACC)lb[i].im * z1;
                            acc_im[i][r] += (ACC)lb[i].re * z1;
                            acc_im[i][r] += (ACC)lb[i].im * x1;
                        }
                    }
                if (d + 1 < nstream) load(d + 1);
            }
            // this row's right-hand side (the forward pass's value in the backward one)
            double br[2][NR], bi[2][NR];
            if (ok) ok = fetch(src, r0, lane, m, br, bi, 2);
            if (!ok && lane == 0) s_abort = 1;
#pragma unroll
            for (int i = 0; i < RW; ++i)
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    ACC sr = acc_re[i][r], si = acc_im[i][r];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        sr += __shfl_xor_sync(0xffffffffu, sr, o);
                        if (C) si += __shfl_xor_sync(0xffffffffu, si, o);
                    }
                    const int q = wid + 8 * i;  // value q sits in lane q % 32, half q / 32
                    if (lane == (q & 31)) {
                        s_acc[q][r][0] = ((i < RW / 2) ? br[0][r] : br[1][r]) - (double)sr;
                        s_acc[q][r][1] = C ? ((i < RW / 2) ? bi[0][r] : bi[1][r]) - (double)si : 0.0;
                    }
                }
            __syncthreads();
            if (s_abort) return;
            // (row gr of S) . v, in A, in all four lanes of the row
            auto gemv = [&](auto zero, const auto* S, const double (*v)[NR][2], double (*out)[2]) {
                using A = decltype(zero);
                A sr[NR], si[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) sr[r] = si[r] = A(0);
#pragma unroll
                for (int i = 0; i < LU_T / 4; ++i) {
                    const int c = gq + 4 * i;
                    const auto l = S[gr * SOLVE_LD + c];
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const A vr = (A)v[c][r][0], vi = (A)v[c][r][1];
                        sr[r] += (A)l.re * vr;
                        if (C) {
                            sr[r] -= (A)l.im * vi;
                            si[r] += (A)l.re * vi;
                            si[r] += (A)l.im * vr;
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    sr[r] += __shfl_xor_sync(0xffffffffu, sr[r], 1);
                    sr[r] += __shfl_xor_sync(0xffffffffu, sr[r], 2);
                    if (C) {
                        si[r] += __shfl_xor_sync(0xffffffffu, si[r], 1);
                        si[r] += __shfl_xor_sync(0xffffffffu, si[r], 2);
                    }
                    out[r][0] = (double)sr[r];
                    out[r][1] = (double)si[r];
                }
            };
            double o[NR][2];
            // critical dependency out of shared memory
            if (jc >= 0) {
                if (wid < 2) {
                    const int c0 = jc * LU_T;
                    double xr[1][NR], xi[1][NR];
                    if (!fetch(dst, c0, 32 * wid + lane, min(LU_T, n - c0), xr, xi, 1)) s_abort = 1;
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        s_x[32 * wid + lane][r][0] = xr[0][r];
                        s_x[32 * wid + lane][r][1] = xi[0][r];
                    }
                }
                __syncthreads();
                if (s_abort) return;
                gemv(ACC(0), sB, s_x, o);
                if (gq == 0 && gr < m)
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        s_acc[gr][r][0] -= o[r][0];
                        s_acc[gr][r][1] -= o[r][1];
                    }
                __syncthreads();
            }
            // inverse(diagonal block) * acc, in FP64
            gemv(0.0, sD, s_acc, o);
            if constexpr (REF) {
                if (gq == 0)
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        s_x[gr][r][0] = o[r][0];
                        s_x[gr][r][1] = o[r][1];
                    }
                __syncthreads();
                double q[NR][2];
                gemv(0.0, sT, s_x, q);
                if (gq == 0)
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        s_r[gr][r][0] = s_acc[gr][r][0] - q[r][0];
                        s_r[gr][r][1] = s_acc[gr][r][1] - q[r][1];
                    }
                __syncthreads();
                gemv(0.0, sD, s_r, q);
                bool finite = true;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    o[r][0] += q[r][0];
                    o[r][1] += q[r][1];
                    if (gr < m) finite = finite && isfinite(o[r][0]) && isfinite(o[r][1]);
                }
                if (__syncthreads_or(!finite)) {
                    // substitution, a warp per right-hand side
                    if (wid < NR)
                        for (int q0 = 0; q0 < m; ++q0) {
                            const int c = fwd ? q0 : m - 1 - q0;
                            const CE<T> d = sT[c * SOLVE_LD + c];
                            CE<double> v{s_acc[c][wid][0], s_acc[c][wid][1]};
                            if (!fwd) v = cdiv<C>(v, CE<double>{(double)d.re, (double)d.im});
                            for (int i = lane; i < m; i += 32) {
                                if (fwd ? i <= c : i >= c) continue;
                                const CE<T> l = sT[i * SOLVE_LD + c];
                                s_acc[i][wid][0] -= (double)l.re * v.re - (C ? (double)l.im * v.im : 0.0);
                                if (C) s_acc[i][wid][1] -= (double)l.re * v.im + (double)l.im * v.re;
                            }
                            if (lane == 0) {
                                s_x[c][wid][0] = v.re;
                                s_x[c][wid][1] = v.im;
                            }
                            __syncwarp();
                        }
                    __syncthreads();
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        o[r][0] = s_x[gr][r][0];
                        o[r][1] = s_x[gr][r][1];
                    }
                }
            }
            if (gq == 0 && gr < m)
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    st_vol(dst + r * vs + (int64_t)W * (r0 + gr), o[r][0]);
                    if (C) st_vol(dst + r * vs + (int64_t)W * (r0 + gr) + 1, o[r][1]);
                }
            __syncthreads();
        }
    }
}

// The same solve for a small matrix (b permuted, x; vs doubles apart): a CTA per
// right-hand side substitutes, tile by tile, with the vector in shared memory.
// There the inverses of the diagonal tiles (49 us, one CTA's chain whatever n)
// and the sweep's hops between CTAs cost more than substitution does, and the
// sweep takes two right-hand sides at a time.  Measured (a whole bem_lu_solve,
// complex FP64, one and eight right-hand sides, the sweep in brackets): 16 rows 53
// and 53 us (82, 147), 80 rows 90 and 89 us (120, 232), 128 rows 115 and 116 us
// (123, 240); 192 rows 164 and 164 us (131, 271), so the sweep goes on from there.
template <typename T, bool C>
__global__ void __launch_bounds__(256) small_solve_kernel(const T* LU, int64_t lda, int n, const double* b, double* x,
                                                          int64_t vs) {
    constexpr int W = C ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CE<double>* sx = reinterpret_cast<CE<double>*>(smem_raw);        // [n]
    CE<T>* sT = reinterpret_cast<CE<T>*>(sx + n);                    // [LU_T][SMALL_LD] diagonal tile
    __shared__ CE<double> s_rd[LU_T];                                // reciprocals of its pivots
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    b += (int64_t)blockIdx.x * vs;
    x += (int64_t)blockIdx.x * vs;
    for (int i = tid; i < n; i += 256) sx[i] = CE<double>{b[W * i], C ? b[W * i + 1] : 0.0};
    const int nbk = (n + LU_T - 1) / LU_T;
    for (int pass = 0; pass < 2; ++pass) {
        const bool fwd = pass == 0;
        for (int t = 0; t < nbk; ++t) {
            const int k0 = (fwd ? t : nbk - 1 - t) * LU_T, m = min(LU_T, n - k0);
            for (int e = tid; e < LU_T * LU_T; e += 256) {
                const int r = e / LU_T, c = e % LU_T;
                if (r < m && c < m) sT[r * SMALL_LD + c] = ldE<T, C>(LU, (int64_t)(k0 + r) * lda + k0 + c);
            }
            __syncthreads();
            if (!fwd) {
                if (tid < m) {
                    const CE<T> u = sT[tid * SMALL_LD + tid];
                    s_rd[tid] = cdiv<C>(CE<double>{1.0, 0.0}, CE<double>{(double)u.re, (double)u.im});
                }
                __syncthreads();
            }
            if (wid == 0) {
                // rows lane and lane + 32 of the tile
                CE<double> v0 = lane < m ? sx[k0 + lane] : CE<double>{0.0, 0.0};
                CE<double> v1 = lane + 32 < m ? sx[k0 + lane + 32] : CE<double>{0.0, 0.0};
                for (int q = 0; q < m; ++q) {
                    const int c = fwd ? q : m - 1 - q;
                    CE<double> p = c < 32 ? v0 : v1;
                    p.re = __shfl_sync(0xffffffffu, p.re, c & 31);
                    if (C) p.im = __shfl_sync(0xffffffffu, p.im, c & 31);
                    if (!fwd) {
                        const CE<double> rd = s_rd[c];
                        if (isfinite(rd.re) && isfinite(rd.im)) {
                            p = CE<double>{p.re * rd.re - (C ? p.im * rd.im : 0.0), C ? p.re * rd.im + p.im * rd.re : 0.0};
                        } else {
                            const CE<T> u = sT[c * SMALL_LD + c];
                            p = cdiv<C>(p, CE<double>{(double)u.re, (double)u.im});
                        }
                        if (lane == (c & 31)) (c < 32 ? v0 : v1) = p;
                    }
                    if (lane < m && (fwd ? lane > c : lane < c)) {
                        const CE<T> l = sT[lane * SMALL_LD + c];
                        v0.re -= (double)l.re * p.re - (C ? (double)l.im * p.im : 0.0);
                        if (C) v0.im -= (double)l.re * p.im + (double)l.im * p.re;
                    }
                    if (lane + 32 < m && (fwd ? lane + 32 > c : lane + 32 < c)) {
                        const CE<T> l = sT[(lane + 32) * SMALL_LD + c];
                        v1.re -= (double)l.re * p.re - (C ? (double)l.im * p.im : 0.0);
                        if (C) v1.im -= (double)l.re * p.im + (double)l.im * p.re;
                    }
                }
                if (lane < m) sx[k0 + lane] = v0;
                if (lane + 32 < m) sx[k0 + lane + 32] = v1;
            }
            __syncthreads();
            // the tile's columns off the rows still to come, a warp per row
            const int r0 = fwd ? k0 + m : 0, r1 = fwd ? n : k0;
            for (int r = r0 + wid; r < r1; r += 8) {
                const T* row = LU + W * ((int64_t)r * lda + k0);
                double sr = 0.0, si = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = lane + 32 * h;
                    if (c >= m) continue;
                    const CE<T> l = ldE<T, C>(row, c);
                    const CE<double> v = sx[k0 + c];
                    sr += (double)l.re * v.re - (C ? (double)l.im * v.im : 0.0);
                    if (C) si += (double)l.re * v.im + (double)l.im * v.re;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    sr += __shfl_xor_sync(0xffffffffu, sr, o);
                    if (C) si += __shfl_xor_sync(0xffffffffu, si, o);
                }
                if (lane == 0) {
                    sx[r].re -= sr;
                    if (C) sx[r].im -= si;
                }
            }
            __syncthreads();
        }
    }
    for (int i = tid; i < n; i += 256) {
        x[W * i] = sx[i].re;
        if (C) x[W * i + 1] = sx[i].im;
    }
}

__global__ void permute_kernel(const double* b, const int32_t* perm, double* out, int n, int W, const int* skip) {
    if (skip != nullptr && *skip != 0) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s = perm[i];
    for (int w = 0; w < W; ++w) out[W * i + w] = bem_not_pending(b[W * s + w]);
}

// y and x start out not written
__global__ void pending_kernel(double* y, double* x, int64_t nd, const int* skip) {
    if (skip != nullptr && *skip != 0) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nd) return;
    y[i] = x[i] = __longlong_as_double((long long)BEM_PENDING);
}

// Queues the triangular solve of NR permuted right-hand sides b (vs doubles
// apart) into x; y is scratch.  err receives BEM_ERR_TIMEOUT if a wait runs out.
template <typename T, bool C, int NR, bool REF>
cudaError_t queue_tri_solve(int sms, const T* LU, int64_t n, int64_t lda, const CE<typename SolveInv<T, REF>::type>* dinv,
                            const double* b, double* y, double* x, int64_t vs, int32_t* err, const int* skip,
                            cudaStream_t s) {
    const int nbk = (int)((n + LU_T - 1) / LU_T);
    const int64_t nd = NR == 1 ? (C ? 2 : 1) * n : NR * vs;
    pending_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, s>>>(y, x, nd, skip);
    const size_t smem = solve_smem_bytes(sizeof(CE<T>), sizeof(*dinv), REF);
    const void* fn = (const void*)tri_solve_kernel<T, C, NR, REF>;
    if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
    int per_sm = 0;
    if (cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tri_solve_kernel<T, C, NR, REF>, 256, smem))
        return e;
    const int P = std::max(1, std::min(nbk, std::min(per_sm * sms, sms)));
    int ni = (int)n;
    int vec = ((uintptr_t)LU % sizeof(CE<T>)) == 0 ? 1 : 0;
    void* args[] = {(void*)&LU, &lda, &ni, (void*)&dinv, (void*)&b, &y, &x, &vs, &vec, &err, (void*)&skip};
    return cudaLaunchCooperativeKernel(fn, P, 256, args, smem, s);
}

// Row permutation of the tile-pivoted factor: every swap of diagonal tile k
// stays inside the tile's rows, so each tile's permutation is built by its own
// thread (64 sequential swaps in registers-free local order).
__global__ void tile_piv_to_perm_kernel(const int32_t* piv, int32_t* perm, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int k0 = k * LU_T;
    if (k0 >= n) return;
    const int m = min(LU_T, n - k0);
    for (int i = 0; i < m; ++i) perm[k0 + i] = k0 + i;
    for (int i = 0; i < m; ++i) {
        const int p = piv[k0 + i];
        if (p != k0 + i && p >= k0 && p < k0 + m) {
            const int t = perm[k0 + i];
            perm[k0 + i] = perm[p];
            perm[p] = t;
        }
    }
}

template <typename T, bool C>
int factor_t(bem_ctx* ctx, T* A, int64_t n, int64_t lda, int32_t* piv, CE<T>* dinv, int32_t* info,
             cudaStream_t s) {
    cudaMemsetAsync(info, 0, sizeof(int32_t), s);
    const size_t asmem = apply_smem_bytes(sizeof(CE<T>));
    const size_t ismem = inv_smem_bytes(sizeof(CE<T>));
    cudaFuncSetAttribute(tile_inv_kernel<T, C, T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ismem);
    cudaFuncSetAttribute(tile_apply_kernel<T, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)asmem);
    if (int rc = bem_lookahead_stream(ctx)) return rc;
    const int ni = (int)n;
    const int W = C ? 2 : 1;
    auto at = [&](int64_t r, int64_t c) { return A + W * (r * lda + c); };
    // A[r0:r0+rows, c0:c0+cols] -= A[r0:r0+rows, q0:q0+kk] A[q0:q0+kk, c0:c0+cols]
    auto update = [&](int64_t r0, int64_t c0, int64_t rows, int64_t cols, int64_t q0, int64_t kk) -> int {
        if (rows <= 0 || cols <= 0 || kk <= 0) return BEM_OK;
        return bem_gemm_update<T, C>(ctx, at(r0, c0), at(r0, q0), at(q0, c0), rows, cols, kk, lda, s);
    };
    // diagonal tile at k0 on the high-priority side stream, after the work queued on s so far
    auto diag_aside = [&](int64_t k0) {
        cudaEventRecord(ctx->ev_next, s);
        cudaStreamWaitEvent(ctx->aux, ctx->ev_next, 0);
        tile_diag_kernel<T, C><<<1, 256, 0, ctx->aux>>>(A, lda, ni, (int)k0, piv, info);
        cudaEventRecord(ctx->ev_diag, ctx->aux);
        ctx->launches++;
    };
    // row swaps of tile k0 outside it, then U12 = Linv A12 and L21 = A21 Uinv
    auto panel = [&](int64_t k0, int m) {
        tile_laswp_kernel<T, C><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A, lda, ni, (int)k0, m, piv);
        ctx->launches++;
        const int64_t rest = n - k0 - m;
        if (rest > 0) {
            const unsigned tiles = (unsigned)((rest + LU_T - 1) / LU_T);
            tile_apply_kernel<T, C><<<dim3(tiles, 2), 256, asmem, s>>>(A, lda, ni, (int)k0, m);
            ctx->launches++;
        }
    };
    // Tiles are taken in pairs (k, k+1) with a delayed update: step k updates
    // only tile k+1's column block (so its diagonal factorisation can start on
    // the side stream) and tile k+1's rows right of it; the trailing block then
    // receives steps k and k+1 together as one rank-128 update (K = 128 halves
    // the read-modify-write traffic of the trailing GEMMs).  The update's first
    // tile column goes first so that the next pair's diagonal tile overlaps the
    // rest of it.
    tile_diag_kernel<T, C><<<1, 256, 0, s>>>(A, lda, ni, 0, piv, info);
    ctx->launches++;
    bool on_aux = false;
    for (int64_t k0 = 0; k0 < n; k0 += 2 * LU_T) {
        const int m1 = (int)std::min<int64_t>(LU_T, n - k0);
        if (on_aux) cudaStreamWaitEvent(s, ctx->ev_diag, 0);
        panel(k0, m1);
        const int64_t k1 = k0 + m1, rest1 = n - k1;
        if (rest1 <= 0) break;
        const int m2 = (int)std::min<int64_t>(LU_T, rest1);
        if (int rc = update(k1, k1, rest1, m2, k0, m1)) return rc;
        diag_aside(k1);
        on_aux = true;
        const int64_t c2 = k1 + m2, rest2 = n - c2;
        if (int rc = update(k1, c2, m2, rest2, k0, m1)) return rc;
        cudaStreamWaitEvent(s, ctx->ev_diag, 0);
        panel(k1, m2);
        if (rest2 <= 0) break;
        const int64_t next = std::min<int64_t>(LU_T, rest2);
        if (int rc = update(c2, c2, rest2, next, k0, (int64_t)m1 + m2)) return rc;
        diag_aside(c2);
        if (int rc = update(c2, c2 + next, rest2, rest2 - next, k0, (int64_t)m1 + m2)) return rc;
        if (int rc = bem_check_cuda(ctx, cudaGetLastError(), "tiled lu step")) return rc;
    }
    // explicit inverses of every diagonal block (for the solves)
    tile_inv_kernel<T, C, T, false><<<(unsigned)((n + LU_T - 1) / LU_T), 256, ismem, s>>>(A, lda, ni, dinv);
    ctx->launches++;
    // No synchronisation: a tensor-core update whose bounded wait ran out
    // records it in flags[4], which the next solve on this context reads
    // (bem_take_factor_error) after its own synchronisation.
    return bem_check_cuda(ctx, cudaGetLastError(), "tiled lu");
}

// Scratch of a tiled solve in the context workspace: the row permutation and
// three vectors (permuted right-hand side, intermediate, solution).
struct SolveWs {
    int32_t* perm;
    double *b, *y, *x;
};

int solve_ws(bem_ctx* ctx, int64_t n, int W, SolveWs* w) {
    // no larger size has been run (a complex FP32 factor of 51200 rows is 21 GB)
    if (n > 51200) return bem_fail(ctx, BEM_ERR_INVALID, "tiled solve: n > 51200");
    const size_t off = ((size_t)n * 4 + 255) & ~size_t(255);
    const size_t vec = (sizeof(double) * W * (size_t)n + 255) & ~size_t(255);
    if (int rc = bem_ws_reserve(ctx, off + 3 * vec)) return rc;
    char* base = (char*)ctx->ws;
    w->perm = (int32_t*)base;
    w->b = (double*)(base + off);
    w->y = (double*)(base + off + vec);
    w->x = (double*)(base + off + 2 * vec);
    return BEM_OK;
}

// One solve queued on the stream: out receives the scratch vector that holds
// the solution; skipped on the device when skip != NULL and *skip != 0.
template <typename T, bool C>
int queue_solve(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const int32_t* piv, const CE<T>* dinv,
                const double* r, double** out, const int* skip, cudaStream_t s) {
    const int W = C ? 2 : 1;
    SolveWs w;
    if (int rc = solve_ws(ctx, n, W, &w)) return rc;
    const unsigned ptiles = (unsigned)((n + LU_T - 1) / LU_T);
    tile_piv_to_perm_kernel<<<(ptiles + 127) / 128, 128, 0, s>>>(piv, w.perm, (int)n);
    permute_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(r, w.perm, w.b, (int)n, W, skip);
    if (int rc = bem_check_cuda(ctx, queue_tri_solve<T, C, 1, false>(ctx->num_sms, LU, n, lda, dinv, w.b, w.y, w.x, 0,
                                                                     ctx->flags + 3, skip, s),
                                "tri_solve_kernel"))
        return rc;
    ctx->launches += 4;
    *out = w.x;
    return bem_check_cuda(ctx, cudaGetLastError(), "tiled solve");
}

template <typename T, bool C>
int solve_t(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const int32_t* piv, const CE<T>* dinv, double* b,
            cudaStream_t s) {
    const int W = C ? 2 : 1;
    int32_t* err = ctx->flags + 3;
    cudaMemsetAsync(err, 0, sizeof(int32_t), s);
    double* x = nullptr;
    if (int rc = queue_solve<T, C>(ctx, LU, n, lda, piv, dinv, b, &x, nullptr, s)) return rc;
    if (int rc = bem_check_cuda(ctx, cudaMemcpyAsync(b, x, sizeof(double) * W * n, cudaMemcpyDeviceToDevice, s),
                                "tiled solve copy"))
        return rc;
    int32_t e[2] = {0, 0};
    cudaMemcpyAsync(&e[0], err, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&e[1], ctx->flags + 4, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    if (int rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "tiled solve")) return rc;
    if (int rc = bem_take_factor_error(ctx, e[1], s)) return rc;
    if (e[0] != 0) return bem_fail(ctx, BEM_ERR_TIMEOUT, "tiled solve: a wait hit its iteration cap");
    return BEM_OK;
}

// One preconditioner application of the asynchronous refinement:
// out = (P^T L U)^{-1} r with the tile-pivoted factor, left in the solve
// workspace (*out), queued without synchronisation and skipped on the device
// when *skip != 0.  The caller resets ctx->flags[3] once before its loop and
// reads it after its final synchronisation.
template <typename T, bool C>
int precond_t(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const int32_t* piv, const CE<T>* dinv,
              const double* r, double** out, const int* skip, cudaStream_t s) {
    return queue_solve<T, C>(ctx, LU, n, lda, piv, dinv, r, out, skip, s);
}

// x = U^{-1} L^{-1} b for nrhs permuted right-hand sides (vs doubles apart), the
// FP64 diagonal inverses refined against the diagonal blocks; two at a time.
template <typename T, bool C>
int lu_tri_t(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const CE<double>* dinv, const double* b, double* y, double* x,
             int nrhs, int64_t vs, int32_t* err, cudaStream_t s) {
    for (int c = 0; c < nrhs;) {
        const int m = nrhs - c >= 2 ? 2 : 1;
        const cudaError_t e =
            m == 2 ? queue_tri_solve<T, C, 2, true>(ctx->num_sms, LU, n, lda, dinv, b + c * vs, y + c * vs, x + c * vs, vs,
                                                    err, nullptr, s)
                   : queue_tri_solve<T, C, 1, true>(ctx->num_sms, LU, n, lda, dinv, b + c * vs, y + c * vs, x + c * vs, vs,
                                                    err, nullptr, s);
        if (int rc = bem_check_cuda(ctx, e, "tri_solve_kernel")) return rc;
        ctx->launches += 2;
        c += m;
    }
    return bem_check_cuda(ctx, cudaGetLastError(), "lu_solve");
}

}  // namespace

extern "C" {

int bem_lu_factor_status(bem_ctx* ctx, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    int32_t e = 0;
    if (int rc = bem_check_cuda(ctx, cudaMemcpyAsync(&e, ctx->flags + 4, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                                "factor status"))
        return rc;
    if (int rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "factor status")) return rc;
    return bem_take_factor_error(ctx, e, s);
}

int64_t bem_lu_dinv_elems(int64_t n) { return ((n + LU_T - 1) / LU_T) * 2 * LU_T * LU_T; }

int bem_lu_factor_tiled(bem_ctx* ctx, int dtype, void* A, int64_t n, int64_t lda, int32_t* piv, void* dinv,
                        int32_t* info, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A || !piv || !dinv || !info || n <= 0 || lda < n || n > (1 << 30))
        return bem_fail(ctx, BEM_ERR_INVALID, "lu_factor_tiled: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64: return factor_t<double, false>(ctx, (double*)A, n, lda, piv, (CE<double>*)dinv, info, s);
        case BEM_C128: return factor_t<double, true>(ctx, (double*)A, n, lda, piv, (CE<double>*)dinv, info, s);
        case BEM_F32: return factor_t<float, false>(ctx, (float*)A, n, lda, piv, (CE<float>*)dinv, info, s);
        case BEM_C64: return factor_t<float, true>(ctx, (float*)A, n, lda, piv, (CE<float>*)dinv, info, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_factor_tiled: unknown dtype");
    }
}

int bem_lu_solve_tiled(bem_ctx* ctx, int dtype, const void* LU, int64_t n, int64_t lda, const int32_t* piv,
                       const void* dinv, void* b, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!LU || !piv || !dinv || !b || n <= 0 || lda < n)
        return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve_tiled: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64: return solve_t<double, false>(ctx, (const double*)LU, n, lda, piv, (const CE<double>*)dinv, (double*)b, s);
        case BEM_C128: return solve_t<double, true>(ctx, (const double*)LU, n, lda, piv, (const CE<double>*)dinv, (double*)b, s);
        case BEM_F32: return solve_t<float, false>(ctx, (const float*)LU, n, lda, piv, (const CE<float>*)dinv, (double*)b, s);
        case BEM_C64: return solve_t<float, true>(ctx, (const float*)LU, n, lda, piv, (const CE<float>*)dinv, (double*)b, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve_tiled: unknown dtype");
    }
}

}  // extern "C"

template <typename T, bool C, typename D, bool EXACT>
int tile_inverses_t(bem_ctx* ctx, const T* A, int64_t n, int64_t lda, CE<D>* dinv, cudaStream_t s) {
    const size_t ismem = inv_smem_bytes(sizeof(CE<D>));
    cudaFuncSetAttribute(tile_inv_kernel<T, C, D, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ismem);
    tile_inv_kernel<T, C, D, EXACT><<<(unsigned)((n + LU_T - 1) / LU_T), 256, ismem, s>>>(A, lda, (int)n, dinv);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "tile_inv_kernel");
}

int bem_tile_inverses(bem_ctx* ctx, bool cplx, const double* A, int64_t n, int64_t lda, void* dinv, cudaStream_t s) {
    CE<double>* d = (CE<double>*)dinv;
    return cplx ? tile_inverses_t<double, true, double, false>(ctx, A, n, lda, d, s)
                : tile_inverses_t<double, false, double, false>(ctx, A, n, lda, d, s);
}

int bem_solve_inverses(bem_ctx* ctx, int dtype, const void* A, int64_t n, int64_t lda, void* dinv, cudaStream_t s) {
    CE<double>* d = (CE<double>*)dinv;
    switch (dtype) {
        case BEM_F64: return tile_inverses_t<double, false, double, true>(ctx, (const double*)A, n, lda, d, s);
        case BEM_C128: return tile_inverses_t<double, true, double, true>(ctx, (const double*)A, n, lda, d, s);
        case BEM_F32: return tile_inverses_t<float, false, double, true>(ctx, (const float*)A, n, lda, d, s);
        case BEM_C64: return tile_inverses_t<float, true, double, true>(ctx, (const float*)A, n, lda, d, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: unknown dtype");
    }
}

template <typename T, bool C>
int small_solve_t(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const double* b, double* x, int nrhs, int64_t vs,
                  cudaStream_t s) {
    const size_t smem = sizeof(CE<double>) * (size_t)n + sizeof(CE<T>) * LU_T * SMALL_LD;
    if (int rc = bem_check_cuda(ctx, cudaFuncSetAttribute(small_solve_kernel<T, C>,
                                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                "small_solve_kernel smem"))
        return rc;
    small_solve_kernel<T, C><<<(unsigned)nrhs, 256, smem, s>>>(LU, lda, (int)n, b, x, vs);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "small_solve_kernel");
}

int bem_lu_small_solve(bem_ctx* ctx, int dtype, const void* LU, int64_t n, int64_t lda, const double* b, double* x,
                       int nrhs, int64_t vs, cudaStream_t s) {
    switch (dtype) {
        case BEM_F64: return small_solve_t<double, false>(ctx, (const double*)LU, n, lda, b, x, nrhs, vs, s);
        case BEM_C128: return small_solve_t<double, true>(ctx, (const double*)LU, n, lda, b, x, nrhs, vs, s);
        case BEM_F32: return small_solve_t<float, false>(ctx, (const float*)LU, n, lda, b, x, nrhs, vs, s);
        case BEM_C64: return small_solve_t<float, true>(ctx, (const float*)LU, n, lda, b, x, nrhs, vs, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: unknown dtype");
    }
}

int bem_lu_tri_solve(bem_ctx* ctx, int dtype, const void* LU, int64_t n, int64_t lda, const void* dinv, const double* b,
                     double* y, double* x, int nrhs, int64_t vs, int32_t* err, cudaStream_t s) {
    switch (dtype) {
        case BEM_F64: return lu_tri_t<double, false>(ctx, (const double*)LU, n, lda, (const CE<double>*)dinv, b, y, x, nrhs, vs, err, s);
        case BEM_C128: return lu_tri_t<double, true>(ctx, (const double*)LU, n, lda, (const CE<double>*)dinv, b, y, x, nrhs, vs, err, s);
        case BEM_F32: return lu_tri_t<float, false>(ctx, (const float*)LU, n, lda, (const CE<double>*)dinv, b, y, x, nrhs, vs, err, s);
        case BEM_C64: return lu_tri_t<float, true>(ctx, (const float*)LU, n, lda, (const CE<double>*)dinv, b, y, x, nrhs, vs, err, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: unknown dtype");
    }
}

int bem_tiled_precond_async(bem_ctx* ctx, int dtype, const void* LU, int64_t n, int64_t lda, const int32_t* piv,
                            const void* dinv, const double* r, double** out, const int* skip, cudaStream_t s) {
    switch (dtype) {
        case BEM_F64: return precond_t<double, false>(ctx, (const double*)LU, n, lda, piv, (const CE<double>*)dinv, r, out, skip, s);
        case BEM_C128: return precond_t<double, true>(ctx, (const double*)LU, n, lda, piv, (const CE<double>*)dinv, r, out, skip, s);
        case BEM_F32: return precond_t<float, false>(ctx, (const float*)LU, n, lda, piv, (const CE<float>*)dinv, r, out, skip, s);
        case BEM_C64: return precond_t<float, true>(ctx, (const float*)LU, n, lda, piv, (const CE<float>*)dinv, r, out, skip, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "tiled precond: unknown dtype");
    }
}

// ----------------------------------------------------------------------------
// Allocation-free variant of bem_lu_solve_tiled.
//
// Its scratch (row permutation, error word, three work vectors) lives in
// one file-scope __device__ array instead of a context workspace, so the call
// needs no bem_ctx and performs no device allocation.  The array is sized for
// n <= BEM_STATIC_SOLVE_MAX_N and is held by every GPU that loads this library
// until the process exits.  Host code only ever sees the array's host-side
// stand-in name; its device address comes from cudaGetSymbolAddress, taken
// once per device (with that device current) on the first call there.
// ----------------------------------------------------------------------------
#include <mutex>

namespace {

constexpr int64_t kStaticSolveMaxN = BEM_STATIC_SOLVE_MAX_N;

struct StaticSolveScratch {
    int32_t perm[kStaticSolveMaxN];
    int32_t err[4];
    double b[2 * kStaticSolveMaxN];
    double y[2 * kStaticSolveMaxN];
    double x[2 * kStaticSolveMaxN];
};

__device__ __align__(256) StaticSolveScratch g_static_solve_scratch;

constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
StaticSolveScratch* g_static_addr[kMaxDevices] = {};

// Device address of the scratch array on the current device (set-up on the
// first call per device).
int static_scratch(StaticSolveScratch** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) return BEM_ERR_INVALID;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_solve_scratch);
        if (e != cudaSuccess || p == nullptr) {
            cudaGetLastError();
            return BEM_ERR_CUDA;
        }
        g_static_addr[dev] = static_cast<StaticSolveScratch*>(p);
    }
    *out = g_static_addr[dev];
    return BEM_OK;
}

template <typename T, bool C>
int solve_static_t(const T* LU, int64_t n, int64_t lda, const int32_t* piv, const CE<T>* dinv, double* b,
                   cudaStream_t s) {
    StaticSolveScratch* sc = nullptr;
    if (int rc = static_scratch(&sc)) return rc;
    const int W = C ? 2 : 1;
    const int nbk = (int)((n + LU_T - 1) / LU_T);
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int32_t* err = sc->err;
    tile_piv_to_perm_kernel<<<(unsigned)((nbk + 127) / 128), 128, 0, s>>>(piv, sc->perm, (int)n);
    permute_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, sc->perm, sc->b, (int)n, W, nullptr);
    if (cudaGetLastError() != cudaSuccess) return BEM_ERR_CUDA;
    // the array keeps the previous call's contents: the error word must start at zero
    if (cudaMemsetAsync(err, 0, sizeof(int32_t), s) != cudaSuccess ||
        queue_tri_solve<T, C, 1, false>(sms, LU, n, lda, dinv, sc->b, sc->y, sc->x, 0, err, nullptr, s) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    if (cudaMemcpyAsync(b, sc->x, sizeof(double) * W * n, cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    int32_t e = 0;
    if (cudaMemcpyAsync(&e, err, sizeof(int32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    return e != 0 ? BEM_ERR_TIMEOUT : BEM_OK;
}

}  // namespace

extern "C" int bem_lu_solve_tiled_static(int dtype, const void* LU, int64_t n, int64_t lda, const int32_t* piv,
                                         const void* dinv, void* b, void* stream) {
    if (!LU || !piv || !dinv || !b || n <= 0 || lda < n) return BEM_ERR_INVALID;
    if (n > kStaticSolveMaxN) return BEM_ERR_INVALID;  // beyond the static scratch
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64: return solve_static_t<double, false>((const double*)LU, n, lda, piv, (const CE<double>*)dinv, (double*)b, s);
        case BEM_C128: return solve_static_t<double, true>((const double*)LU, n, lda, piv, (const CE<double>*)dinv, (double*)b, s);
        case BEM_F32: return solve_static_t<float, false>((const float*)LU, n, lda, piv, (const CE<float>*)dinv, (double*)b, s);
        case BEM_C64: return solve_static_t<float, true>((const float*)LU, n, lda, piv, (const CE<float>*)dinv, (double*)b, s);
        default: return BEM_ERR_INVALID;
    }
}
