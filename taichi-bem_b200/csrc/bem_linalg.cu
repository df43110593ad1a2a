// Dense LU with partial pivoting, triangular solves, GEMV and mixed-precision
// iterative refinement (replaces torch.linalg.solve at
// src/managers/BEM_manager.py:1056; no cuSOLVER).
//
// Factorisation (right-looking, block width LU_NB):
//   panel   : one thread-block cluster holding the panel in shared memory
//             (lu_panel_cluster_kernel); panels with too many rows for that by
//             one cooperative launch, each CTA owning a slice of the rows: per
//             column one grid barrier publishes every CTA's pivot candidate,
//             after which all CTAs agree on the pivot, swap it in and apply
//             the rank-1 update to their rows (lu_panel_kernel).
//   next    : FP64: the three steps below for the next panel's columns in one
//             launch (lu_next_kernel), so that the next panel starts beside
//             them for all other columns (look-ahead).
//   laswp   : the panel's row swaps applied to the columns outside the panel.
//   trsm    : U12 = L11^-1 A12, L11 staged in shared memory.
//   update  : A22 -= L21 U12 (bem_gemm.cuh: FP64 tensor cores for the plain
//             path, tcgen05 TF32 tensor-core tiles for the FP32 factor).
// Every device-side wait (grid barriers, mbarriers) is bounded; a timeout sets a flag and
// the host call returns BEM_ERR_TIMEOUT.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <complex>
#include <functional>
#include <type_traits>
#include <vector>

#include <cmath>
#include <vector>

#include "bem_gemm.cuh"
#include "bem_internal.cuh"

namespace {

constexpr int LU_NB = 64;
constexpr unsigned SPIN_CAP = 1u << 22;  // x ~256 ns sleep ~ 1 s

struct GridBar {
    unsigned count;
    unsigned gen;
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acq_rel(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Bounded software grid barrier (the launch is cooperative, so all CTAs are
// co-resident).  The last CTA to arrive resets the counter and releases the
// generation word; the others poll it with acquire loads, first without and
// then with a short sleep.  Returns false when the wait hit its cap (flag set)
// or another CTA reported a failure.
__device__ __forceinline__ bool grid_barrier(GridBar* bar, unsigned nblocks, int32_t* flag) {
    __syncthreads();
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned g = ld_acquire(&bar->gen);
        __threadfence();
        const unsigned arrived = atom_add_acq_rel(&bar->count, 1u);
        if (arrived == nblocks - 1) {
            bar->count = 0u;
            st_release(&bar->gen, g + 1u);
        } else {
            unsigned it = 0;
            while (ld_acquire(&bar->gen) == g) {
                if (++it > SPIN_CAP) {
                    atomicExch(flag, BEM_ERR_TIMEOUT);
                    ok = 0;
                    break;
                }
                if ((it & 63u) == 0u && *(volatile int32_t*)flag != 0) {
                    ok = 0;
                    break;
                }
                if (it > 4096u) __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

template <typename T, bool C>
struct alignas(2 * sizeof(T)) El {
    T re, im;
};

template <typename T, bool C>
__device__ __forceinline__ El<T, C> ld(const T* A, int64_t i) {
    El<T, C> e;
    if (C) {
        e.re = A[2 * i];
        e.im = A[2 * i + 1];
    } else {
        e.re = A[i];
        e.im = T(0);
    }
    return e;
}
template <typename T, bool C>
__device__ __forceinline__ void st(T* A, int64_t i, El<T, C> e) {
    if (C) {
        A[2 * i] = e.re;
        A[2 * i + 1] = e.im;
    } else {
        A[i] = e.re;
    }
}
template <typename T, bool C>
__device__ __forceinline__ T mag1(El<T, C> e) {
    return C ? fabs(e.re) + fabs(e.im) : fabs(e.re);
}
template <typename T, bool C>
__device__ __forceinline__ El<T, C> ld_volatile(const El<T, C>* p) {
    const volatile T* v = reinterpret_cast<const volatile T*>(p);
    El<T, C> e;
    e.re = v[0];
    e.im = C ? v[1] : T(0);
    return e;
}

struct PivSlot {
    double val;
    int idx;
    int pad;
};

// 1/a of a pivot candidate; not finite for zero
template <typename T, bool C>
__device__ __forceinline__ El<T, C> pivot_inverse(El<T, C> a) {
    if (!C) return El<T, C>{T(1) / a.re, T(0)};
    const T s = bem_unit_scale(a.re, a.im);
    a = El<T, C>{a.re * s, a.im * s};
    const T rd = T(1) / (a.re * a.re + a.im * a.im);
    return El<T, C>{a.re * rd * s, -a.im * rd * s};
}

// ----------------------------------------------------------------------------
// panel factorisation (cooperative)
//
// Each CTA owns a contiguous slice of the panel's rows, held in shared memory
// for the whole panel (SMEM_ROWS) or read from global memory when the slice
// does not fit.  Per column j: every CTA publishes its best pivot candidate
// (value, row) and a copy of that row, and the owner of row jj publishes row
// jj, into buffers indexed by the parity of j; one grid barrier; every CTA
// reads the winner's row and row jj from those buffers (never from another
// CTA's slice), swaps, and updates its own rows.  Double buffering by parity
// keeps a CTA that is one column ahead from overwriting buffers still read.
// ----------------------------------------------------------------------------
constexpr int PANEL_MAXB = 256;

template <typename T, bool C, bool SMEM_ROWS>
__global__ void __launch_bounds__(256) lu_panel_kernel(T* A, int64_t lda, int n, int k0, int nb, int chunk,
                                                       int32_t* piv, int32_t* info, GridBar* bar, PivSlot* slots,
                                                       El<T, C>* rowbuf, int32_t* flag) {
    using E = El<T, C>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    E* srows = reinterpret_cast<E*>(smem_raw);  // [chunk][nb] when SMEM_ROWS
    const unsigned nblk = gridDim.x;
    const int r_begin = k0 + blockIdx.x * chunk;
    const int r_end = min(n, r_begin + chunk);
    __shared__ E s_prow[LU_NB];
    __shared__ E s_jrow[LU_NB];
    __shared__ double s_red_v[8];
    __shared__ int s_red_i[8];
    __shared__ int s_red_b[8];
    __shared__ int s_best_idx;
    __shared__ int s_p, s_pb;
    __shared__ double s_pv;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;

    auto row_ptr_g = [&](int r) { return A + (C ? 2 : 1) * ((int64_t)r * lda + k0); };
    auto get = [&](int r, int c) -> E {
        if (SMEM_ROWS) return srows[(r - r_begin) * nb + c];
        return ld<T, C>(row_ptr_g(r), c);
    };
    auto put = [&](int r, int c, E v) {
        if (SMEM_ROWS)
            srows[(r - r_begin) * nb + c] = v;
        else
            st<T, C>(row_ptr_g(r), c, v);
    };
    if (SMEM_ROWS) {
        for (int e = threadIdx.x; e < (r_end - r_begin) * nb; e += blockDim.x) {
            int r = e / nb, c = e - r * nb;
            srows[e] = ld<T, C>(row_ptr_g(r_begin + r), c);
        }
        __syncthreads();
    }

    for (int j = 0; j < nb; ++j) {
        const int jj = k0 + j;
        const int par = j & 1;
        PivSlot* slot = slots + par * PANEL_MAXB;
        E* rb = rowbuf + (size_t)par * (PANEL_MAXB + 1) * LU_NB;
        // 1. local pivot candidate
        double best = -1.0;
        int bidx = 0x7fffffff;
        for (int r = max(r_begin, jj) + threadIdx.x; r < r_end; r += blockDim.x) {
            double v = (double)mag1<T, C>(get(r, j));
            if (v > best || (v == best && r < bidx)) {
                best = v;
                bidx = r;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            double ov = __shfl_xor_sync(0xffffffffu, best, o);
            int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
            if (ov > best || (ov == best && oi < bidx)) {
                best = ov;
                bidx = oi;
            }
        }
        if (lane == 0) {
            s_red_v[wid] = best;
            s_red_i[wid] = bidx;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < nwarps; ++w)
                if (s_red_v[w] > best || (s_red_v[w] == best && s_red_i[w] < bidx)) {
                    best = s_red_v[w];
                    bidx = s_red_i[w];
                }
            slot[blockIdx.x].val = best;
            slot[blockIdx.x].idx = bidx;
            s_best_idx = bidx;
        }
        __syncthreads();
        const int cand = s_best_idx;
        if (cand >= r_begin && cand < r_end)
            for (int c = threadIdx.x; c < nb; c += blockDim.x) rb[(size_t)blockIdx.x * LU_NB + c] = get(cand, c);
        if (jj >= r_begin && jj < r_end)
            for (int c = threadIdx.x; c < nb; c += blockDim.x) rb[(size_t)PANEL_MAXB * LU_NB + c] = get(jj, c);
        // 2. publish
        if (!grid_barrier(bar, nblk, flag)) return;
        // 3. global pivot, slots read in parallel
        {
            double bv = -1.0;
            int bi = 0x7fffffff, bb = -1;
            for (unsigned b = threadIdx.x; b < nblk; b += blockDim.x) {
                double v = ((volatile PivSlot*)slot)[b].val;
                int i = ((volatile PivSlot*)slot)[b].idx;
                if (v > bv || (v == bv && i < bi)) {
                    bv = v;
                    bi = i;
                    bb = (int)b;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                double ov = __shfl_xor_sync(0xffffffffu, bv, o);
                int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                int ob = __shfl_xor_sync(0xffffffffu, bb, o);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                    bb = ob;
                }
            }
            if (lane == 0) {
                s_red_v[wid] = bv;
                s_red_i[wid] = bi;
                s_red_b[wid] = bb;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int w = 1; w < nwarps; ++w)
                    if (s_red_v[w] > bv || (s_red_v[w] == bv && s_red_i[w] < bi)) {
                        bv = s_red_v[w];
                        bi = s_red_i[w];
                        bb = s_red_b[w];
                    }
                if (bb < 0 || bi < jj || bi >= n) {  // no candidate: keep the diagonal
                    bi = jj;
                    bb = -1;
                    bv = 0.0;
                }
                s_p = bi;
                s_pb = bb;
                s_pv = bv;
                if (blockIdx.x == 0) {
                    piv[jj] = bi;
                    if (!(bv > 0.0) && *info == 0) *info = jj + 1;
                }
            }
            __syncthreads();
        }
        const int p = s_p;
        for (int c = threadIdx.x; c < nb; c += blockDim.x) {
            E ej = ld_volatile<T, C>(rb + (size_t)PANEL_MAXB * LU_NB + c);
            s_jrow[c] = ej;
            s_prow[c] = s_pb >= 0 ? ld_volatile<T, C>(rb + (size_t)s_pb * LU_NB + c) : ej;
        }
        __syncthreads();
        // 4. swap rows jj and p (panel columns)
        if (p != jj) {
            if (jj >= r_begin && jj < r_end)
                for (int c = threadIdx.x; c < nb; c += blockDim.x) put(jj, c, s_prow[c]);
            if (p >= r_begin && p < r_end)
                for (int c = threadIdx.x; c < nb; c += blockDim.x) put(p, c, s_jrow[c]);
        }
        __syncthreads();
        // 5. scale column jj below the diagonal, rank-1 update of the panel
        const E pv = s_prow[j];
        const bool nonzero = s_pv > 0.0;
        const E inv = nonzero ? pivot_inverse<T, C>(pv) : E{T(0), T(0)};
        for (int r = max(r_begin, jj + 1) + wid; r < r_end; r += nwarps) {
            E a = get(r, j);
            E l;
            l.re = a.re * inv.re - (C ? a.im * inv.im : T(0));
            l.im = C ? a.re * inv.im + a.im * inv.re : T(0);
            for (int c = j + 1 + lane; c < nb; c += 32) {
                E v = get(r, c);
                E u = s_prow[c];
                v.re -= l.re * u.re - (C ? l.im * u.im : T(0));
                if (C) v.im -= l.re * u.im + l.im * u.re;
                put(r, c, v);
            }
            __syncwarp();
            if (lane == 0) put(r, j, l);
        }
        __syncthreads();
    }
    if (SMEM_ROWS) {
        for (int e = threadIdx.x; e < (r_end - r_begin) * nb; e += blockDim.x) {
            int r = e / nb, c = e - r * nb;
            st<T, C>(row_ptr_g(r_begin + r), c, srows[e]);
        }
    }
}

// ----------------------------------------------------------------------------
// panel factorisation on one thread-block cluster
//
// The panel is a chain of nb column steps (pivot, exchange, update) whose
// arithmetic is small, so its time is the latency of a step.  When the panel
// fits the shared memory of one cluster (up to 16 CTAs), the step needs no
// grid-wide barrier through L2: every thread owns one row, sub-blocks of
// PCL_SB columns of it in registers, and per column
//   * each CTA reduces its pivot candidate (largest |re| + |im|, lowest
//     position) and pushes value, position and the candidate's PCL_SB
//     elements into every CTA's mailbox (distributed shared memory, st.async
//     counted by the mailbox's mbarrier: a CTA goes on when all candidates
//     have arrived, without the round trip of a cluster barrier);
//   * every CTA takes the best of the mailboxes and updates its rows'
//     registers; the pivot row's CTA pushes the row's remaining elements.
// A mailbox or U row is written again only by a CTA that has received a later
// candidate of this one, which was sent after this one read the old contents.
// Rows never move: a row carries its position, the row at the diagonal
// position takes the pivot's, and the panel is written out by position (the
// swap sequence in piv is that of moved rows).  After a sub-block the pivot
// rows' remaining elements are solved against the sub-block's unit lower
// triangle and applied as one rank-PCL_SB update, so shared memory is swept once per PCL_SB columns (FP64: on the FP64 tensor
// cores).  Measured (B200, a column step averaged over a whole factorisation):
// 2999 complex rows 1.44 us (6.0 us of the cooperative kernel below, a grid
// barrier a column; 1.95 with a cluster barrier a column and the panel read
// through registers), 1280 real rows 1.19 us (5.8; 1.73).  What a step consists
// of are some twelve dependent shared-memory and warp-reduction latencies of
// 30 to 200 cycles; a loop over the columns instead of eight copies of the step
// (registers turned instead of indexed) and half the warps were both slower.
// ----------------------------------------------------------------------------
constexpr int PCL_SB = 8;
constexpr int PCL_MAXC = 16;
constexpr int PCL_MAXROWS = PCL_MAXC * 512;
constexpr uint32_t PCL_SPIN_CAP = 1u << 20;

// A pivot candidate as integers that order like the rule "largest value,
// then lowest position": hi is the value's high word plus one (0: not a
// candidate, or the diagonal row holding a NaN, whose lo is 1), lo its low word.
struct alignas(16) PivKey {
    unsigned hi, lo;
    int pos;
    int row;  // the candidate's row in its CTA
};

// the lane with the best of a warp's keys: usually one lane has the largest
// high word, and one warp reduction settles it
__device__ __forceinline__ int best_lane(const PivKey& k) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, k.hi);
    unsigned who = __ballot_sync(0xffffffffu, k.hi == hi);
    if (who & (who - 1)) {
        const unsigned lo = __reduce_max_sync(0xffffffffu, k.hi == hi ? k.lo : 0u);
        const bool mine = k.hi == hi && k.lo == lo;
        const int pos = __reduce_min_sync(0xffffffffu, mine ? k.pos : 0x7fffffff);
        who = __ballot_sync(0xffffffffu, mine && k.pos == pos);
    }
    return __ffs((int)who) - 1;
}

template <typename T, bool C>
struct PanelShared {
    // mailboxes, per column of the sub-block and sending CTA: the candidate's reciprocal and its elements in the
    // other columns of the sub-block
    El<T, C> rec[PCL_SB][PCL_MAXC][PCL_SB];
    El<T, C> warp[2][16][PCL_SB];            // candidate rows of this CTA's warps, by parity of the column
    El<T, C> U[PCL_SB][LU_NB];               // the sub-block's pivot rows right of it
    PivKey key[2][PCL_MAXC];
    PivKey wkey[2][16];
    unsigned long long rec_bar[PCL_SB], u_bar;  // mbarriers of the mailboxes and of U
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// offset from a shared address of this CTA to the same one of another CTA of the cluster
__device__ __forceinline__ uint32_t peer_offset(const void* p, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
    return r - smem_addr(p);
}
// 8 or 16 bytes into a CTA of the cluster, counted by its mbarrier `bar`
template <typename V>
__device__ __forceinline__ void push(uint32_t dst, const V& v, uint32_t bar) {
    static_assert(sizeof(V) == 8 || sizeof(V) == 16, "8 or 16 bytes");
    if constexpr (sizeof(V) == 16) {
        const int4 w = *reinterpret_cast<const int4*>(&v);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                     "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w), "r"(bar)
                     : "memory");
    } else {
        const long long w = *reinterpret_cast<const long long*>(&v);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(w), "r"(bar)
                     : "memory");
    }
}
__device__ __forceinline__ void bar_expect(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// waits for the mbarrier's phase; false at the iteration limit
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, uint32_t parity) {
    const uint32_t addr = smem_addr(bar);
    for (uint32_t it = 0; it < PCL_SPIN_CAP; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// one element of the panel in shared memory (complex: one 2 sizeof(T) access)
template <typename T, bool C>
__device__ __forceinline__ El<T, C> ld_p(const T* P, int i) {
    if (C) return *reinterpret_cast<const El<T, C>*>(P + 2 * i);
    return El<T, C>{P[i], T(0)};
}
template <typename T, bool C>
__device__ __forceinline__ void st_p(T* P, int i, El<T, C> e) {
    if (C)
        *reinterpret_cast<El<T, C>*>(P + 2 * i) = e;
    else
        P[i] = e.re;
}

// P[r][c0 + c] -= sum_q L[r][q] U[q][c] for the rows not yet pivots: L = the
// sub-block's PCL_SB columns of P (from column jb), nt columns from c0.  FP64
// on the FP64 tensor cores (m8n8k4, fragments as in bem_gemm.cuh), a warp per
// 8 x 8 tile; FP32 a thread per row.
template <typename T, bool C, int THREADS>
__device__ __forceinline__ void panel_rank8(T* P, int ldc, int cnt, int jb, int c0, int nt,
                                            const El<T, C> (*U)[LU_NB], const unsigned char* s_done,
                                            const El<T, C>* a, bool active) {
    using E = El<T, C>;
    const int tid = threadIdx.x;
    if constexpr (sizeof(T) == 8) {
        constexpr int NP = C ? 2 : 1;
        const int lane = tid & 31, wid = tid >> 5;
        const int row8 = lane >> 2, k4 = lane & 3;
        const int ct = (nt + 7) / 8;
        for (int rt = wid; rt * 8 < cnt; rt += THREADS / 32) {
            const int r = rt * 8 + row8;
            const bool rok = r < cnt;
            const bool store = rok && !s_done[r];
            E fa[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                fa[h] = store ? ld_p<T, C>(P, (jb + 4 * h + k4) * ldc + r) : E{T(0), T(0)};
#pragma unroll 4
            for (int t = 0; t < ct; ++t) {
                const int cc = t * 8 + 2 * k4;
                double acc[2][NP];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const E v = rok && cc + e < nt ? ld_p<T, C>(P, (c0 + cc + e) * ldc + r) : E{T(0), T(0)};
                    acc[e][0] = v.re;
                    if (C) acc[e][NP - 1] = v.im;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const E u = U[4 * h + k4][min(t * 8 + row8, LU_NB - 1)];
                    bem_gemm_detail::dmma_acc(acc[0][0], acc[1][0], -fa[h].re, u.re);
                    if (C) {
                        bem_gemm_detail::dmma_acc(acc[0][0], acc[1][0], fa[h].im, u.im);
                        bem_gemm_detail::dmma_acc(acc[0][NP - 1], acc[1][NP - 1], -fa[h].re, u.im);
                        bem_gemm_detail::dmma_acc(acc[0][NP - 1], acc[1][NP - 1], -fa[h].im, u.re);
                    }
                }
                if (store)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (cc + e < nt) st_p<T, C>(P, (c0 + cc + e) * ldc + r, E{(T)acc[e][0], C ? (T)acc[e][NP - 1] : T(0)});
            }
        }
    } else if (active) {
        for (int c = 0; c < nt; ++c) {
            E v = ld_p<T, C>(P, (c0 + c) * ldc + tid);
#pragma unroll
            for (int q = 0; q < PCL_SB; ++q) {
                const E u = U[q][c];
                v.re -= a[q].re * u.re - (C ? a[q].im * u.im : T(0));
                if (C) v.im -= a[q].re * u.im + a[q].im * u.re;
            }
            st_p<T, C>(P, (c0 + c) * ldc + tid, v);
        }
    }
}

template <typename T, bool C, int THREADS>
__global__ void __launch_bounds__(THREADS) lu_panel_cluster_kernel(T* A, int64_t lda, int n, int k0, int nb, int chunk,
                                                                   int ldc, int32_t* piv, int32_t* info, int32_t* flag,
                                                                   int32_t* src) {
    using E = El<T, C>;
    constexpr int W = C ? 2 : 1;
    constexpr int NW = THREADS / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PanelShared<T, C>& sh = *reinterpret_cast<PanelShared<T, C>*>(smem_raw);
    T* P = reinterpret_cast<T*>(smem_raw + ((sizeof(PanelShared<T, C>) + 15) & ~size_t(15)));  // [nb][ldc], by columns
    int* s_pos = reinterpret_cast<int*>(P + (size_t)W * LU_NB * ldc);                          // [chunk]
    unsigned char* s_done = reinterpret_cast<unsigned char*>(s_pos + chunk);                   // [chunk]
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank(), nc = (int)cluster.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int r0 = k0 + rank * chunk;
    const int cnt = max(0, min(chunk, n - r0));
    // a warp a row, without registers in between: all of the panel in flight.
    // Complex elements in one copy each where A allows it (16 or 8 bytes).
    const bool whole = reinterpret_cast<uintptr_t>(A) % (W * sizeof(T)) == 0;
    for (int r = wid; r < cnt; r += NW)
        for (int c = lane; c < nb; c += 32) {
            const uint32_t dst = smem_addr(P + (size_t)W * (c * ldc + r));
            const T* src = A + W * ((int64_t)(r0 + r) * lda + k0 + c);
            if (whole) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"((int)(W * sizeof(T))));
            } else {
                for (int h = 0; h < W; ++h)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + (uint32_t)(h * sizeof(T))),
                                 "l"(src + h), "n"((int)sizeof(T)));
            }
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const bool mine = tid < cnt;
    int pos = r0 + tid;
    bool done = !mine;
    int bad = 0;  // 1 + first column without a nonzero pivot
    // thread (destination, element) of the pushes
    const int dest = tid >> 4, elem = tid & 15;
    const uint32_t peer = peer_offset(smem_raw, min(dest, nc - 1));
    bool lost = false;  // a wait ran out: the rest runs without waiting, and flag reports it
    if (mine) s_done[tid] = 0;
    if (tid < 2 * PCL_MAXC) sh.key[tid / PCL_MAXC][tid % PCL_MAXC] = PivKey{0u, 0u, 0x7fffffff, 0};
    if (tid == 0) {
        for (int q = 0; q < PCL_SB; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.rec_bar[q])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.u_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    cluster.sync();

    for (int jb = 0; jb < nb; jb += PCL_SB) {
        const int sw = min(PCL_SB, nb - jb);
        const int nt = nb - jb - sw;  // columns of the panel right of the sub-block (0 unless sw == PCL_SB)
        const uint32_t parity = (uint32_t)(jb / PCL_SB) & 1u;
        if (tid == 0) {
            for (int q = 0; q < sw; ++q) bar_expect(&sh.rec_bar[q], nc * (uint32_t)(PCL_SB * sizeof(E) + sizeof(PivKey)));
            if (nt > 0) bar_expect(&sh.u_bar, (uint32_t)(PCL_SB * nt * sizeof(E)));
        }
        E a[PCL_SB];
        int myq = -1;
#pragma unroll
        for (int c = 0; c < PCL_SB; ++c) a[c] = mine && c < sw ? ld_p<T, C>(P, (jb + c) * ldc + tid) : E{T(0), T(0)};
        uint32_t senders = 0;  // 4 bits a column: the CTA its pivot came from
        int own = -1;          // this CTA's row that became the last pivot
        // the rest of pivot row q, to every CTA
        auto push_row = [&](int q) {
            if (own < 0 || nt <= 0 || dest >= nc) return;
#pragma unroll 1
            for (int c = elem; c < nt; c += 16)
                push(smem_addr(&sh.U[q][c]) + peer, ld_p<T, C>(P, (jb + PCL_SB + c) * ldc + own),
                     smem_addr(&sh.u_bar) + peer);
        };
#pragma unroll
        for (int jj = 0; jj < PCL_SB; ++jj) {
            if (jj < sw) {  // uniform over the cluster
                const int jd = k0 + jb + jj;
                // candidate of this row; NaN never wins, but the diagonal row stays as the last resort
                PivKey key{0u, 0u, 0x7fffffff, tid};
                if (!done) {
                    const double v = (double)mag1<T, C>(a[jj]);
                    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
                    if (hi < 0x7ff00000u || (hi == 0x7ff00000u && lo == 0u)) {  // |.| >= 0: not NaN
                        key.hi = hi + 1u;
                        key.lo = lo;
                        key.pos = pos;
                    } else if (pos == jd) {
                        key.lo = 1u;
                        key.pos = pos;
                    }
                }
                // every row's reciprocal beside the reductions, so that the pivot's is at hand
                const E rc = pivot_inverse<T, C>(a[jj]);
                if (lane == best_lane(key)) {
#pragma unroll
                    for (int c = 0; c < PCL_SB; ++c) sh.warp[jj & 1][wid][c] = c == jj ? rc : a[c];
                    sh.wkey[jj & 1][wid] = key;
                }
                __syncthreads();
                {
                    PivKey k{0u, 0u, 0x7fffffff, 0};
                    if (lane < NW) k = sh.wkey[jj & 1][lane];
                    const int bw = min(best_lane(k), NW - 1);
                    // thread (destination, element) pushes one element of the candidate
                    if (dest < nc) {
                        const uint32_t bar = smem_addr(&sh.rec_bar[jj]) + peer;
                        if (elem < PCL_SB)
                            push(smem_addr(&sh.rec[jj][rank][elem]) + peer, sh.warp[jj & 1][bw][elem], bar);
                        else if (elem == PCL_SB)
                            push(smem_addr(&sh.key[jj & 1][rank]) + peer, sh.wkey[jj & 1][bw], bar);
                    }
                }
                if (jj > 0) push_row(jj - 1);
                if (!lost) lost = !bar_wait(&sh.rec_bar[jj], parity);
                PivKey k{0u, 0u, 0x7fffffff, 0};
                if (lane < nc) k = sh.key[jj & 1][lane];
                const int from = min(best_lane(k), nc - 1);
                const E* prow = sh.rec[jj][from];
                const PivKey gb = sh.key[jj & 1][from];
                const int bp = gb.pos >= jd && gb.pos < n ? gb.pos : jd;
                const bool nonzero = gb.hi > 0u && ((gb.hi - 1u) | gb.lo) != 0u;
                const E inv = nonzero ? prow[jj] : E{T(0), T(0)};
                senders |= (uint32_t)from << (4 * jj);
                if (!nonzero && bad == 0) bad = jd + 1;
                if (rank == 0 && tid == 0) piv[jd] = bp;
                if (!done) {
                    if (pos == bp) {
                        pos = jd;
                        done = true;
                        s_done[tid] = 1;
                        myq = jj;
                    } else {
                        if (pos == jd) pos = bp;
                        E l;
                        l.re = a[jj].re * inv.re - (C ? a[jj].im * inv.im : T(0));
                        l.im = C ? a[jj].re * inv.im + a[jj].im * inv.re : T(0);
                        a[jj] = l;
#pragma unroll
                        for (int c = jj + 1; c < PCL_SB; ++c) {
                            const E u = prow[c];
                            a[c].re -= l.re * u.re - (C ? l.im * u.im : T(0));
                            if (C) a[c].im -= l.re * u.im + l.im * u.re;
                        }
                    }
                }
                own = from == rank ? min(gb.row, ldc - 1) : -1;
            }
        }
        push_row(PCL_SB - 1);
        if (mine)
#pragma unroll
            for (int c = 0; c < PCL_SB; ++c)
                if (c < sw) st_p<T, C>(P, (jb + c) * ldc + tid, a[c]);
        if (nt > 0) {
            if (!lost) lost = !bar_wait(&sh.u_bar, parity);
            __syncthreads();
            if (tid < nt) {
                E x[PCL_SB];
#pragma unroll
                for (int q = 0; q < PCL_SB; ++q) {
                    x[q] = sh.U[q][tid];
#pragma unroll
                    for (int w = 0; w < q; ++w) {
                        const E l = sh.rec[q][(senders >> (4 * q)) & 15u][w];
                        x[q].re -= l.re * x[w].re - (C ? l.im * x[w].im : T(0));
                        if (C) x[q].im -= l.re * x[w].im + l.im * x[w].re;
                    }
                    sh.U[q][tid] = x[q];
                }
            }
            __syncthreads();
            panel_rank8<T, C, THREADS>(P, ldc, cnt, jb, jb + PCL_SB, nt, sh.U, s_done, a, !done);
            if (myq >= 0)
                for (int c = 0; c < nt; ++c) st_p<T, C>(P, (jb + PCL_SB + c) * ldc + tid, sh.U[myq][c]);
            __syncthreads();
        }
    }
    if (rank == 0 && tid == 0 && bad != 0 && *info == 0) *info = bad;
    if (lost) atomicExch(flag, BEM_ERR_TIMEOUT);
    if (mine) {
        s_pos[tid] = pos;
        src[pos - k0] = r0 + tid;
    }
    __syncthreads();
    for (int r = wid; r < cnt; r += NW)
        for (int c = lane; c < nb; c += 32) st<T, C>(A, (int64_t)s_pos[r] * lda + k0 + c, ld_p<T, C>(P, c * ldc + r));
    cluster.sync();  // no CTA leaves while another may still push to it
}

// row swaps of one panel applied to the columns from c0 (to n) outside [x0, x1)
template <typename T, bool C>
__global__ void laswp_kernel(T* A, int64_t lda, int c0, int n, int x0, int x1, int k0, int nb, const int32_t* piv) {
    int c = c0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n || (c >= x0 && c < x1)) return;
    for (int j = 0; j < nb; ++j) {
        int r1 = k0 + j, r2 = piv[k0 + j];
        if (r1 == r2) continue;
        El<T, C> a = ld<T, C>(A, (int64_t)r1 * lda + c);
        El<T, C> b = ld<T, C>(A, (int64_t)r2 * lda + c);
        st<T, C>(A, (int64_t)r1 * lda + c, b);
        st<T, C>(A, (int64_t)r2 * lda + c, a);
    }
}

// U12 = L11^{-1} A12 (unit lower L11 = rows/cols k0..k0+nb): L11 and a tile
// of TRSM_COLS columns of A12 in shared memory, forward substitution in blocks
// of TRSM_B rows: one thread per column solves a block's triangle in
// registers, then all threads apply its rank-TRSM_B update to the rows below
// (TRSM_ROWS threads a column).  The substitution is a serial chain, so its
// length in dependent shared-memory reads is what it costs: nb / TRSM_B block
// steps instead of nb^2 / 2 terms one after the other.  Measured (2999
// complex, a step): 15 us against 90 us with one thread per column throughout.
constexpr int TRSM_COLS = 32;
constexpr int TRSM_B = 8;
constexpr int TRSM_ROWS = 8;

template <typename T, bool C>
__global__ void __launch_bounds__(TRSM_COLS* TRSM_ROWS) trsm_kernel(T* A, int64_t lda, int col0, int n, int k0,
                                                                              int nb) {
    using E = El<T, C>;
    constexpr int THREADS = TRSM_COLS * TRSM_ROWS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    E* L = reinterpret_cast<E*>(smem_raw);  // [nb][nb]
    E* X = L + nb * nb;                     // [nb][TRSM_COLS]
    const int c0 = col0 + blockIdx.x * TRSM_COLS;  // of the columns [col0, n)
    const int ncol = min(TRSM_COLS, n - c0);
    for (int idx = threadIdx.x; idx < nb * nb; idx += THREADS) {
        int r = idx / nb, c = idx - r * nb;
        L[idx] = ld<T, C>(A, (int64_t)(k0 + r) * lda + k0 + c);
    }
    for (int idx = threadIdx.x; idx < nb * TRSM_COLS; idx += THREADS) {
        int r = idx / TRSM_COLS, c = idx - r * TRSM_COLS;
        X[idx] = c < ncol ? ld<T, C>(A, (int64_t)(k0 + r) * lda + c0 + c) : E{T(0), T(0)};
    }
    __syncthreads();
    const int c = threadIdx.x % TRSM_COLS, part = threadIdx.x / TRSM_COLS;
    for (int b = 0; b < nb; b += TRSM_B) {
        const int w = min(TRSM_B, nb - b);
        E x[TRSM_B];
        if (part == 0) {
#pragma unroll
            for (int q = 0; q < TRSM_B; ++q)
                if (q < w) {
                    x[q] = X[(b + q) * TRSM_COLS + c];
#pragma unroll
                    for (int p = 0; p < q; ++p) {
                        const E l = L[(b + q) * nb + b + p];
                        x[q].re -= l.re * x[p].re - (C ? l.im * x[p].im : T(0));
                        if (C) x[q].im -= l.re * x[p].im + l.im * x[p].re;
                    }
                    X[(b + q) * TRSM_COLS + c] = x[q];
                }
        }
        if (b + w >= nb) break;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < TRSM_B; ++q) x[q] = X[(b + q) * TRSM_COLS + c];
        for (int r = b + TRSM_B + part; r < nb; r += TRSM_ROWS) {
            E acc = X[r * TRSM_COLS + c];
#pragma unroll
            for (int q = 0; q < TRSM_B; ++q) {
                const E l = L[r * nb + b + q];
                acc.re -= l.re * x[q].re - (C ? l.im * x[q].im : T(0));
                if (C) acc.im -= l.re * x[q].im + l.im * x[q].re;
            }
            X[r * TRSM_COLS + c] = acc;
        }
        __syncthreads();
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nb * TRSM_COLS; idx += THREADS) {
        int r = idx / TRSM_COLS, cc = idx - r * TRSM_COLS;
        if (cc < ncol) st<T, C>(A, (int64_t)(k0 + r) * lda + c0 + cc, X[idx]);
    }
}

// The next panel's columns [c0, c1) after the cluster's panel at k0 (LU_NB
// columns): row swaps, U12 = L11^{-1} A12 and A22 -= L21 U12 in one launch.
// These columns are the serial chain of the factorisation (panel, its
// application to the next panel, next panel), so what counts is latency: as
// separate launches they cost 5 + 15 + 24 us and three launch gaps a step (2999
// complex), here 21 us.  A
// cluster takes NX_COLS columns, its CTAs a share of the rows each; every CTA
// reads the LU_NB rows of A12 and its own rows at their places before the
// swaps (src, written by the panel), and solves A12 itself.  All reads of A come
// before the cluster barrier and all writes after it, so the swap needs no copy.
// The products run from zero on the FP64 tensor cores and are subtracted once.
constexpr int NX_COLS = 8;
constexpr int NX_LD = LU_NB + 1;  // odd: conflict-free down a column of L11
template <bool C>
__global__ void __launch_bounds__(256) lu_next_kernel(double* A, int64_t lda, int n, int k0, int c0, int c1, int chunk,
                                                      const int32_t* src) {
    using E = El<double, C>;
    constexpr int W = C ? 2 : 1, NP = C ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* L = reinterpret_cast<double*>(smem_raw);  // [LU_NB][NX_LD]
    double* X = L + W * LU_NB * NX_LD;                // [LU_NB][NX_COLS]
    double* Y = X + W * LU_NB * NX_COLS;              // [chunk][NX_COLS]
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int k1 = k0 + LU_NB, r0 = k1 + (int)blockIdx.x * chunk, cnt = max(0, min(chunk, n - r0));
    const int cb = c0 + (int)blockIdx.y * NX_COLS, ncol = min(NX_COLS, c1 - cb);
    const bool whole = reinterpret_cast<uintptr_t>(A) % (W * sizeof(double)) == 0;
    auto fetch = [&](double* dst, int64_t row, int col) {
        const double* a = A + W * (row * lda + col);
        if (whole) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(a), "n"(8 * W));
        } else {
            for (int h = 0; h < W; ++h)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst + h)), "l"(a + h));
        }
    };
    for (int e = tid; e < LU_NB * LU_NB; e += 256) {
        const int r = e / LU_NB, c = e % LU_NB;
        if (c < r) fetch(L + W * (r * NX_LD + c), k0 + r, k0 + c);
    }
    const int cc = tid & 7;  // column of this thread in the copies and the solve
    for (int r = tid >> 3; r < LU_NB + cnt; r += 32) {
        const int row = r < LU_NB ? r : r0 - k1 + r;  // position in the panel
        double* dst = r < LU_NB ? X + W * (r * NX_COLS + cc) : Y + W * ((r - LU_NB) * NX_COLS + cc);
        if (cc < ncol)
            fetch(dst, min(max(src[row], k0), n - 1), cb + cc);
        else
            for (int h = 0; h < W; ++h) dst[h] = 0.0;
    }
    // a warp per 8 x 8 tile of rows; its part of L21, one tile ahead
    const int row8 = lane >> 2, k4 = lane & 3;
    E f[LU_NB / 4];
    auto rows_of = [&](int rt) {
        const int r = rt * 8 + row8;
#pragma unroll
        for (int h = 0; h < LU_NB / 4; ++h)
            f[h] = r < cnt ? ld<double, C>(A, (int64_t)(r0 + r) * lda + k0 + 4 * h + k4) : E{0.0, 0.0};
    };
    rows_of(wid);
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster.sync();
    // X = L11^{-1} X in blocks of TRSM_B rows, as in trsm_kernel
    for (int b = 0; b < LU_NB; b += TRSM_B) {
        E x[TRSM_B];
        if (tid < NX_COLS) {
#pragma unroll
            for (int q = 0; q < TRSM_B; ++q) {
                x[q] = ld_p<double, C>(X, (b + q) * NX_COLS + tid);
#pragma unroll
                for (int p = 0; p < q; ++p) {
                    const E l = ld_p<double, C>(L, (b + q) * NX_LD + b + p);
                    x[q].re -= l.re * x[p].re - (C ? l.im * x[p].im : 0.0);
                    if (C) x[q].im -= l.re * x[p].im + l.im * x[p].re;
                }
                st_p<double, C>(X, (b + q) * NX_COLS + tid, x[q]);
            }
        }
        __syncthreads();
        if (b + TRSM_B >= LU_NB) break;
#pragma unroll
        for (int q = 0; q < TRSM_B; ++q) x[q] = ld_p<double, C>(X, (b + q) * NX_COLS + cc);
        for (int r = b + TRSM_B + (tid >> 3); r < LU_NB; r += 32) {
            E acc = ld_p<double, C>(X, r * NX_COLS + cc);
#pragma unroll
            for (int q = 0; q < TRSM_B; ++q) {
                const E l = ld_p<double, C>(L, r * NX_LD + b + q);
                acc.re -= l.re * x[q].re - (C ? l.im * x[q].im : 0.0);
                if (C) acc.im -= l.re * x[q].im + l.im * x[q].re;
            }
            st_p<double, C>(X, r * NX_COLS + cc, acc);
        }
        __syncthreads();
    }
    if (blockIdx.x == 0)
        for (int r = tid >> 3; r < LU_NB; r += 32)
            if (cc < ncol) st<double, C>(A, (int64_t)(k0 + r) * lda + cb + cc, ld_p<double, C>(X, r * NX_COLS + cc));
    // the real and imaginary products on separate chains
    for (int rt = wid; rt * 8 < cnt; rt += 8) {
        const int r = rt * 8 + row8;
        const bool ok = r < cnt;
        double p[NP][2] = {}, q[NP][2] = {};  // re re, re im; im im, im re
#pragma unroll
        for (int h = 0; h < LU_NB / 4; ++h) {
            const E u = ld_p<double, C>(X, (4 * h + k4) * NX_COLS + row8);
            bem_gemm_detail::dmma_acc(p[0][0], p[0][1], f[h].re, u.re);
            if (C) {
                bem_gemm_detail::dmma_acc(q[0][0], q[0][1], f[h].im, u.im);
                bem_gemm_detail::dmma_acc(p[NP - 1][0], p[NP - 1][1], f[h].re, u.im);
                bem_gemm_detail::dmma_acc(q[NP - 1][0], q[NP - 1][1], f[h].im, u.re);
            }
        }
        rows_of(rt + 8);
        if (ok)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 2 * k4 + e;
                if (c >= ncol) continue;
                E v = ld_p<double, C>(Y, r * NX_COLS + c);
                v.re -= C ? p[0][e] - q[0][e] : p[0][e];
                if (C) v.im -= p[NP - 1][e] + q[NP - 1][e];
                st<double, C>(A, (int64_t)(r0 + r) * lda + cb + c, v);
            }
    }
}

// perm[i] = original row that ends up at row i after the LAPACK swap sequence.
// The swaps are sequential, but a row's path through them is not: each thread
// follows one row (its position moves when a swap names it), with the swap
// targets read in tiles from shared memory.  n threads of n compares, 38 us at
// 3000 against 122 us with the sequence run by one thread.
constexpr int PERM_TILE = 2048;
__global__ void __launch_bounds__(256) piv_to_perm_kernel(const int32_t* piv, int32_t* perm, int n) {
    __shared__ int32_t sp[PERM_TILE];
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    int pos = row;
    for (int i0 = 0; i0 < n; i0 += PERM_TILE) {
        const int m = min(PERM_TILE, n - i0);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const int p = piv[i0 + i];
            sp[i] = p >= 0 && p < n ? p : i0 + i;
        }
        __syncthreads();
        for (int i = 0; i < m; ++i) {
            const int a = i0 + i, p = sp[i];
            pos = pos == a ? p : (pos == p ? a : pos);
        }
    }
    if (row < n) perm[pos] = row;
}

// right-hand sides of the triangular solve, each contiguous and permuted, and back
__global__ void gather_rhs_kernel(const double* b, int64_t ldb, const int32_t* perm, double* out, int64_t vs, int n,
                                  int nrhs, int W) {
    const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (id >= (int64_t)n * nrhs) return;
    const int i = (int)(id / nrhs), c = (int)(id % nrhs);
    const int64_t src = W * ((int64_t)perm[i] * ldb + c);
    for (int w = 0; w < W; ++w) out[c * vs + (int64_t)W * i + w] = bem_not_pending(b[src + w]);
}
__global__ void scatter_rhs_kernel(const double* x, int64_t vs, double* b, int64_t ldb, int n, int nrhs, int W) {
    const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (id >= (int64_t)n * nrhs) return;
    const int i = (int)(id / nrhs), c = (int)(id % nrhs);
    for (int w = 0; w < W; ++w) b[W * ((int64_t)i * ldb + c) + w] = x[c * vs + (int64_t)W * i + w];
}

// sum_q A[q] x[q] of one row over a warp.  What counts is bytes in flight: U
// elements a lane are loaded before the first is used, complex ones by one load
// where `al` (A and x aligned) allows it.  Streaming loads leave the caches to x
// and other operands; a real matrix that fits the L2 cache is read without the
// hint (stream false), so that a repeated product finds it there.  Complex rows
// start at different chunks, since rows a multiple of a few KB apart otherwise keep
// asking the same memory channels.  Measured, a product repeated / after the cache
// was flushed, against one element in flight a lane: complex FP64 2999 x 2999 51 ->
// 33 / 55 -> 33 us, 6000 x 6000 108 -> 109 / 121 -> 114 us (without the rotation
// 116 / 131), 8000 x 8000 231 -> 171 / 242 -> 178 us; real FP64 3000 x 3000 19 ->
// 19 / 32 -> 30 us (with the hint 27 / 25), 6000 x 6000 62 -> 57 / 73 -> 58 us;
// complex FP32 8000 x 8000 125 -> 108 / 130 -> 107 us.
template <typename T, bool C, bool STREAM>
__device__ __forceinline__ void row_dot_as(const T* a, const double* x, int64_t n, int64_t row, bool al, double& sr,
                                           double& si) {
    constexpr int U = C && sizeof(T) == 4 ? 4 : 8;
    using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    const int lane = threadIdx.x & 31;
    double r[2] = {0.0, 0.0}, m[2] = {0.0, 0.0};
    auto add = [&](int u, El<T, C> e, double xr, double xi) {
        r[u & 1] += (double)e.re * xr - (C ? (double)e.im * xi : 0.0);
        if (C) m[u & 1] += (double)e.re * xi + (double)e.im * xr;
    };
    const int64_t chunks = n / (U * 32);
    int64_t c = C && chunks ? row % chunks : 0;
    for (int64_t k = 0; k < chunks; ++k) {
        const int64_t q = c * (U * 32) + lane;
        El<T, C> e[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!C) {
                e[u] = El<T, C>{STREAM ? __ldcs(a + q + 32 * u) : a[q + 32 * u], T(0)};
            } else if (al) {
                const V2 v = __ldcs(reinterpret_cast<const V2*>(a) + q + 32 * u);
                e[u].re = v.x;
                e[u].im = v.y;
            } else {
                e[u] = ld<T, C>(a, q + 32 * u);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = q + 32 * u;
            if (C && al) {
                const double2 v = reinterpret_cast<const double2*>(x)[i];
                add(u, e[u], v.x, v.y);
            } else {
                add(u, e[u], C ? x[2 * i] : x[i], C ? x[2 * i + 1] : 0.0);
            }
        }
        if (++c == chunks) c = 0;
    }
    for (int64_t q = chunks * (U * 32) + lane; q < n; q += 32)
        add(0, ld<T, C>(a, q), C ? x[2 * q] : x[q], C ? x[2 * q + 1] : 0.0);
    sr = r[0] + r[1];
    si = m[0] + m[1];
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        if (C) si += __shfl_xor_sync(0xffffffffu, si, o);
    }
}
template <typename T, bool C>
__device__ __forceinline__ void row_dot(const T* a, const double* x, int64_t n, int64_t row, bool al, bool stream,
                                        double& sr, double& si) {
    if (C || stream)
        row_dot_as<T, C, true>(a, x, n, row, al, sr, si);
    else
        row_dot_as<T, C, false>(a, x, n, row, al, sr, si);
}
// complex elements of A and x can be read 16 bytes at a time (rows of A too: lda counts elements)
__device__ __forceinline__ bool aligned16(const void* a, const void* x) {
    return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(x)) % 16 == 0;
}

// y = alpha A x + beta y, A stored as T (real/complex), x/y FP64
template <typename T, bool C>
__global__ void __launch_bounds__(256) gemv_kernel(const T* A, int64_t m, int64_t n, int64_t lda, const double* x,
                                                    double* y, double alpha, double beta, int stream) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= m) return;
    double sr, si;
    row_dot<T, C>(A + (C ? 2 : 1) * row * lda, x, n, row, aligned16(A, x), stream != 0, sr, si);
    if (lane == 0) {
        if (C) {
            double yr = beta == 0.0 ? 0.0 : beta * y[2 * row];
            double yi = beta == 0.0 ? 0.0 : beta * y[2 * row + 1];
            y[2 * row] = yr + alpha * sr;
            y[2 * row + 1] = yi + alpha * si;
        } else {
            double yr = beta == 0.0 ? 0.0 : beta * y[row];
            y[row] = yr + alpha * sr;
        }
    }
}

__global__ void sumsq_kernel(const double* v, int64_t n, double* out) {
    __shared__ double s[8];
    double acc = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        acc += v[i] * v[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
        atomicAdd(out, t);
    }
}

__global__ void axpy_kernel(double* y, const double* x, int64_t n, double a) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) y[i] += a * x[i];
}

// ---- asynchronous refinement: state and step kernels ----------------------
// Every kernel of an iteration returns at once when `done` is set, so the
// host can queue several iterations and synchronise once.
struct RefState {
    double bn2;    // ||b||^2
    double rn2;    // ||r||^2 of the current iteration (accumulated)
    double prev2;  // ||r||^2 of the previous iteration
    double rel2;   // last ||r||^2 / ||b||^2
    int done;      // 0 running, 1 converged, 2 stagnated, 3 maxit
    int it;        // iterations completed
};

__global__ void ref_init_kernel(RefState* st) {
    st->bn2 = st->rn2 = st->prev2 = st->rel2 = 0.0;
    st->done = 0;
    st->it = 0;
}

__global__ void ref_start_kernel(RefState* st) {
    st->prev2 = st->bn2;
    if (st->bn2 == 0.0) st->done = 1;  // b = 0: x = 0 is exact
}

__global__ void ref_axpy_kernel(double* y, const double* x, int64_t n, const RefState* st) {
    if (st->done) return;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) y[i] += x[i];
}

__global__ void ref_sumsq_kernel(const double* v, int64_t n, RefState* st) {
    if (st->done) return;
    __shared__ double s[8];
    double acc = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        acc += v[i] * v[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
        atomicAdd(&st->rn2, t);
    }
}

// r = b - A x, one warp per row (the FP64 residual of the refinement)
template <typename T, bool C>
__global__ void __launch_bounds__(256) ref_residual_kernel(const T* A, int64_t n, int64_t lda, const double* x,
                                                            const double* b, double* r, const RefState* st,
                                                            int stream) {
    if (st->done) return;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    double sr, si;
    row_dot<T, C>(A + (C ? 2 : 1) * row * lda, x, n, row, aligned16(A, x), stream != 0, sr, si);
    if (lane == 0) {
        if (C) {
            r[2 * row] = b[2 * row] - sr;
            r[2 * row + 1] = b[2 * row + 1] - si;
        } else {
            r[row] = b[row] - sr;
        }
    }
}

// convergence test of one iteration: relative residual <= tol (done = 1),
// stagnation after three iterations (residual above half the previous, 2),
// iteration cap (3)
__global__ void ref_decide_kernel(RefState* st, double tol2, int maxit) {
    if (st->done) return;
    st->it += 1;
    const double rn2 = st->rn2;
    st->rn2 = 0.0;
    st->rel2 = rn2 / st->bn2;
    if (rn2 <= tol2 * st->bn2)
        st->done = 1;
    else if (st->it >= 3 && rn2 > 0.25 * st->prev2)
        st->done = 2;
    else if (st->it >= maxit)
        st->done = 3;
    st->prev2 = rn2;
}

// row_dot's stream: m x n elements do not fit the L2 cache
template <typename T, bool C>
int beyond_l2(const bem_ctx* ctx, int64_t m, int64_t n) {
    return (double)m * (double)n * sizeof(T) * (C ? 2 : 1) > (double)ctx->l2_bytes ? 1 : 0;
}

struct LinWs {
    GridBar* bar;
    PivSlot* slots;  // [2][PANEL_MAXB]
    void* rowbuf;    // [2][PANEL_MAXB+1][LU_NB] panel-row copies (16 B per element)
    int32_t* src;    // [PCL_MAXROWS] rows of a cluster's panel: where each came from
};

// at_least: bytes the workspace has to have for a later call too
int linws(bem_ctx* ctx, size_t at_least, LinWs* w) {
    const size_t off_slots = 256;
    const size_t off_rows = off_slots + sizeof(PivSlot) * 2 * PANEL_MAXB;
    const size_t off_src = off_rows + 16 * (size_t)2 * (PANEL_MAXB + 1) * LU_NB;
    const size_t total = off_src + sizeof(int32_t) * PCL_MAXROWS;
    if (int rc = bem_ws_reserve(ctx, std::max(total, at_least))) return rc;
    char* base = (char*)ctx->ws;
    w->bar = (GridBar*)base;
    w->slots = (PivSlot*)(base + off_slots);
    w->rowbuf = (void*)(base + off_rows);
    w->src = (int32_t*)(base + off_src);
    return BEM_OK;
}

int coop_blocks(bem_ctx* ctx, const void* fn, int threads, size_t smem, int want) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    int maxb = per_sm * ctx->num_sms;
    if (maxb < 1) return 0;
    return std::max(1, std::min(want, std::min(maxb, ctx->num_sms)));
}

int check_flag(bem_ctx* ctx, cudaStream_t s, const char* what) {
    int32_t f = 0;
    if (int rc = bem_check_cuda(ctx, cudaMemcpyAsync(&f, ctx->flags + 2, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                                "flag readback"))
        return rc;
    if (int rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), what)) return rc;
    if (f != 0) {
        cudaMemsetAsync(ctx->flags + 2, 0, sizeof(int32_t), s);
        return bem_fail(ctx, BEM_ERR_TIMEOUT, std::string(what) + ": device wait hit its iteration cap");
    }
    return BEM_OK;
}

// The panel on one cluster; 1 when its rows do not fit (the cooperative
// kernel takes those: more than about 3100 complex or 6200 real FP64 rows).
template <typename T, bool C>
int lu_panel_cluster(bem_ctx* ctx, T* A, int64_t lda, int n, int k0, int nb, int32_t* piv, int32_t* info,
                     int32_t* flag, int32_t* src, cudaStream_t s) {
    constexpr size_t E = sizeof(T) * (C ? 2 : 1);
    constexpr size_t FIXED = (sizeof(PanelShared<T, C>) + 15) & ~size_t(15);
    constexpr size_t SMEM = 226 * 1024;
    const int rows = n - k0;
    // a thread per row: 64 to 512 rows a CTA; 16 CTAs from 1024 rows on (the
    // rank-8 updates shrink with the rows a CTA has, the barrier grows little)
    int nc = 1;
    while (nc < PCL_MAXC && (rows + nc - 1) / nc > 64) nc *= 2;
    const int chunk = (rows + nc - 1) / nc;
    const int ldc = chunk | 1;  // odd column stride: no bank conflict along a row
    const size_t smem = FIXED + E * LU_NB * ldc + (sizeof(int) + 1) * (size_t)chunk;
    if (chunk > 512 || smem > SMEM) return 1;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)nc);
    // all of an SM's shared memory: the panel is the factorisation's serial
    // chain, so no CTA of the update beside it (look-ahead) shares its SMs
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    auto go = [&](auto* kernel, int threads) -> int {
        cfg.blockDim = dim3((unsigned)threads);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
        if (nc > 8) {
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            int fit = 0;
            if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) {
                cudaGetLastError();
                return 1;
            }
        }
        ctx->launches++;
        return bem_check_cuda(ctx, cudaLaunchKernelEx(&cfg, kernel, A, lda, n, k0, nb, chunk, ldc, piv, info, flag, src),
                              "lu_panel_cluster_kernel");
    };
    return chunk <= 256 ? go(lu_panel_cluster_kernel<T, C, 256>, 256) : go(lu_panel_cluster_kernel<T, C, 512>, 512);
}

// queues lu_next_kernel for the columns [c0, c1) (rows below k0 + LU_NB exist)
template <bool C>
int lu_next(bem_ctx* ctx, double* A, int64_t lda, int n, int k0, int c0, int c1, const int32_t* src, cudaStream_t s) {
    constexpr size_t E = sizeof(double) * (C ? 2 : 1);
    const int rows = n - k0 - LU_NB;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    int nc = 1;
    while (nc < PCL_MAXC && (rows + nc - 1) / nc > 32) nc *= 2;
    int chunk = 0;
    for (;; nc = 8) {
        chunk = (rows + nc - 1) / nc;
        at[0].val.clusterDim.x = (unsigned)nc;
        cfg.gridDim = dim3((unsigned)nc, (unsigned)((c1 - c0 + NX_COLS - 1) / NX_COLS));
        cfg.dynamicSmemBytes = E * (LU_NB * NX_LD + (LU_NB + (size_t)chunk) * NX_COLS);
        cudaFuncSetAttribute(lu_next_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
        if (nc <= 8) break;
        cudaFuncSetAttribute(lu_next_kernel<C>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, lu_next_kernel<C>, &cfg) == cudaSuccess && fit >= 1) break;
        cudaGetLastError();
    }
    ctx->launches++;
    return bem_check_cuda(ctx, cudaLaunchKernelEx(&cfg, lu_next_kernel<C>, A, lda, n, k0, c0, c1, chunk, src),
                          "lu_next_kernel");
}

// Workspace of lu_solve: permutation, the inverses of the diagonal tiles (FP64),
// three sets of nrhs vectors vs doubles apart.
struct SolveLayout {
    size_t off_dinv, off_vec, total;
    int64_t vs;
    SolveLayout(int W, int64_t n, int64_t nrhs) {
        auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
        off_dinv = up(sizeof(int32_t) * (size_t)n);
        off_vec = off_dinv + up(2 * sizeof(double) * (size_t)bem_lu_dinv_elems(n));
        vs = (int64_t)(up(sizeof(double) * W * (size_t)n) / sizeof(double));
        total = off_vec + 3 * sizeof(double) * (size_t)(nrhs * vs);
    }
};

template <typename T, bool C>
int lu_factor_t(bem_ctx* ctx, T* A, int64_t n, int64_t lda, int32_t* piv, int32_t* info, cudaStream_t s) {
    // one growth of the workspace for the factorisation and a solve with it
    LinWs w;
    if (int rc = linws(ctx, SolveLayout(C ? 2 : 1, n, 1).total, &w)) return rc;
    cudaMemsetAsync(w.bar, 0, sizeof(GridBar), s);
    cudaMemsetAsync(info, 0, sizeof(int32_t), s);
    cudaMemsetAsync(ctx->flags + 2, 0, sizeof(int32_t), s);
    const int threads = 256;
    int32_t* flag = ctx->flags + 2;
    // CTAs of the panel: at most one per SM and at most PANEL_MAXB; each keeps
    // its row slice in shared memory when it fits in PANEL_SMEM bytes
    const size_t PANEL_SMEM = 200 * 1024;
    const int maxb = std::min(PANEL_MAXB, ctx->num_sms);
    const size_t smem_full = sizeof(El<T, C>) * (size_t)((n + maxb - 1) / maxb) * LU_NB;
    const bool use_smem = smem_full <= PANEL_SMEM;
    const void* pk = use_smem ? (const void*)lu_panel_kernel<T, C, true> : (const void*)lu_panel_kernel<T, C, false>;
    if (use_smem)
        cudaFuncSetAttribute(lu_panel_kernel<T, C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)PANEL_SMEM);
    int nblk = std::min(maxb, coop_blocks(ctx, pk, threads, use_smem ? smem_full : 0, maxb));
    if (nblk < 1) return bem_fail(ctx, BEM_ERR_CUDA, "lu_panel_kernel cannot be made co-resident");
    if (use_smem && sizeof(El<T, C>) * (size_t)std::max<int64_t>(32, (n + nblk - 1) / nblk) * LU_NB > PANEL_SMEM)
        return bem_fail(ctx, BEM_ERR_CUDA, "lu_panel_kernel: fewer co-resident CTAs than SMs");
    // Look-ahead: the panel occupies one cluster, so the next panel's columns are
    // brought up to date first, on the high-priority side stream, and factored
    // there while the caller's stream works on all other columns (2999 complex:
    // 10.5 -> 7.3 ms with the solves).  FP32 stays on one stream (its
    // tensor-core updates share a scratch).
    const bool ahead = sizeof(T) == 8;
    if (ahead)
        if (int rc = bem_lookahead_stream(ctx)) return rc;
    const cudaStream_t sp = ahead ? ctx->aux : s;
    auto order = [&](cudaStream_t first, cudaEvent_t ev, cudaStream_t then) {
        if (!ahead) return;
        cudaEventRecord(ev, first);
        cudaStreamWaitEvent(then, ev, 0);
    };
    // panel k0 applied to the columns [c0, c1), and its swaps to the finished ones left of `left`
    const size_t tsmem_max = sizeof(El<T, C>) * LU_NB * (LU_NB + TRSM_COLS);
    cudaFuncSetAttribute(trsm_kernel<T, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem_max);
    auto apply = [&](int k0, int nb, int left, int c0, int c1, cudaStream_t st) -> int {
        const int first = left > 0 ? 0 : c0;
        if (c1 > first) {
            laswp_kernel<T, C><<<(unsigned)((c1 - first + 255) / 256), 256, 0, st>>>(A, lda, first, c1, left, c0, k0, nb, piv);
            ctx->launches++;
        }
        const int cols = c1 - c0, k1 = k0 + nb;
        if (cols <= 0) return BEM_OK;
        trsm_kernel<T, C><<<(unsigned)((cols + TRSM_COLS - 1) / TRSM_COLS), TRSM_COLS * TRSM_ROWS,
                            sizeof(El<T, C>) * nb * (nb + TRSM_COLS), st>>>(A, lda, c0, c1, k0, nb);
        ctx->launches++;
        // A22 -= L21 U12
        auto at = [&](int64_t r, int64_t c) { return A + (C ? 2 : 1) * (r * lda + c); };
        return bem_gemm_update<T, C>(ctx, at(k1, c0), at(k1, k0), at(k0, c0), n - k1, cols, nb, lda, st);
    };
    auto steps = [&]() -> int {
        for (int64_t k0 = 0; k0 < n; k0 += LU_NB) {
            int nb = (int)std::min<int64_t>(LU_NB, n - k0);
            int rows = (int)(n - k0);
            int ni = (int)n, k0i = (int)k0;
            const int rc = lu_panel_cluster<T, C>(ctx, A, lda, ni, k0i, nb, piv, info, flag, w.src, sp);
            if (rc < 0) return rc;
            if (rc == 1) {
                // the panel does not fit a cluster's shared memory
                order(sp, ctx->ev_diag, s);
                int blocks = std::min(nblk, std::max(1, (rows + 31) / 32));
                int chunk = (rows + blocks - 1) / blocks;
                El<T, C>* rb = (El<T, C>*)w.rowbuf;
                size_t smem = use_smem ? sizeof(El<T, C>) * (size_t)chunk * LU_NB : 0;
                void* args[] = {&A, &lda, &ni, &k0i, &nb, &chunk, &piv, &info, &w.bar, &w.slots, &rb, &flag};
                if (int e = bem_check_cuda(ctx, cudaLaunchCooperativeKernel(pk, blocks, threads, args, smem, s),
                                           "lu_panel_kernel"))
                    return e;
                ctx->launches++;
                order(s, ctx->ev_next, sp);
            }
            const int k1 = k0i + nb, k2 = ahead ? std::min(ni, k1 + LU_NB) : k1;
            order(sp, ctx->ev_diag, s);
            if (k2 > k1) {
                // the columns' earlier updates ran on s
                if (ahead) cudaStreamWaitEvent(sp, ctx->ev_next, 0);
                if constexpr (sizeof(T) == 8) {
                    if (int e = rc == 1 ? apply(k0i, nb, 0, k1, k2, sp)
                                        : lu_next<C>(ctx, A, lda, ni, k0i, k1, k2, w.src, sp))
                        return e;
                }
            }
            if (int e = apply(k0i, nb, k0i, k2, ni, s)) return e;
            if (ahead) cudaEventRecord(ctx->ev_next, s);
            if (int e = bem_check_cuda(ctx, cudaGetLastError(), "lu step")) return e;
        }
        return BEM_OK;
    };
    order(s, ctx->ev_next, sp);
    const int rc = steps();
    order(sp, ctx->ev_diag, s);
    if (rc) return rc;
    return check_flag(ctx, s, "lu_factor");
}

template <typename T, bool C>
int lu_solve_t(bem_ctx* ctx, const T* LU, int64_t n, int64_t lda, const int32_t* piv, double* b, int64_t nrhs,
               int64_t ldb, cudaStream_t s) {
    if (nrhs < 1 || nrhs > 8) return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve supports 1..8 right-hand sides");
    // no larger size has been run (a complex FP64 factor of 51200 rows is 42 GB)
    if (n > 51200) return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: n > 51200");
    const int W = C ? 2 : 1;
    const SolveLayout lay(W, n, nrhs);
    if (int rc = bem_ws_reserve(ctx, lay.total)) return rc;
    const int64_t vs = lay.vs;
    char* base = (char*)ctx->ws;
    int32_t* perm = (int32_t*)base;
    void* dinv = base + lay.off_dinv;
    double* vb = (double*)(base + lay.off_vec);
    double *vy = vb + nrhs * vs, *vx = vy + nrhs * vs;
    int32_t* flag = ctx->flags + 2;
    cudaMemsetAsync(flag, 0, sizeof(int32_t), s);
    const int dtype = sizeof(T) == 8 ? (C ? BEM_C128 : BEM_F64) : (C ? BEM_C64 : BEM_F32);
    piv_to_perm_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(piv, perm, (int)n);
    const unsigned blocks = (unsigned)((n * nrhs + 255) / 256);
    gather_rhs_kernel<<<blocks, 256, 0, s>>>(b, ldb, perm, vb, vs, (int)n, (int)nrhs, W);
    ctx->launches += 2;
    if (n <= BEM_SMALL_SOLVE) {
        if (int rc = bem_lu_small_solve(ctx, dtype, LU, n, lda, vb, vx, (int)nrhs, vs, s)) return rc;
    } else {
        if (int rc = bem_solve_inverses(ctx, dtype, LU, n, lda, dinv, s)) return rc;
        if (int rc = bem_lu_tri_solve(ctx, dtype, LU, n, lda, dinv, vb, vy, vx, (int)nrhs, vs, flag, s)) return rc;
    }
    scatter_rhs_kernel<<<blocks, 256, 0, s>>>(vx, vs, b, ldb, (int)n, (int)nrhs, W);
    ctx->launches++;
    if (int rc = bem_check_cuda(ctx, cudaGetLastError(), "lu_solve")) return rc;
    return check_flag(ctx, s, "lu_solve");
}

// Refinement with the tile-pivoted factor, queued in batches of iterations
// with one synchronisation per batch (normally one per call): the convergence
// test runs on the device and the remaining kernels of a finished refinement
// return at once.  Same iterations and stopping rules as the synchronous
// loop of bem_refine_solve.
int refine_async(bem_ctx* ctx, bool C, const void* A_hi, const void* LU_lo, const int32_t* piv, const void* dinv,
                 int64_t n, int64_t lda, const double* b, double* x, double tol, int maxit, int* iters,
                 double* relres, cudaStream_t s) {
    const int W = C ? 2 : 1;
    const int64_t nd = W * n;
    // r (nd) and the state
    double* r = nullptr;
    if (int rc = bem_check_cuda(ctx, cudaMallocAsync((void**)&r, sizeof(double) * nd + 64, s), "refine alloc"))
        return rc;
    RefState* st = reinterpret_cast<RefState*>(r + nd);
    int rc = BEM_OK;
    const unsigned vblocks = (unsigned)((nd + 255) / 256);
    const unsigned sblocks = (unsigned)std::min<int64_t>(ctx->num_sms * 4, (nd + 255) / 256);
    ref_init_kernel<<<1, 1, 0, s>>>(st);
    sumsq_kernel<<<sblocks, 256, 0, s>>>(b, nd, &st->bn2);
    ref_start_kernel<<<1, 1, 0, s>>>(st);
    ctx->launches += 3;
    cudaMemsetAsync(ctx->flags + 3, 0, sizeof(int32_t), s);
    cudaMemsetAsync(x, 0, sizeof(double) * nd, s);
    cudaMemcpyAsync(r, b, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s);
    const int* skip = &st->done;
    RefState h{};
    int32_t flg[2] = {0, 0};
    int queued = 0;
    while (rc == BEM_OK) {
        const int batch = std::min(3, maxit - queued);
        for (int i = 0; i < batch && rc == BEM_OK; ++i) {
            double* d = nullptr;
            rc = bem_tiled_precond_async(ctx, C ? BEM_C64 : BEM_F32, LU_lo, n, lda, piv, dinv, r, &d, skip, s);
            if (rc) break;
            ref_axpy_kernel<<<vblocks, 256, 0, s>>>(x, d, nd, st);
            const unsigned rblocks = (unsigned)((n + 7) / 8);
            if (C)
                ref_residual_kernel<double, true><<<rblocks, 256, 0, s>>>((const double*)A_hi, n, lda, x, b, r, st,
                                                                         beyond_l2<double, true>(ctx, n, n));
            else
                ref_residual_kernel<double, false><<<rblocks, 256, 0, s>>>((const double*)A_hi, n, lda, x, b, r, st,
                                                                          beyond_l2<double, false>(ctx, n, n));
            ref_sumsq_kernel<<<sblocks, 256, 0, s>>>(r, nd, st);
            ref_decide_kernel<<<1, 1, 0, s>>>(st, tol * tol, maxit);
            ctx->launches += 4;
            rc = bem_check_cuda(ctx, cudaGetLastError(), "refinement step");
            ++queued;
        }
        if (rc) break;
        cudaMemcpyAsync(&h, st, sizeof(RefState), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&flg[0], ctx->flags + 3, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&flg[1], ctx->flags + 4, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
        rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "refinement");
        if (rc) break;
        if ((rc = bem_take_factor_error(ctx, flg[1], s))) break;
        if (flg[0] != 0) {
            rc = bem_fail(ctx, BEM_ERR_TIMEOUT, "tiled solve: a ready-flag wait hit its iteration cap");
            break;
        }
        if (h.done != 0 || queued >= maxit) break;
    }
    cudaFreeAsync(r, s);
    if (rc) return rc;
    if (iters) *iters = h.it;
    if (relres) *relres = std::sqrt(h.rel2);
    if (h.done != 1) return bem_fail(ctx, BEM_ERR_NOCONVERGE, "refinement did not reach tol in maxit iterations");
    return BEM_OK;
}

// ---- GMRES: block inner products and updates on FP64 vectors ------------
// out[i] = sum_q conj(V_i[q]) w[q] for the k vectors V_i (stride nd doubles);
// grid (chunks, k), partial sums of a chunk added atomically
template <bool C>
__global__ void gm_dot_kernel(const double* V, int64_t nd, int k, const double* w, double* out) {
    __shared__ double s_re[8], s_im[8];
    const int i = blockIdx.y;
    const double* v = V + (int64_t)i * nd;
    const int W = C ? 2 : 1;
    const int64_t n = nd / W;
    double re = 0.0, im = 0.0;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        if (C) {
            const double vr = v[2 * q], vi = v[2 * q + 1], wr = w[2 * q], wi = w[2 * q + 1];
            re += vr * wr + vi * wi;
            im += vr * wi - vi * wr;
        } else {
            re += v[q] * w[q];
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_re[threadIdx.x >> 5] = re;
        s_im[threadIdx.x >> 5] = im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tr = 0.0, ti = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
            tr += s_re[q];
            ti += s_im[q];
        }
        atomicAdd(out + 2 * i, tr);
        if (C) atomicAdd(out + 2 * i + 1, ti);
    }
}

// w[q] -= sum_i V_i[q] h_i (h: k complex values, interleaved; real part only
// when !C)
template <bool C>
__global__ void gm_update_kernel(double* w, const double* V, int64_t nd, int k, const double* h) {
    const int W = C ? 2 : 1;
    const int64_t n = nd / W;
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    double ar = 0.0, ai = 0.0;
    for (int i = 0; i < k; ++i) {
        const double* v = V + (int64_t)i * nd;
        const double hr = h[2 * i], hi = h[2 * i + 1];
        if (C) {
            const double vr = v[2 * q], vi = v[2 * q + 1];
            ar += vr * hr - vi * hi;
            ai += vr * hi + vi * hr;
        } else {
            ar += v[q] * hr;
        }
    }
    if (C) {
        w[2 * q] -= ar;
        w[2 * q + 1] -= ai;
    } else {
        w[q] -= ar;
    }
}

__global__ void gm_scale_kernel(double* dst, const double* src, int64_t nd, double a) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < nd) dst[i] = a * src[i];
}

// Restarted GMRES(m) in FP64 on A_hi x = b, right-preconditioned by the
// low-precision factors (tile-pivoted when dinv != NULL, else partial
// pivoting).  Arnoldi with classical Gram-Schmidt applied twice, Givens
// rotations of the Hessenberg matrix on the host.  Each restart starts from
// the true FP64 residual; a restart cycle that no longer halves it ends the
// iteration once the residual is <= accept (its floor is about
// eps * cond(A)).
}  // namespace

int bem_fgmres(bem_ctx* ctx, bool C, int64_t n, const std::function<int(const double*, double*)>& apply_op,
               const std::function<int(double*)>& precond, const double* b, double* x, double tol, int maxit,
               int restart, double accept, int* iters, double* relres, cudaStream_t s) {
    const int W = C ? 2 : 1;
    const int64_t nd = W * n;
    const int m = std::max(1, std::min(restart, 200));
    // V (m+1 vectors), Z (m vectors), w, r, dots (2 (m+1) doubles)
    const size_t doubles = (size_t)(2 * m + 3) * nd + 2 * (m + 2);
    double* buf = nullptr;
    if (int rc = bem_check_cuda(ctx, cudaMallocAsync((void**)&buf, sizeof(double) * doubles, s), "gmres alloc"))
        return rc;
    double* V = buf;
    double* Z = V + (size_t)(m + 1) * nd;
    double* w = Z + (size_t)m * nd;
    double* r = w + nd;
    double* dots = r + nd;
    const unsigned vblocks = (unsigned)((n + 255) / 256);
    const unsigned sblocks = (unsigned)std::min<int64_t>(ctx->num_sms * 4, (nd + 255) / 256);
    const unsigned dchunks = (unsigned)std::min<int64_t>(ctx->num_sms, (n + 255) / 256);
    int rc = BEM_OK;
    auto norm = [&](const double* v, double* out) -> int {
        cudaMemsetAsync(dots, 0, sizeof(double), s);
        sumsq_kernel<<<sblocks, 256, 0, s>>>(v, nd, dots);
        ctx->launches++;
        double h = 0.0;
        if (int e = bem_check_cuda(ctx, cudaMemcpyAsync(&h, dots, sizeof(double), cudaMemcpyDeviceToHost, s),
                                   "gmres norm"))
            return e;
        if (int e = bem_check_cuda(ctx, cudaStreamSynchronize(s), "gmres norm")) return e;
        *out = std::sqrt(h);
        return BEM_OK;
    };
    // r = b - op(x), with w as the scratch of op(x)
    auto residual = [&](double* out_norm) -> int {
        if (int e = apply_op(x, w)) return e;
        if (int e = bem_check_cuda(ctx, cudaMemcpyAsync(r, b, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s),
                                   "r=b"))
            return e;
        axpy_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, s>>>(r, w, nd, -1.0);
        ctx->launches++;
        return norm(r, out_norm);
    };
    using cplx = std::complex<double>;
    double bnorm = 0.0;
    rc = norm(b, &bnorm);
    if (bnorm == 0.0) bnorm = 1.0;
    int its = 0;
    double rel = 0.0, prev = INFINITY;
    bool done = false;
    std::vector<cplx> H((size_t)(m + 1) * m), g(m + 1), cs(m), sn(m), y(m);
    std::vector<double> hbuf(2 * (m + 1));
    while (rc == BEM_OK && its < maxit) {
        double beta = 0.0;
        if ((rc = residual(&beta))) break;
        rel = beta / bnorm;
        if (rel <= tol || (rel > 0.5 * prev && rel <= accept)) {
            done = true;
            break;
        }
        prev = rel;
        const int mm = std::min(m, maxit - its);
        gm_scale_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, s>>>(V, r, nd, 1.0 / beta);
        ctx->launches++;
        std::fill(H.begin(), H.end(), cplx(0.0));
        std::fill(g.begin(), g.end(), cplx(0.0));
        g[0] = beta;
        int jd = 0;
        for (int j = 0; j < mm && rc == BEM_OK; ++j) {
            double* Vj = V + (size_t)j * nd;
            double* Zj = Z + (size_t)j * nd;
            if ((rc = bem_check_cuda(ctx, cudaMemcpyAsync(Zj, Vj, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s),
                                     "z=v")))
                break;
            if ((rc = precond(Zj))) break;
            if ((rc = apply_op(Zj, w))) break;
            for (int pass = 0; pass < 2 && rc == BEM_OK; ++pass) {
                cudaMemsetAsync(dots, 0, sizeof(double) * 2 * (j + 1), s);
                if (C)
                    gm_dot_kernel<true><<<dim3(dchunks, j + 1), 256, 0, s>>>(V, nd, j + 1, w, dots);
                else
                    gm_dot_kernel<false><<<dim3(dchunks, j + 1), 256, 0, s>>>(V, nd, j + 1, w, dots);
                if (C)
                    gm_update_kernel<true><<<vblocks, 256, 0, s>>>(w, V, nd, j + 1, dots);
                else
                    gm_update_kernel<false><<<vblocks, 256, 0, s>>>(w, V, nd, j + 1, dots);
                ctx->launches += 2;
                if ((rc = bem_check_cuda(ctx, cudaMemcpyAsync(hbuf.data(), dots, sizeof(double) * 2 * (j + 1),
                                                              cudaMemcpyDeviceToHost, s), "gmres dots")))
                    break;
                if ((rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "gmres dots"))) break;
                for (int i = 0; i <= j; ++i) H[(size_t)i * m + j] += cplx(hbuf[2 * i], C ? hbuf[2 * i + 1] : 0.0);
            }
            if (rc) break;
            double hn = 0.0;
            if ((rc = norm(w, &hn))) break;
            ++its;
            jd = j + 1;
            if (hn > 0.0) {
                gm_scale_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, s>>>(V + (size_t)(j + 1) * nd, w, nd,
                                                                              1.0 / hn);
                ctx->launches++;
            }
            // Givens rotations: the earlier ones on column j, a new one for H[j+1][j]
            for (int i = 0; i < j; ++i) {
                const cplx a = H[(size_t)i * m + j], c2 = H[(size_t)(i + 1) * m + j];
                H[(size_t)i * m + j] = std::conj(cs[i]) * a + std::conj(sn[i]) * c2;
                H[(size_t)(i + 1) * m + j] = -sn[i] * a + cs[i] * c2;
            }
            const cplx a = H[(size_t)j * m + j];
            const double den = std::sqrt(std::norm(a) + hn * hn);
            if (den > 0.0) {
                cs[j] = a / den;
                sn[j] = cplx(hn / den, 0.0);
            } else {
                cs[j] = 1.0;
                sn[j] = 0.0;
            }
            H[(size_t)j * m + j] = std::conj(cs[j]) * a + std::conj(sn[j]) * hn;
            g[j + 1] = -sn[j] * g[j];
            g[j] = std::conj(cs[j]) * g[j];
            const double est = std::abs(g[j + 1]) / bnorm;
            if (est <= 0.5 * tol || hn == 0.0) break;
        }
        if (rc) break;
        // y = R^{-1} g, x += Z y
        for (int i = jd - 1; i >= 0; --i) {
            cplx t = g[i];
            for (int q = i + 1; q < jd; ++q) t -= H[(size_t)i * m + q] * y[q];
            const cplx d = H[(size_t)i * m + i];
            y[i] = std::abs(d) > 0.0 ? t / d : cplx(0.0);
        }
        for (int i = 0; i < jd; ++i) {
            hbuf[2 * i] = -y[i].real();
            hbuf[2 * i + 1] = -y[i].imag();
        }
        if ((rc = bem_check_cuda(ctx, cudaMemcpyAsync(dots, hbuf.data(), sizeof(double) * 2 * jd,
                                                      cudaMemcpyHostToDevice, s), "gmres y")))
            break;
        if (C)
            gm_update_kernel<true><<<vblocks, 256, 0, s>>>(x, Z, nd, jd, dots);
        else
            gm_update_kernel<false><<<vblocks, 256, 0, s>>>(x, Z, nd, jd, dots);
        ctx->launches++;
        if ((rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "gmres update"))) break;
    }
    if (rc == BEM_OK && !done) {
        double rn = 0.0;
        rc = residual(&rn);
        rel = rn / bnorm;
    }
    cudaFreeAsync(buf, s);
    if (rc) return rc;
    if (iters) *iters = its;
    if (relres) *relres = rel;
    if (!done && rel > std::max(tol, accept))
        return bem_fail(ctx, BEM_ERR_NOCONVERGE, "GMRES-IR did not reach tol in maxit iterations");
    return BEM_OK;
}

namespace {

int gmres_run(bem_ctx* ctx, int dtype_hi, const void* A_hi, const void* LU_lo, const int32_t* piv, const void* dinv,
              int64_t n, int64_t lda, const double* b, double* x, double tol, int maxit, int restart, double accept,
              int* iters, double* relres, cudaStream_t s) {
    const bool C = dtype_hi == BEM_C128;
    const int lo_dtype = C ? BEM_C64 : BEM_F32;
    auto op = [&](const double* z, double* w) -> int {
        return bem_gemv(ctx, dtype_hi, A_hi, n, n, lda, z, w, 1.0, 0.0, s);
    };
    auto precond = [&](double* z) -> int {
        return dinv ? bem_lu_solve_tiled(ctx, lo_dtype, LU_lo, n, lda, piv, dinv, z, s)
                    : bem_lu_solve(ctx, lo_dtype, LU_lo, n, lda, piv, z, 1, 1, s);
    };
    return bem_fgmres(ctx, C, n, op, precond, b, x, tol, maxit, restart, accept, iters, relres, s);
}

// ---------------------------------------------------------------------------
// CGS2 column append of a growing orthonormal basis, one cooperative launch
// (bem_cgs2_append).  With x = v:
//   twice: h = Q^H x, x -= Q h, r += h;   r_jj = ||x||, x /= r_jj;
//   twice: h = Q^H x, x -= Q h;           x /= ||x||;
//   Q[:, j] = x, Rt[j, 0..j-1] = r, Rt[j, j] = r_jj.
// CTA b owns the rows [b rb, (b + 1) rb) of x and keeps them in shared memory
// for the whole step.  A projection is two grid barriers: the partial dot
// products of every CTA over its rows (thread c takes column c, so the reads
// of a Q row are coalesced) go to part[b][c]; CTA c % nblk sums column c over
// the CTAs in a fixed order into h[c]; then every CTA forms its rows of Q h
// (one warp per row, lanes over the columns).  Norms: per-CTA partial sums,
// one barrier, the same fixed-order sum in every CTA.  Ten barriers per
// column, no host synchronisation; the sums are deterministic.
// ---------------------------------------------------------------------------
constexpr int CG_THREADS = 256;

template <bool C>
struct Cx {
    double re, im;
};

template <bool C>
__device__ __forceinline__ Cx<C> cx_ld(const double* p, int64_t i) {
    return C ? Cx<C>{p[2 * i], p[2 * i + 1]} : Cx<C>{p[i], 0.0};
}
template <bool C>
__device__ __forceinline__ void cx_st(double* p, int64_t i, Cx<C> v) {
    if (C) {
        p[2 * i] = v.re;
        p[2 * i + 1] = v.im;
    } else {
        p[i] = v.re;
    }
}

__device__ __forceinline__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < CG_THREADS / 32; ++w) t += red[w];
    __syncthreads();
    if (threadIdx.x == 0) red[0] = t;
    __syncthreads();
    const double out = red[0];
    __syncthreads();
    return out;
}

template <bool C>
__global__ void __launch_bounds__(CG_THREADS) cgs2_append_kernel(double* Q, int64_t n, int64_t ldq, int j,
                                                                  const double* v, int64_t ldv, double* Rt,
                                                                  int64_t ldr, double* part, double* hbuf,
                                                                  double* rbuf, double* npart, GridBar* bar,
                                                                  int32_t* flag) {
    extern __shared__ double cg_smem[];
    __shared__ double red[CG_THREADS / 32];
    const int W = C ? 2 : 1;
    const unsigned nblk = gridDim.x;
    const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t rb = (n + nblk - 1) / nblk;
    const int64_t r0 = (int64_t)b * rb, r1 = r0 + rb < n ? r0 + rb : n;
    const int nr = r1 > r0 ? (int)(r1 - r0) : 0;
    double* sx = cg_smem;                 // [rb] this CTA's rows of x
    double* sh = cg_smem + (size_t)W * rb;  // [j] h
    for (int i = tid; i < nr; i += CG_THREADS) {
        const Cx<C> e = cx_ld<C>(v, (r0 + i) * ldv);
        sx[W * i] = e.re;
        if (C) sx[W * i + 1] = e.im;
    }
    __syncthreads();

    auto project = [&](bool accumulate, bool first) -> bool {
        // partial h over this CTA's rows
        for (int c = tid; c < j; c += CG_THREADS) {
            double ar = 0.0, ai = 0.0;
#pragma unroll 4
            for (int i = 0; i < nr; ++i) {
                const Cx<C> q = cx_ld<C>(Q, (r0 + i) * ldq + c);
                const double xr = sx[W * i], xi = C ? sx[W * i + 1] : 0.0;
                ar += q.re * xr + q.im * xi;  // conj(q) x
                if (C) ai += q.re * xi - q.im * xr;
            }
            cx_st<C>(part, (int64_t)b * j + c, Cx<C>{ar, ai});
        }
        if (!grid_barrier(bar, nblk, flag)) return false;
        // column c: the fixed-order sum over the CTAs
        for (int c = b; c < j; c += (int)nblk) {
            double sr = 0.0, si = 0.0;
            for (unsigned bb = tid; bb < nblk; bb += CG_THREADS) {
                const Cx<C> e = cx_ld<C>(part, (int64_t)bb * j + c);
                sr += e.re;
                si += e.im;
            }
            sr = block_sum(sr, red);
            if (C) si = block_sum(si, red);
            if (tid == 0) {
                cx_st<C>(hbuf, c, Cx<C>{sr, si});
                if (accumulate) {
                    Cx<C> r = first ? Cx<C>{0.0, 0.0} : cx_ld<C>(rbuf, c);
                    cx_st<C>(rbuf, c, Cx<C>{r.re + sr, r.im + si});
                }
            }
        }
        if (!grid_barrier(bar, nblk, flag)) return false;
        for (int c = tid; c < j; c += CG_THREADS) {
            const Cx<C> e = cx_ld<C>(hbuf, c);
            sh[W * c] = e.re;
            if (C) sh[W * c + 1] = e.im;
        }
        __syncthreads();
        // x -= Q h on this CTA's rows
        for (int i = warp; i < nr; i += CG_THREADS / 32) {
            double ar = 0.0, ai = 0.0;
            for (int c = lane; c < j; c += 32) {
                const Cx<C> q = cx_ld<C>(Q, (r0 + i) * ldq + c);
                const double hr = sh[W * c], hi = C ? sh[W * c + 1] : 0.0;
                ar += q.re * hr - q.im * hi;
                if (C) ai += q.re * hi + q.im * hr;
            }
            for (int o = 16; o > 0; o >>= 1) {
                ar += __shfl_xor_sync(0xffffffffu, ar, o);
                if (C) ai += __shfl_xor_sync(0xffffffffu, ai, o);
            }
            if (lane == 0) {
                sx[W * i] -= ar;
                if (C) sx[W * i + 1] -= ai;
            }
        }
        __syncthreads();
        return true;
    };
    auto norm = [&](double& out) -> bool {
        double p = 0.0;
        for (int i = tid; i < nr; i += CG_THREADS) {
            p += sx[W * i] * sx[W * i];
            if (C) p += sx[W * i + 1] * sx[W * i + 1];
        }
        p = block_sum(p, red);
        if (tid == 0) npart[b] = p;
        if (!grid_barrier(bar, nblk, flag)) return false;
        double t = 0.0;
        for (unsigned bb = tid; bb < nblk; bb += CG_THREADS) t += npart[bb];
        t = block_sum(t, red);
        out = sqrt(t > 0.0 ? t : 0.0);
        return true;
    };
    auto scale = [&](double d) {
        const double f = 1.0 / (d > 1e-300 ? d : 1e-300);
        for (int i = tid; i < nr * W; i += CG_THREADS) sx[i] *= f;
        __syncthreads();
    };

    double rjj = 0.0, qn = 0.0;
    if (j > 0 && (!project(true, true) || !project(true, false))) return;
    if (!norm(rjj)) return;
    scale(rjj);
    if (j > 0 && (!project(false, false) || !project(false, false))) return;
    if (!norm(qn)) return;
    scale(qn);
    for (int i = tid; i < nr; i += CG_THREADS)
        cx_st<C>(Q, (r0 + i) * ldq + j, Cx<C>{sx[W * i], C ? sx[W * i + 1] : 0.0});
    if (b == 0) {
        for (int c = tid; c < j; c += CG_THREADS) cx_st<C>(Rt, (int64_t)j * ldr + c, cx_ld<C>(rbuf, c));
        if (tid == 0) cx_st<C>(Rt, (int64_t)j * ldr + j, Cx<C>{rjj, 0.0});
    }
}

template <bool C>
int cgs2_append_t(bem_ctx* ctx, double* Q, int64_t n, int64_t ldq, int j, const double* v, int64_t ldv,
                  double* Rt, int64_t ldr, int check, cudaStream_t s) {
    const int W = C ? 2 : 1;
    int nblk0 = ctx->num_sms;
    const int64_t rb0 = (n + nblk0 - 1) / nblk0;
    const size_t smem = sizeof(double) * W * ((size_t)rb0 + (size_t)std::max(j, 1));
    if (smem > 200 * 1024) return bem_fail(ctx, BEM_ERR_INVALID, "cgs2_append: n or j too large");
    cudaFuncSetAttribute(cgs2_append_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int nblk = coop_blocks(ctx, (const void*)cgs2_append_kernel<C>, CG_THREADS, smem, ctx->num_sms);
    if (nblk < 1) return bem_fail(ctx, BEM_ERR_CUDA, "cgs2_append_kernel cannot be made co-resident");
    if (nblk != nblk0) return bem_fail(ctx, BEM_ERR_CUDA, "cgs2_append_kernel: fewer co-resident CTAs than SMs");
    const size_t jb = (size_t)std::max(j, 1);
    const size_t bytes = 256 + sizeof(double) * W * ((size_t)nblk * jb + 2 * jb) + sizeof(double) * nblk;
    if (int rc = bem_ws_reserve(ctx, bytes)) return rc;
    char* base = static_cast<char*>(ctx->ws);
    GridBar* bar = reinterpret_cast<GridBar*>(base);
    double* part = reinterpret_cast<double*>(base + 256);
    double* hbuf = part + (size_t)W * nblk * jb;
    double* rbuf = hbuf + (size_t)W * jb;
    double* npart = rbuf + (size_t)W * jb;
    if (int rc = bem_check_cuda(ctx, cudaMemsetAsync(bar, 0, sizeof(GridBar), s), "cgs2 barrier reset")) return rc;
    int32_t* flag = ctx->flags + 7;
    void* args[] = {&Q, &n, &ldq, &j, (void*)&v, &ldv, &Rt, &ldr, &part, &hbuf, &rbuf, &npart, &bar, &flag};
    if (int rc = bem_check_cuda(ctx, cudaLaunchCooperativeKernel((const void*)cgs2_append_kernel<C>, nblk,
                                                                CG_THREADS, args, smem, s),
                                "cgs2_append_kernel"))
        return rc;
    ctx->launches++;
    if (!check) return BEM_OK;
    int32_t f = 0;
    if (int rc = bem_check_cuda(ctx, cudaMemcpyAsync(&f, flag, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                                "cgs2 flag readback"))
        return rc;
    if (int rc = bem_check_cuda(ctx, cudaStreamSynchronize(s), "cgs2_append")) return rc;
    if (f != 0) {
        cudaMemsetAsync(flag, 0, sizeof(int32_t), s);
        return bem_fail(ctx, BEM_ERR_TIMEOUT, "cgs2_append: a grid barrier hit its iteration cap");
    }
    return BEM_OK;
}

template <typename T, bool C>
int gemv_t(bem_ctx* ctx, const T* A, int64_t m, int64_t n, int64_t lda, const double* x, double* y, double alpha,
           double beta, cudaStream_t s) {
    unsigned blocks = (unsigned)((m + 7) / 8);
    gemv_kernel<T, C><<<blocks, 256, 0, s>>>(A, m, n, lda, x, y, alpha, beta, beyond_l2<T, C>(ctx, m, n));
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "gemv_kernel");
}

}  // namespace

extern "C" {

int bem_cgs2_append(bem_ctx* ctx, int dtype, void* Q, int64_t n, int64_t ldq, int j, const void* v, int64_t ldv,
                    void* Rt, int64_t ldr, int check, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!Q || !v || !Rt || n <= 0 || j < 0 || ldq <= j || ldr <= j || ldv <= 0)
        return bem_fail(ctx, BEM_ERR_INVALID, "cgs2_append: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64:
            return cgs2_append_t<false>(ctx, (double*)Q, n, ldq, j, (const double*)v, ldv, (double*)Rt, ldr, check, s);
        case BEM_C128:
            return cgs2_append_t<true>(ctx, (double*)Q, n, ldq, j, (const double*)v, ldv, (double*)Rt, ldr, check, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "cgs2_append: dtype must be BEM_F64 or BEM_C128");
    }
}

int bem_lu_factor(bem_ctx* ctx, int dtype, void* A, int64_t n, int64_t lda, int32_t* piv, int32_t* info,
                  void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A || !piv || !info || n <= 0 || lda < n) return bem_fail(ctx, BEM_ERR_INVALID, "lu_factor: bad arguments");
    if (n > (int64_t)1 << 30) return bem_fail(ctx, BEM_ERR_INVALID, "lu_factor: n too large");
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64: return lu_factor_t<double, false>(ctx, (double*)A, n, lda, piv, info, s);
        case BEM_C128: return lu_factor_t<double, true>(ctx, (double*)A, n, lda, piv, info, s);
        case BEM_F32: return lu_factor_t<float, false>(ctx, (float*)A, n, lda, piv, info, s);
        case BEM_C64: return lu_factor_t<float, true>(ctx, (float*)A, n, lda, piv, info, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_factor: unknown dtype");
    }
}

int bem_lu_solve(bem_ctx* ctx, int dtype, const void* LU, int64_t n, int64_t lda, const int32_t* piv, void* b,
                 int64_t nrhs, int64_t ldb, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!LU || !piv || !b || n <= 0 || lda < n || ldb < nrhs)
        return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    switch (dtype) {
        case BEM_F64: return lu_solve_t<double, false>(ctx, (const double*)LU, n, lda, piv, (double*)b, nrhs, ldb, s);
        case BEM_C128: return lu_solve_t<double, true>(ctx, (const double*)LU, n, lda, piv, (double*)b, nrhs, ldb, s);
        case BEM_F32: return lu_solve_t<float, false>(ctx, (const float*)LU, n, lda, piv, (double*)b, nrhs, ldb, s);
        case BEM_C64: return lu_solve_t<float, true>(ctx, (const float*)LU, n, lda, piv, (double*)b, nrhs, ldb, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "lu_solve: unknown dtype");
    }
}

int bem_gemv(bem_ctx* ctx, int a_dtype, const void* A, int64_t m, int64_t n, int64_t lda, const void* x, void* y,
             double alpha, double beta, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A || !x || !y || m <= 0 || n <= 0 || lda < n) return bem_fail(ctx, BEM_ERR_INVALID, "gemv: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    switch (a_dtype) {
        case BEM_F64: return gemv_t<double, false>(ctx, (const double*)A, m, n, lda, (const double*)x, (double*)y, alpha, beta, s);
        case BEM_C128: return gemv_t<double, true>(ctx, (const double*)A, m, n, lda, (const double*)x, (double*)y, alpha, beta, s);
        case BEM_F32: return gemv_t<float, false>(ctx, (const float*)A, m, n, lda, (const double*)x, (double*)y, alpha, beta, s);
        case BEM_C64: return gemv_t<float, true>(ctx, (const float*)A, m, n, lda, (const double*)x, (double*)y, alpha, beta, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "gemv: unknown dtype");
    }
}

int bem_refine_solve(bem_ctx* ctx, int dtype_hi, const void* A_hi, const void* LU_lo, const int32_t* piv,
                     const void* dinv, int64_t n, int64_t lda, const void* b, void* x, double tol, int maxit,
                     int* iters, double* relres, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A_hi || !LU_lo || !piv || !b || !x || n <= 0 || lda < n || maxit < 1 || !(tol > 0))
        return bem_fail(ctx, BEM_ERR_INVALID, "refine_solve: bad arguments");
    if (dtype_hi != BEM_F64 && dtype_hi != BEM_C128)
        return bem_fail(ctx, BEM_ERR_INVALID, "refine_solve: A_hi must be F64 or C128");
    const bool C = dtype_hi == BEM_C128;
    const int W = C ? 2 : 1;
    const int64_t nd = W * n;
    cudaStream_t s = (cudaStream_t)stream;
    if (dinv) return refine_async(ctx, C, A_hi, LU_lo, piv, dinv, n, lda, (const double*)b, (double*)x, tol, maxit,
                                  iters, relres, s);
    // workspace beyond the lu_solve scratch: r (nd), d (nd), norms (2)
    double* r = nullptr;
    if (int rc = bem_check_cuda(ctx, cudaMallocAsync((void**)&r, sizeof(double) * (2 * nd + 4), s), "refine alloc"))
        return rc;
    double* d = r + nd;
    double* nrm = d + nd;
    const double* bd = (const double*)b;
    double* xd = (double*)x;
    int rc = BEM_OK;
    double bnorm = 0.0, rnorm = 0.0;
    int it = 0;
    auto norm2 = [&](const double* v, double* out_host) -> int {
        cudaMemsetAsync(nrm, 0, sizeof(double), s);
        sumsq_kernel<<<std::min<int64_t>(ctx->num_sms * 4, (nd + 255) / 256), 256, 0, s>>>(v, nd, nrm);
        ctx->launches++;
        if (int e = bem_check_cuda(ctx, cudaMemcpyAsync(out_host, nrm, sizeof(double), cudaMemcpyDeviceToHost, s),
                                   "norm readback"))
            return e;
        if (int e = bem_check_cuda(ctx, cudaStreamSynchronize(s), "norm")) return e;
        *out_host = std::sqrt(*out_host);
        return BEM_OK;
    };
    rc = norm2(bd, &bnorm);
    if (rc == BEM_OK) rc = bem_check_cuda(ctx, cudaMemsetAsync(xd, 0, sizeof(double) * nd, s), "x=0");
    if (rc == BEM_OK) rc = bem_check_cuda(ctx, cudaMemcpyAsync(r, bd, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s), "r=b");
    rnorm = bnorm;
    if (bnorm == 0.0) {
        cudaFreeAsync(r, s);
        if (iters) *iters = 0;
        if (relres) *relres = 0.0;
        return rc;
    }
    while (rc == BEM_OK && it < maxit) {
        // d = LU_lo^{-1} r
        rc = bem_check_cuda(ctx, cudaMemcpyAsync(d, r, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s), "d=r");
        if (rc) break;
        if (dinv)
            rc = bem_lu_solve_tiled(ctx, C ? BEM_C64 : BEM_F32, LU_lo, n, lda, piv, dinv, d, s);
        else
            rc = bem_lu_solve(ctx, C ? BEM_C64 : BEM_F32, LU_lo, n, lda, piv, d, 1, 1, s);
        if (rc) break;
        axpy_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, s>>>(xd, d, nd, 1.0);
        ctx->launches++;
        // r = b - A_hi x
        rc = bem_check_cuda(ctx, cudaMemcpyAsync(r, bd, sizeof(double) * nd, cudaMemcpyDeviceToDevice, s), "r=b");
        if (rc) break;
        rc = bem_gemv(ctx, dtype_hi, A_hi, n, n, lda, xd, r, -1.0, 1.0, s);
        if (rc) break;
        ++it;
        const double prev = rnorm;
        rc = norm2(r, &rnorm);
        if (rc) break;
        if (rnorm <= tol * bnorm) break;
        if (it >= 3 && rnorm > 0.5 * prev) break;  // stagnation: the factor is not a good enough preconditioner
    }
    cudaFreeAsync(r, s);
    if (iters) *iters = it;
    if (relres) *relres = rnorm / bnorm;
    if (rc == BEM_OK && rnorm > tol * bnorm)
        return bem_fail(ctx, BEM_ERR_NOCONVERGE, "refinement did not reach tol in maxit iterations");
    return rc;
}

int bem_gmres_ir(bem_ctx* ctx, int dtype_hi, const void* A_hi, const void* LU_lo, const int32_t* piv,
                 const void* dinv, int64_t n, int64_t lda, const void* b, void* x, double tol, int maxit, int restart,
                 double accept, int* iters, double* relres, void* stream) {
    if (!ctx) return BEM_ERR_INVALID;
    if (!A_hi || !LU_lo || !piv || !b || !x || n <= 0 || lda < n || maxit < 1 || restart < 1 || !(tol > 0))
        return bem_fail(ctx, BEM_ERR_INVALID, "gmres_ir: bad arguments");
    if (dtype_hi != BEM_F64 && dtype_hi != BEM_C128)
        return bem_fail(ctx, BEM_ERR_INVALID, "gmres_ir: A_hi must be F64 or C128");
    return gmres_run(ctx, dtype_hi, A_hi, LU_lo, piv, dinv, n, lda, (const double*)b, (double*)x, tol, maxit,
                     restart, accept, iters, relres, (cudaStream_t)stream);
}

}  // extern "C"
