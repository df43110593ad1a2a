// FP64 separate pairs of one operator (the plain path), each unordered panel
// pair evaluated once.
//
// The reference integrates every ordered pair of every operator on its own
// (single_layer_3d.py:371-433, double_layer_3d.py:376-438,
// hypersingular_layer_3d.py:437-500).  The separate-pair rule puts the same
// points on a panel whichever side it is on, so one evaluation of r, 1/r and
// e^{ikr} at (x in panel i, y in panel j), d = x - y, serves both orders:
//   V, W   the integrand is symmetric: entry (i, j) and entry (j, i);
//   K, K'  sum w phi_b(y) ( d.n_j) F / r^3   (K: row i, hats of j; K': hats of j, column i)
//          sum w phi_a(x) (-d.n_i) F / r^3   (K: row j, hats of i; K': hats of i, column j)
// with F = (1 - ikr) e^{ikr}.  The lists may differ (a Mix partition): a pair
// whose reversed order is in the call too is evaluated by the order with the
// smaller test panel and added for both, any other one for its own (so is every
// further entry of a panel that a list names twice: the maps hold one of them).
//
// Bound: FP64 issue.  What a point pair costs is therefore its count of FP64
// instructions (V Helmholtz: 3 differences, 3 for r^2, 6 for r and 1/r, the
// phase, 13 for sine and cosine, 3 to accumulate), and everything that does
// not depend on both points is taken out: e^{ikr} = e^{ikR} e^{ik(r - R)} with
// R the centroid distance leaves a phase of a few panel diameters, which the
// host bounds (PH) so that no argument reduction runs; d.n_j = D.n_j + x.n_j
// and d.n_i = D.n_i - y.n_i (offsets lie in their panel's plane).  FP64
// throughout, as the general kernel.
// Measured (B200, this kernel against the general one per ordered pair with
// the library's rsqrt and sincos): V Helmholtz, 5120 panels, GaussQR 5: 16.9
// against 58.4 ms (FP64 pipe 78 % busy, 29 FP64 instructions a point pair);
// K Laplace product, 2970 panels: 5.0 against 7.9 ms; V and K of 1280 panels:
// 0.63 and 0.97 against 1.19 and 1.57 ms.
#include <algorithm>
#include <cmath>

#include "bem_farfield.cuh"

namespace {

struct Far64Args {
    int n_test, n_trial;
    const int32_t* test_panels;
    const int32_t* test_dof;
    const int32_t* trial_panels;
    const int32_t* trial_dof;
    const int32_t* test_local;   // [nt] index of a global panel in the test list, -1 = absent
    const int32_t* trial_local;  // [nt]
    const int32_t* tris;
    const double* centroid;
    const double* normal;
    const double* curl;
    const double4* pts;   // offset from the centroid, weight with 2A
    const double* phi64;  // [Q2*3]
    int Q2, ti;           // points per panel, test panels per CTA
    int op;
    double k, k2;
    int mode;
    double* out;
    int64_t ld;
    double scale;
    double* out_t;
    double scale_t;
    const double* x;
    double* y;
    int conj_x;
};

struct Cx {
    double re, im;
};

// (total, phi_1, phi_2) moments -> the three hats
__device__ __forceinline__ void hats3(const double* m, double* v) {
    v[0] = m[0] - m[1] - m[2];
    v[1] = m[1];
    v[2] = m[2];
}

template <bool HELM>
__device__ __forceinline__ Cx load_x(const Far64Args& a, int col) {
    if (col < 0) return Cx{0.0, 0.0};
    if (!HELM) return Cx{a.x[col], 0.0};
    return Cx{a.x[2 * (int64_t)col], a.conj_x ? -a.x[2 * (int64_t)col + 1] : a.x[2 * (int64_t)col + 1]};
}

template <bool HELM>
__device__ __forceinline__ void cfma(Cx& acc, double vr, double vi, const Cx& x) {
    acc.re += vr * x.re;
    if (HELM) {
        acc.re -= vi * x.im;
        acc.im += vr * x.im + vi * x.re;
    }
}

template <bool HELM>
__device__ __forceinline__ void add_y(const Far64Args& a, int row, const Cx& c) {
    if (row < 0) return;
    if (HELM) {
        atomicAdd(a.y + 2 * (int64_t)row, a.scale * c.re);
        atomicAdd(a.y + 2 * (int64_t)row + 1, a.scale * c.im);
    } else {
        atomicAdd(a.y + row, a.scale * c.re);
    }
}

template <bool HELM>
__device__ __forceinline__ void put(const Far64Args& a, int row, int col, double re, double im, bool atomic) {
    if (row < 0 || col < 0) return;
    add_entry<HELM>(a.out, (int64_t)row * a.ld + col, a.scale * re, a.scale * im, atomic);
    if (a.out_t) add_entry<HELM>(a.out_t, (int64_t)col * a.ld + row, a.scale_t * re, a.scale_t * im, true);
}

// SYM: V and W (KIND 0: V, 1: W), NB bases per panel on both sides; otherwise
// (KIND 2) K and K', NB bases on the P1 (or P0 data) side and one on the other.
template <int KIND, bool HELM, int NB, int PH>
__global__ void __launch_bounds__(FAR_THREADS) far64_kernel(Far64Args a) {
    constexpr bool SYM = KIND != 2;
    // phi-weighted moments of a symmetric operator: every one with P1 bases but Laplace W (no mass term)
    constexpr bool PHI = NB == 3 && !(KIND == 1 && !HELM);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double4* sx = reinterpret_cast<double4*>(smem_raw);           // [ti][Q2]
    double2* sp = reinterpret_cast<double2*>(sx + a.ti * a.Q2);  // [Q2] phi_1, phi_2
    __shared__ int s_gi[FAR_TI];
    __shared__ int s_ri[FAR_TI];  // index of the test panel in the trial list, -1 = absent
    __shared__ int s_tri[FAR_TI][3];
    __shared__ double s_cen[FAR_TI][3];
    __shared__ double s_nrm[FAR_TI][3];

    const int Q2 = a.Q2;
    const int lj = blockIdx.x * FAR_THREADS + threadIdx.x;
    const int li0 = blockIdx.y * a.ti;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < a.ti) {
        const int li = li0 + threadIdx.x;
        const int gi = li < a.n_test ? a.test_panels[li] : -1;
        s_gi[threadIdx.x] = gi;
        s_ri[threadIdx.x] = gi >= 0 && a.test_local[gi] == li ? a.trial_local[gi] : -1;
        for (int c = 0; c < 3; ++c) {
            s_tri[threadIdx.x][c] = gi >= 0 ? a.tris[3 * gi + c] : -1;
            s_cen[threadIdx.x][c] = gi >= 0 ? a.centroid[3 * gi + c] : 0.0;
            s_nrm[threadIdx.x][c] = gi >= 0 ? a.normal[3 * gi + c] : 0.0;
        }
    }
    for (int q = threadIdx.x; q < Q2; q += FAR_THREADS) sp[q] = make_double2(a.phi64[3 * q + 1], a.phi64[3 * q + 2]);
    __syncthreads();
    for (int idx = threadIdx.x; idx < a.ti * Q2; idx += FAR_THREADS) {
        const int t = idx / Q2, q = idx - t * Q2;
        if (s_gi[t] >= 0) sx[idx] = a.pts[(size_t)s_gi[t] * Q2 + q];
    }
    __syncthreads();

    const bool valid_j = lj < a.n_trial;
    const int gj = valid_j ? a.trial_panels[lj] : 0;
    const int rj = valid_j && a.trial_local[gj] == lj ? a.test_local[gj] : -1;  // index of the trial panel in the test list
    int tri_j[3];
    double cj[3], nj[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        tri_j[c] = a.tris[3 * gj + c];
        cj[c] = a.centroid[3 * gj + c];
        nj[c] = a.normal[3 * gj + c];
    }
    const double4* ptsj = a.pts + (size_t)gj * Q2;
    const double k = a.k;
    const bool kp = a.op == BEM_OP_KP;
    constexpr int NJ = SYM ? NB : 3;
    Cx rowj[NJ];  // apply: this thread's sum for the rows of test panel gj
#pragma unroll
    for (int b = 0; b < NJ; ++b) rowj[b] = Cx{0.0, 0.0};

    for (int t = 0; t < a.ti; ++t) {
        const int gi = s_gi[t];
        if (gi < 0) break;  // uniform across the CTA
        const int li = li0 + t, ri = s_ri[t];
        const bool both = ri >= 0 && rj >= 0;
        const bool live = valid_j && !(both && gi > gj) && bem_relation(s_tri[t], tri_j, gi == gj) == REL_SEPARATE;
        Cx rowi[NJ];  // apply: this pair's contribution to the rows of test panel gi
#pragma unroll
        for (int b = 0; b < NJ; ++b) rowi[b] = Cx{0.0, 0.0};
        if (live) {
            const double D0 = s_cen[t][0] - cj[0], D1 = s_cen[t][1] - cj[1], D2 = s_cen[t][2] - cj[2];
            double phR = 0.0;  // k R, rounded once: the phase is taken relative to this very value
            if (HELM) phR = k * sqrt(D0 * D0 + D1 * D1 + D2 * D2);
            const double Dnj = D0 * nj[0] + D1 * nj[1] + D2 * nj[2];
            const double Dni = D0 * s_nrm[t][0] + D1 * s_nrm[t][1] + D2 * s_nrm[t][2];
            const double4* sxt = sx + t * Q2;
            // SYM: [0] total, then (x, y) hats (0,1) (0,2) (1,0) (1,1) (1,2) (2,0) (2,1) (2,2) with 0 = total;
            // K: [0..2] (d.n_j) with the hats of y, [3..5] (-d.n_i) with those of x
            constexpr int NM = SYM ? (PHI ? 9 : 1) : 6;
            double Mr[NM], Mi[NM];
#pragma unroll
            for (int m = 0; m < NM; ++m) Mr[m] = Mi[m] = 0.0;
            for (int b = 0; b < Q2; ++b) {
                const double4 yb = ptsj[b];
                const double e0 = D0 - yb.x, e1 = D1 - yb.y, e2 = D2 - yb.z;
                constexpr int NS = SYM ? (PHI ? 3 : 1) : (NB == 3 ? 4 : 2);
                double sr[NS], si[NS];
#pragma unroll
                for (int m = 0; m < NS; ++m) sr[m] = si[m] = 0.0;
#pragma unroll 5
                for (int q = 0; q < Q2; ++q) {
                    const double4 xa = sxt[q];
                    const double dx = xa.x + e0, dy = xa.y + e1, dz = xa.z + e2;
                    double r, rinv;
                    dev_r_rinv(fma(dx, dx, fma(dy, dy, dz * dz)), r, rinv);
                    double cs = 1.0, sn = 0.0;
                    if (HELM) dev_sincos_ph<PH>(fma(k, r, -phR), &sn, &cs);
                    const double wr = xa.w * rinv;
                    double2 ph = make_double2(0.0, 0.0);
                    if (NB == 3) ph = sp[q];
                    if constexpr (SYM) {
                        if constexpr (!HELM) {
                            sr[0] += wr;
                            if constexpr (PHI) {
                                sr[1] = fma(ph.x, wr, sr[1]);
                                sr[2] = fma(ph.y, wr, sr[2]);
                            }
                        } else if constexpr (!PHI) {
                            sr[0] = fma(wr, cs, sr[0]);
                            si[0] = fma(wr, sn, si[0]);
                        } else {
                            const double gr = wr * cs, gi_ = wr * sn;
                            sr[0] += gr;
                            si[0] += gi_;
                            sr[1] = fma(ph.x, gr, sr[1]);
                            si[1] = fma(ph.x, gi_, si[1]);
                            sr[2] = fma(ph.y, gr, sr[2]);
                            si[2] = fma(ph.y, gi_, si[2]);
                        }
                    } else {
                        const double wr3 = wr * (rinv * rinv);
                        const double dnj = fma(xa.x, nj[0], fma(xa.y, nj[1], fma(xa.z, nj[2], Dnj)));
                        double hr = wr3, hi = 0.0;
                        if (HELM) {
                            const double kr = k * r;
                            hr = wr3 * fma(kr, sn, cs);
                            hi = wr3 * fma(-kr, cs, sn);
                        }
                        sr[0] = fma(dnj, hr, sr[0]);
                        sr[1] += hr;
                        if constexpr (NB == 3) {
                            sr[2] = fma(ph.x, hr, sr[2]);
                            sr[3] = fma(ph.y, hr, sr[3]);
                        }
                        if (HELM) {
                            si[0] = fma(dnj, hi, si[0]);
                            si[1] += hi;
                            if constexpr (NB == 3) {
                                si[2] = fma(ph.x, hi, si[2]);
                                si[3] = fma(ph.y, hi, si[3]);
                            }
                        }
                    }
                }
                const double wb = yb.w;
                double wb1 = 0.0, wb2 = 0.0;
                if (NB == 3) {
                    const double2 ph = sp[b];
                    wb1 = wb * ph.x;
                    wb2 = wb * ph.y;
                }
                auto acc = [&](int m, double w, int src) {
                    Mr[m] = fma(w, sr[src], Mr[m]);
                    if (HELM) Mi[m] = fma(w, si[src], Mi[m]);
                };
                if constexpr (SYM) {
                    acc(0, wb, 0);
                    if constexpr (PHI) {
                        acc(1, wb1, 0);
                        acc(2, wb2, 0);
                        acc(3, wb, 1);
                        acc(4, wb1, 1);
                        acc(5, wb2, 1);
                        acc(6, wb, 2);
                        acc(7, wb1, 2);
                        acc(8, wb2, 2);
                    }
                } else {
                    // -d.n_i, constant over the points of panel i
                    const double ndni = fma(yb.x, s_nrm[t][0], fma(yb.y, s_nrm[t][1], fma(yb.z, s_nrm[t][2], -Dni)));
                    acc(0, wb, 0);
                    acc(3, wb * ndni, 1);
                    if constexpr (NB == 3) {
                        acc(1, wb1, 0);
                        acc(2, wb2, 0);
                        acc(4, wb * ndni, 2);
                        acc(5, wb * ndni, 3);
                    }
                }
            }
            // e^{ikR} / (4 pi)
            double fr = BEM_INV4PI, fi = 0.0;
            if (HELM) {
                double sR, cR;
                dev_sincos_frame(phR, &sR, &cR);
                fi = fr * sR;
                fr = fr * cR;
            }
            auto times_f = [&](double& re, double& im) {
                const double u = re, v = im;
                re = HELM ? u * fr - v * fi : u * fr;
                im = HELM ? u * fi + v * fr : 0.0;
            };
            // W: after the curl product (below), as the general kernel does
            if (KIND != 1)
#pragma unroll
                for (int m = 0; m < NM; ++m) times_f(Mr[m], Mi[m]);
            if constexpr (SYM) {
                double vr[NB][NB], vi[NB][NB];
                if constexpr (NB == 1) {
                    vr[0][0] = Mr[0];
                    vi[0][0] = Mi[0];
                } else {
                    if constexpr (PHI) {
                        // hats of y per x moment, then hats of x
                        double hr[3][3], hi[3][3];
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            hats3(Mr + 3 * x, hr[x]);
                            hats3(Mi + 3 * x, hi[x]);
                        }
#pragma unroll
                        for (int y = 0; y < 3; ++y) {
                            vr[0][y] = hr[0][y] - hr[1][y] - hr[2][y];
                            vi[0][y] = hi[0][y] - hi[1][y] - hi[2][y];
                            vr[1][y] = hr[1][y];
                            vi[1][y] = hi[1][y];
                            vr[2][y] = hr[2][y];
                            vi[2][y] = hi[2][y];
                        }
                    }
                    if constexpr (KIND == 1) {
                        // G curl.curl - k2 (n_x.n_y) G phi_x phi_y (hypersingular_layer_3d.py:206-211)
                        const double k2n =
                            a.k2 * (s_nrm[t][0] * nj[0] + s_nrm[t][1] * nj[1] + s_nrm[t][2] * nj[2]);
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            const double* cx = a.curl + 9 * gi + 3 * x;
#pragma unroll
                            for (int y = 0; y < 3; ++y) {
                                const double* cy = a.curl + 9 * gj + 3 * y;
                                const double cd = cx[0] * cy[0] + cx[1] * cy[1] + cx[2] * cy[2];
                                vr[x][y] = PHI ? Mr[0] * cd - k2n * vr[x][y] : Mr[0] * cd;
                                vi[x][y] = PHI ? Mi[0] * cd - k2n * vi[x][y] : Mi[0] * cd;
                                times_f(vr[x][y], vi[x][y]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int x = 0; x < NB; ++x)
#pragma unroll
                    for (int y = 0; y < NB; ++y) {
                        if (a.mode == 0) {
                            put<HELM>(a, a.test_dof[li * NB + x], a.trial_dof[lj * NB + y], vr[x][y], vi[x][y],
                                      NB == 3);
                            if (both)
                                put<HELM>(a, a.test_dof[rj * NB + y], a.trial_dof[ri * NB + x], vr[x][y], vi[x][y],
                                          NB == 3);
                        } else {
                            cfma<HELM>(rowi[x], vr[x][y], vi[x][y], load_x<HELM>(a, a.trial_dof[lj * NB + y]));
                            if (both)
                                cfma<HELM>(rowj[y], vr[x][y], vi[x][y], load_x<HELM>(a, a.trial_dof[ri * NB + x]));
                        }
                    }
            } else {
                double ar[3], ai[3], br[3], bi[3];  // hats of y with d.n_j; hats of x with -d.n_i
                if constexpr (NB == 3) {
                    hats3(Mr, ar);
                    hats3(Mi, ai);
                    hats3(Mr + 3, br);
                    hats3(Mi + 3, bi);
                } else {
                    ar[0] = Mr[0];
                    ai[0] = Mi[0];
                    br[0] = Mr[3];
                    bi[0] = Mi[3];
                }
#pragma unroll
                for (int h = 0; h < NB; ++h) {
                    if (a.mode == 0) {
                        if (!kp) {
                            put<HELM>(a, a.test_dof[li], a.trial_dof[lj * NB + h], ar[h], ai[h], NB == 3);
                            if (both) put<HELM>(a, a.test_dof[rj], a.trial_dof[ri * NB + h], br[h], bi[h], NB == 3);
                        } else {
                            put<HELM>(a, a.test_dof[li * NB + h], a.trial_dof[lj], br[h], bi[h], NB == 3);
                            if (both) put<HELM>(a, a.test_dof[rj * NB + h], a.trial_dof[ri], ar[h], ai[h], NB == 3);
                        }
                    } else if (!kp) {
                        cfma<HELM>(rowi[0], ar[h], ai[h], load_x<HELM>(a, a.trial_dof[lj * NB + h]));
                        if (both) cfma<HELM>(rowj[0], br[h], bi[h], load_x<HELM>(a, a.trial_dof[ri * NB + h]));
                    } else {
                        cfma<HELM>(rowi[h], br[h], bi[h], load_x<HELM>(a, a.trial_dof[lj]));
                        if (both) cfma<HELM>(rowj[h], ar[h], ai[h], load_x<HELM>(a, a.trial_dof[ri]));
                    }
                }
            }
        }
        if (a.mode != 0) {
            const int rows = SYM ? NB : (kp ? NB : 1);
#pragma unroll
            for (int b = 0; b < NJ; ++b) {
                if (b >= rows) break;
                Cx c = rowi[b];
                c.re = warp_sum(c.re);
                if (HELM) c.im = warp_sum(c.im);
                if (lane == 0) add_y<HELM>(a, a.test_dof[li * rows + b], c);
            }
        }
    }
    if (a.mode != 0 && rj >= 0) {
        const int rows = SYM ? NB : (kp ? NB : 1);
#pragma unroll
        for (int b = 0; b < NJ; ++b)
            if (b < rows && (rowj[b].re != 0.0 || rowj[b].im != 0.0)) add_y<HELM>(a, a.test_dof[rj * rows + b], rowj[b]);
    }
}

template <int KIND, bool HELM, int NB, int PH>
int launch_far64(bem_ctx* ctx, const Far64Args& a, cudaStream_t s) {
    const dim3 grid((a.n_trial + FAR_THREADS - 1) / FAR_THREADS, (a.n_test + a.ti - 1) / a.ti);
    if (grid.y > 65535) return bem_fail(ctx, BEM_ERR_INVALID, "too many test panels for one launch");
    const size_t smem = (size_t)a.ti * a.Q2 * sizeof(double4) + a.Q2 * sizeof(double2);
    far64_kernel<KIND, HELM, NB, PH><<<grid, FAR_THREADS, smem, s>>>(a);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "far64_kernel launch");
}

template <int KIND, int NB>
int dispatch_far64(bem_ctx* ctx, const Far64Args& a, bool helm, int ph, cudaStream_t s) {
    if (!helm) return launch_far64<KIND, false, NB, 0>(ctx, a, s);
    if (ph == 2) return launch_far64<KIND, true, NB, 2>(ctx, a, s);
    if (ph == 1) return launch_far64<KIND, true, NB, 1>(ctx, a, s);
    return launch_far64<KIND, true, NB, 0>(ctx, a, s);
}

}  // namespace

// The far pairs of an FP64 call whose bases the kernel above has (the spaces
// of the boundary-value problems: V P0 x P0 and P1 x P1, W P1 x P1, K with P0
// rows, K' with P0 columns); returns 1 for the others and for k-derivatives,
// which the general far_kernel takes.  The local maps of both lists have to be
// filled (bem_fill_local_map).
int bem_launch_far64(bem_ctx* ctx, const bem_op_desc* op, const bem_space* test, const bem_space* trial, int mode,
                     void* out, int64_t ld, double scale, void* out_t, double scale_t, const void* x, void* y,
                     int conj_x, cudaStream_t s) {
    if (op->precision != BEM_PREC_FP64 || op->deriv_k) return 1;
    // one point a panel (GaussQR 1): what is left is the writing of both orders, which
    // costs more than the second evaluation.  One order against both, k = 2: K block of
    // 1280 panels 81 against 103 us, V block of 5120 panels 578 against 685 us, K'
    // product of 320 panels 42 against 89 us.
    if (ctx->Q2 == 1) return 1;
    const int nx = test->nb, ny = trial->nb;
    const bool v1 = op->op == BEM_OP_V && nx == 1 && ny == 1, v3 = op->op == BEM_OP_V && nx == 3 && ny == 3;
    const bool w3 = op->op == BEM_OP_W && nx == 3 && ny == 3;
    const bool k = (op->op == BEM_OP_K && nx == 1) || (op->op == BEM_OP_KP && ny == 1);
    if (!v1 && !v3 && !w3 && !k) return 1;
    if (test->n_panels <= 0 || trial->n_panels <= 0) return BEM_OK;
    Far64Args a{};
    a.n_test = test->n_panels;
    a.n_trial = trial->n_panels;
    a.test_panels = test->panels;
    a.test_dof = test->dof;
    a.trial_panels = trial->panels;
    a.trial_dof = trial->dof;
    a.test_local = ctx->test_local;
    a.trial_local = ctx->trial_local;
    a.tris = ctx->tris;
    a.centroid = ctx->centroid;
    a.normal = ctx->normal;
    a.curl = ctx->curl;
    a.pts = ctx->pts64;
    a.phi64 = ctx->phi64;
    a.Q2 = ctx->Q2;
    a.op = op->op;
    a.k = op->k;
    a.k2 = op->k2;
    a.mode = mode;
    a.out = (double*)out;
    a.ld = ld;
    a.scale = scale;
    a.out_t = (double*)out_t;
    a.scale_t = scale_t;
    a.x = (const double*)x;
    a.y = (double*)y;
    a.conj_x = conj_x;
    // test panels per CTA: eight share one read of the trial panel's data where
    // the call has CTAs for several waves; a small mesh is spread over the SMs
    // instead (80 panels, Helmholtz: V 22 and K 24 us, 133 and 159 us with eight)
    a.ti = FAR_TI;
    const int64_t cols = (a.n_trial + FAR_THREADS - 1) / FAR_THREADS;
    while (a.ti > 1 && cols * ((a.n_test + a.ti - 1) / a.ti) < 16 * (int64_t)ctx->num_sms) a.ti /= 2;
    // |k (r - R)| <= |k| (rho_i + rho_j)
    const bool helm = op->kernel == BEM_KERNEL_HELMHOLTZ;
    const int ph = helm ? bem_phase_class(std::fabs(op->k) * 2.0 * ctx->rho_max) : 0;
    if (v1) return dispatch_far64<0, 1>(ctx, a, helm, ph, s);
    if (v3) return dispatch_far64<0, 3>(ctx, a, helm, ph, s);
    if (w3) return dispatch_far64<1, 3>(ctx, a, helm, ph, s);
    return (op->op == BEM_OP_K ? ny : nx) == 1 ? dispatch_far64<2, 1>(ctx, a, helm, ph, s)
                                               : dispatch_far64<2, 3>(ctx, a, helm, ph, s);
}
