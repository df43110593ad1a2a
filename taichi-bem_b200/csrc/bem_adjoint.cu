// Shape derivatives of Galerkin BEM bilinear forms (the adjoint of the
// assembly): for the Laplace single layer V (P0 x P0) and double layer K
// (P0 test x P1 trial)
//
//   grad[v] += d/dX_v  sum_{rows r, cols c} lam[r] A[r, c] u[c]
//
// with X the vertex positions.  Nothing is stored between the forward solve
// and this pass: every quadrature point of every pair is recomputed, with the
// same rules as the assembly (separate pairs: the GaussQR^2 x GaussQR^2 tensor
// rule; coincident / edge / vertex pairs: the Sauter-Schwab points of
// bem_quadrature.cuh).  Per point x = sum_a beta_a(xi) P_a on panel i,
// y = sum_b beta_b(eta) Q_b on panel j, weight w = w_xi w_eta J_i J_j
// (J = 2 x area), the integrand's dependence on the vertices is
//   * through d = x - y:   d/dP_a = beta_a(xi) d/dd,   d/dQ_b = -beta_b(eta) d/dd;
//   * through J_i (and J_j for V):  dJ/dP_a = n x (P_{a+2} - P_{a+1});
//   * for K through N_j = J_j n_j = (Q_1 - Q_0) x (Q_2 - Q_1), linear in each
//     trial vertex.
// The near-field integrands keep the singularity order of the assembled ones
// (d/dd G ~ 1/r^2 multiplies beta_a(xi) - beta_a(eta) ~ r at a shared
// vertex), so the same quadrature integrates them.  All in FP64.
#include <cuda_runtime.h>

#include "bem_farfield.cuh"
#include "bem_internal.cuh"
#include "bem_quadrature.cuh"

namespace {

constexpr int ADJ_THREADS = 128;
constexpr int ADJ_TI = 8;

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// d(2A)/dP_a for the vertices v[3][3] in the panel's stored order, unit normal n
__device__ __forceinline__ void jac_grad(const double v[3][3], const double n[3], int a, double g[3]) {
    const double* p2 = v[(a + 2) % 3];
    const double* p1 = v[(a + 1) % 3];
    const double e[3] = {p2[0] - p1[0], p2[1] - p1[1], p2[2] - p1[2]};
    g[0] = n[1] * e[2] - n[2] * e[1];
    g[1] = n[2] * e[0] - n[0] * e[2];
    g[2] = n[0] * e[1] - n[1] * e[0];
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// d(w . N)/dQ_b with N = (Q1 - Q0) x (Q2 - Q1): Q0: w x (Q2 - Q1), Q1: (Q2 - Q0) x w, Q2: w x (Q1 - Q0)
__device__ __forceinline__ void normal_grad(const double q[3][3], const double w[3], int b, double g[3]) {
    double e[3];
    if (b == 0) {
        for (int c = 0; c < 3; ++c) e[c] = q[2][c] - q[1][c];
        cross3(w, e, g);
    } else if (b == 1) {
        for (int c = 0; c < 3; ++c) e[c] = q[2][c] - q[0][c];
        cross3(e, w, g);
    } else {
        for (int c = 0; c < 3; ++c) e[c] = q[1][c] - q[0][c];
        cross3(w, e, g);
    }
}

// Per-pair moments.  For V: k = 1/(4 pi r); for K: k = (d_e . n_j)/(4 pi r^3)
// times the trial density u(eta), d_e = sgn d.
struct PairMoments {
    double S0;        // sum w k
    double SX[3][3];  // sum w beta_a(xi) dk/dd        (test vertex a)
    double SY[3][3];  // sum w beta_b(eta) dk/dd       (trial vertex b, enters with -)
    double SU[3];     // K: sum w (d_e . n_j)/(4 pi r^3) hat_b, the entries K(i, b)
    double SN[3];     // K: sum (w / J_j) u d_e / (4 pi r^3)   (derivative with respect to N_j)
    __device__ __forceinline__ void zero() {
        S0 = 0.0;
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 3; ++c) SX[a][c] = SY[a][c] = 0.0;
        SN[0] = SN[1] = SN[2] = 0.0;
        SU[0] = SU[1] = SU[2] = 0.0;
    }
    __device__ __forceinline__ void reduce() {
        S0 = warp_sum_d(S0);
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 3; ++c) {
                SX[a][c] = warp_sum_d(SX[a][c]);
                SY[a][c] = warp_sum_d(SY[a][c]);
            }
        for (int c = 0; c < 3; ++c) {
            SN[c] = warp_sum_d(SN[c]);
            SU[c] = warp_sum_d(SU[c]);
        }
    }
};

// one point: d = x - y, weight w (with J_i J_j), barycentric weights bx, by,
// trial hats hy and density uy (K; hy . data), argument sign sgn (the swapped coincide term of K),
// 1/J_j (K)
template <int OP>
__device__ __forceinline__ void adj_point(PairMoments& M, const double d[3], double w, const double bx[3],
                                          const double by[3], const double hy[3], double uy, double sgn, const double nj[3],
                                          double invJj) {
    const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    double r, rinv;
    dev_r_rinv(r2, r, rinv);
    const double rinv2 = rinv * rinv;
    double g[3];
    if (OP == BEM_OP_V) {
        const double G = BEM_INV4PI * rinv;
        M.S0 += w * G;
        const double f = -G * rinv2;  // dG/dd = -d / (4 pi r^3)
        for (int c = 0; c < 3; ++c) g[c] = w * f * d[c];
    } else {
        const double de[3] = {sgn * d[0], sgn * d[1], sgn * d[2]};
        const double dn = de[0] * nj[0] + de[1] * nj[1] + de[2] * nj[2];
        const double g3 = BEM_INV4PI * rinv * rinv2;  // 1/(4 pi r^3)
        const double wu = w * uy;
        M.S0 += wu * dn * g3;
        for (int b = 0; b < 3; ++b) M.SU[b] += w * dn * g3 * hy[b];
        // d/dd [(d_e . n) g3(r)] = sgn [n g3 - 3 (d_e . n) d_e / (4 pi r^5)]
        for (int c = 0; c < 3; ++c) g[c] = sgn * wu * (nj[c] * g3 - 3.0 * dn * de[c] * g3 * rinv2);
        for (int c = 0; c < 3; ++c) M.SN[c] += wu * invJj * de[c] * g3;
    }
    for (int a = 0; a < 3; ++a)
        for (int c = 0; c < 3; ++c) {
            M.SX[a][c] += bx[a] * g[c];
            M.SY[a][c] += by[a] * g[c];
        }
}

struct AdjArgs {
    int n_test, n_trial;
    const int32_t* test_panels;
    const int32_t* test_dof;
    const int32_t* trial_panels;
    const int32_t* trial_dof;
    int nby;  // 1 (V) or 3 (K)
    const int32_t* tris;
    const double* verts;
    const double* centroid;
    const double* normal;
    const double* area;
    const double4* pts;   // FP64 separate-rule points (offset, weight with 2A)
    const double* phi64;  // [Q2*3] barycentric weights of the separate-rule points
    int Q2, ti;           // points per panel, test panels per CTA (separate pairs)
    int64_t n_near;
    const int4* near;
    const int32_t* test_local;
    const int32_t* trial_local;
    const double* gp;
    const double* gw;
    int Q;
    int quirk;
    const double* lam;
    const double* u;
    double* grad;
    double* data;  // K, optional: data[c] += sum_r lam[r] K(r, c)
};

__device__ __forceinline__ void load_tri(const AdjArgs& a, int g, double v[3][3], double n[3]) {
    for (int b = 0; b < 3; ++b)
        for (int c = 0; c < 3; ++c) v[b][c] = a.verts[3 * a.tris[3 * g + b] + c];
    for (int c = 0; c < 3; ++c) n[c] = a.normal[3 * g + c];
}

// contributions of one pair's moments (scaled by cw) to its six vertices:
// test vertex a: cw [(dJ_i/dP_a)/J_i S0 + SX[a]]
// trial vertex b: V: cw [(dJ_j/dQ_b)/J_j S0 - SY[b]];  K: cw [-SY[b] + d(SN . N_j)/dQ_b]
template <int OP>
__device__ __forceinline__ void pair_grads(const PairMoments& M, double cw, const double vi[3][3], const double ni[3],
                                           double Ji, const double vj[3][3], const double nj[3], double Jj,
                                           double gx[3][3], double gy[3][3]) {
    for (int a = 0; a < 3; ++a) {
        double jg[3];
        jac_grad(vi, ni, a, jg);
        for (int c = 0; c < 3; ++c) gx[a][c] = cw * (jg[c] / Ji * M.S0 + M.SX[a][c]);
    }
    for (int b = 0; b < 3; ++b) {
        double t[3];
        if (OP == BEM_OP_V) {
            jac_grad(vj, nj, b, t);
            for (int c = 0; c < 3; ++c) gy[b][c] = cw * (t[c] / Jj * M.S0 - M.SY[b][c]);
        } else {
            normal_grad(vj, M.SN, b, t);
            for (int c = 0; c < 3; ++c) gy[b][c] = cw * (t[c] - M.SY[b][c]);
        }
    }
}

// ---- separate pairs: CTA = a.ti test panels (shared memory) x ADJ_THREADS trial panels ----
//
// As in the FP64 assembly, both orders of a pair come from one evaluation (the
// order with the smaller test panel does it when the reversed one is in the
// call too).  With t = w/r^3, the trial density u_j(y) and lam_i of the pair,
// and u_i(x), lam_j of the reversed one,
//   V   cw = lam_i u_j + lam_j u_i,   d/dd = -cw t d;
//   K   A = lam_i u_j(y), B = lam_j u_i(x):
//       d/dd = t (A n_j - B n_i) - 3 t/r^2 (A d.n_j - B d.n_i) d,
// and K's J_i, J_j, N_i and N_j parts.  The sums over the test points carry
// (total, phi_1, phi_2) moments of t, of B t and of the vector along d; hats of
// the trial side, n_j, n_i and lam_i u_j(y) are constant over them and enter
// once per trial point.  Bound: FP64 issue, 27 (V) and 50 (K) instructions a
// point pair for both orders, two thirds of the FP64 pipe at 168 and 252
// registers (capping K at 168 measured the same).  5120 panels, GaussQR 4
// (B200), whole calls: V 8.3 and K 14.8 ms, against 22.6 and 36.4 ms per ordered
// pair with the hats of both sides applied at every point.
//
// DATA (K): the product K^T lam, the derivative in the nodal data, from the
// same points.  d.n_i is constant over the test points and sum_q t d.n_j is
// there already, so it costs nothing per point pair and six multiply-adds a
// trial point: 1 ms at 5120 panels, GaussQR 4, in place of a dense FP64 block
// and its product (7.4 ms).
template <int OP, bool DATA>
__global__ void __launch_bounds__(ADJ_THREADS) adj_far_kernel(AdjArgs a) {
    constexpr bool K = OP == BEM_OP_K;
    static_assert(K || !DATA, "the data derivative is the double layer's");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double4* sx = reinterpret_cast<double4*>(smem_raw);             // [ti][Q2]
    double2* sp = reinterpret_cast<double2*>(sx + a.ti * a.Q2);    // [Q2] phi_1, phi_2
    double* su = reinterpret_cast<double*>(sp + a.Q2);             // K: [ti][Q2] u_i at the test points
    __shared__ int s_gi[ADJ_TI];
    __shared__ int s_ri[ADJ_TI];  // index of the test panel in the trial list, -1 = absent
    __shared__ int s_tri[ADJ_TI][3];
    __shared__ double s_lam[ADJ_TI];
    __shared__ double s_u[ADJ_TI][3];  // trial data of the test panel (the reversed pair's density)
    const int Q2 = a.Q2;
    const int lj = blockIdx.x * ADJ_THREADS + threadIdx.x;
    const int li0 = blockIdx.y * a.ti;
    const int lane = threadIdx.x & 31;
    // trial coefficient (V, P0 data: the same at every vertex) or nodal data of trial-list entry l
    auto trial_data = [&](int l, double u[3]) {
        u[0] = u[1] = u[2] = 0.0;
        if (l < 0) return;
        for (int b = 0; b < a.nby; ++b) {
            const int col = a.trial_dof[l * a.nby + b];
            u[b] = col >= 0 ? a.u[col] : 0.0;
        }
    };
    for (int q = threadIdx.x; q < Q2; q += ADJ_THREADS) sp[q] = make_double2(a.phi64[3 * q + 1], a.phi64[3 * q + 2]);
    if (threadIdx.x < a.ti) {
        const int t = threadIdx.x, li = li0 + t;
        const int gi = li < a.n_test ? a.test_panels[li] : -1;
        s_gi[t] = gi;
        s_ri[t] = gi >= 0 && a.test_local[gi] == li ? a.trial_local[gi] : -1;
        const int row = li < a.n_test ? a.test_dof[li] : -1;
        s_lam[t] = row >= 0 ? a.lam[row] : 0.0;
        double u[3];
        trial_data(s_ri[t], u);
        for (int c = 0; c < 3; ++c) {
            s_u[t][c] = u[c];
            s_tri[t][c] = gi >= 0 ? a.tris[3 * gi + c] : -1;
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < a.ti * Q2; idx += ADJ_THREADS) {
        const int t = idx / Q2, q = idx - t * Q2;
        if (s_gi[t] < 0) continue;
        sx[idx] = a.pts[(size_t)s_gi[t] * Q2 + q];
        // the hats in the order of the general rule: beta . u
        if (K) {
            const double p1 = sp[q].x, p2 = sp[q].y;
            su[idx] = (1.0 - p1 - p2) * s_u[t][0] + p1 * s_u[t][1] + p2 * s_u[t][2];
        }
    }
    __syncthreads();

    const bool valid_j = lj < a.n_trial;
    const int gj = valid_j ? a.trial_panels[lj] : 0;
    // index of the trial panel in the test list; -1 also for a list's further entries of one panel
    const int rj = valid_j && a.trial_local[gj] == lj ? a.test_local[gj] : -1;
    int tri_j[3];
    for (int c = 0; c < 3; ++c) tri_j[c] = a.tris[3 * gj + c];
    const double nj[3] = {a.normal[3 * gj], a.normal[3 * gj + 1], a.normal[3 * gj + 2]};
    const double cj[3] = {a.centroid[3 * gj], a.centroid[3 * gj + 1], a.centroid[3 * gj + 2]};
    double uj[3];
    trial_data(valid_j ? lj : -1, uj);
    double lamj = 0.0;
    if (rj >= 0) {
        const int row = a.test_dof[rj];
        lamj = row >= 0 ? a.lam[row] : 0.0;
    }
    double gyacc[3][3] = {{0.0}};
    double kyacc[3] = {0.0};  // DATA: K^T lam at the trial panel's hats
    const double4* ptsj = a.pts + (size_t)gj * Q2;

    for (int t = 0; t < a.ti; ++t) {
        const int gi = s_gi[t];
        if (gi < 0) break;  // uniform across the CTA
        const bool both = s_ri[t] >= 0 && rj >= 0;
        const double lami = s_lam[t], lamb = both ? lamj : 0.0;
        const bool live = valid_j && !(both && gi > gj) && (lami != 0.0 || lamb != 0.0) &&
                          bem_relation(s_tri[t], tri_j, gi == gj) == REL_SEPARATE;
        double gx[3][3] = {{0.0}}, kx[3] = {0.0};
        if (live) {
            double ni[3], D[3];
            for (int c = 0; c < 3; ++c) {
                ni[c] = a.normal[3 * gi + c];
                D[c] = a.centroid[3 * gi + c] - cj[c];
            }
            const double4* sxt = sx + t * Q2;
            const double* sut = su + t * Q2;
            // vector sums along d: [hat moment (total, phi_1, phi_2)][component], x and y side
            double X[3][3] = {{0.0}}, Y[3][3] = {{0.0}};
            double S0 = 0.0;                                          // V: sum w/r
            double xa[3] = {0.0}, ya[3] = {0.0};                      // K: moments of A t (along n_j)
            double xb[3] = {0.0}, yb3[3] = {0.0};                     // K: moments of B t (along -n_i)
            double kj[3] = {0.0}, ki[3] = {0.0};                      // DATA: hat moments of K_ij and of -K_ji
            double sij = 0.0, sji = 0.0, Nj[3] = {0.0}, Ni[3] = {0.0};  // K: J_i, J_j, N_j and N_i parts
            const double Dnj = D[0] * nj[0] + D[1] * nj[1] + D[2] * nj[2];
            const double Dni = D[0] * ni[0] + D[1] * ni[1] + D[2] * ni[2];
            for (int b = 0; b < Q2; ++b) {
                const double4 yb = ptsj[b];
                const double e0 = D[0] - yb.x, e1 = D[1] - yb.y, e2 = D[2] - yb.z;
                const double2 pb = sp[b];
                double A = 0.0, dni = 0.0, lamdni = 0.0;
                if (K) {
                    A = lami * ((1.0 - pb.x - pb.y) * uj[0] + pb.x * uj[1] + pb.y * uj[2]);
                    dni = Dni - (yb.x * ni[0] + yb.y * ni[1] + yb.z * ni[2]);
                    lamdni = lamb * dni;
                }
                double v[3][3] = {{0.0}};  // [moment][component]
                double s0 = 0.0, ta[3] = {0.0}, tb[3] = {0.0}, tdn = 0.0, td[3] = {0.0}, tbd[3] = {0.0};
#pragma unroll 4
                for (int q = 0; q < Q2; ++q) {
                    const double4 xp = sxt[q];
                    const double2 ph = sp[q];
                    const double dx = xp.x + e0, dy = xp.y + e1, dz = xp.z + e2;
                    double r, rinv;
                    dev_r_rinv(fma(dx, dx, fma(dy, dy, dz * dz)), r, rinv);
                    const double rinv2 = rinv * rinv;
                    const double h = xp.w * rinv;
                    const double w3 = h * rinv2;  // w / r^3
                    double c;
                    if (!K) {
                        s0 += h;
                        c = w3;
                    } else {
                        const double ui = sut[q];
                        const double dnj = fma(xp.x, nj[0], fma(xp.y, nj[1], fma(xp.z, nj[2], Dnj)));
                        const double B = w3 * ui;  // without lam_j
                        // A d.n_j - B d.n_i, with lam_j
                        const double e = fma(A, dnj, -(lamdni * ui));
                        c = (w3 * rinv2) * e;
                        ta[0] += w3;
                        ta[1] = fma(ph.x, w3, ta[1]);
                        ta[2] = fma(ph.y, w3, ta[2]);
                        tb[0] += B;
                        tb[1] = fma(ph.x, B, tb[1]);
                        tb[2] = fma(ph.y, B, tb[2]);
                        tdn = fma(w3, dnj, tdn);
                        td[0] = fma(w3, dx, td[0]);
                        td[1] = fma(w3, dy, td[1]);
                        td[2] = fma(w3, dz, td[2]);
                        tbd[0] = fma(B, dx, tbd[0]);
                        tbd[1] = fma(B, dy, tbd[1]);
                        tbd[2] = fma(B, dz, tbd[2]);
                    }
                    const double vx = c * dx, vy = c * dy, vz = c * dz;
                    v[0][0] += vx;
                    v[0][1] += vy;
                    v[0][2] += vz;
                    v[1][0] = fma(ph.x, vx, v[1][0]);
                    v[1][1] = fma(ph.x, vy, v[1][1]);
                    v[1][2] = fma(ph.x, vz, v[1][2]);
                    v[2][0] = fma(ph.y, vx, v[2][0]);
                    v[2][1] = fma(ph.y, vy, v[2][1]);
                    v[2][2] = fma(ph.y, vz, v[2][2]);
                }
                const double w = yb.w;
                const double wp[3] = {w, w * pb.x, w * pb.y};
#pragma unroll
                for (int m = 0; m < 3; ++m)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        X[m][c] = fma(w, v[m][c], X[m][c]);
                        Y[m][c] = fma(wp[m], v[0][c], Y[m][c]);
                    }
                if (!K) {
                    S0 = fma(w, s0, S0);
                } else {
                    const double wA = w * A, wB = w * lamb;
                    sij = fma(wA, tdn, sij);
                    sji = fma(-wB * dni, tb[0], sji);
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        xa[m] = fma(wA, ta[m], xa[m]);
                        ya[m] = fma(wp[m] * A, ta[0], ya[m]);
                        xb[m] = fma(wB, tb[m], xb[m]);
                        yb3[m] = fma(wp[m] * lamb, tb[0], yb3[m]);
                        Nj[m] = fma(wA, td[m], Nj[m]);
                        Ni[m] = fma(-wB, tbd[m], Ni[m]);
                        if (DATA) {
                            kj[m] = fma(wp[m], tdn, kj[m]);
                            ki[m] = fma(w * dni, ta[m], ki[m]);
                        }
                    }
                }
            }
            // hats from the moments, and the vertices' gradients
            double vi[3][3], vj[3][3], n_[3];
            load_tri(a, gi, vi, n_);
            load_tri(a, gj, vj, n_);
            // one division a panel instead of one a component of a vertex, which at few points
            // cost as much as the points.  K, 5120 panels: GaussQR 1 2.48 -> 1.59 ms, 2 3.43 ->
            // 2.53 ms, 4 15.6 -> 14.8 ms; V 1.43 -> 1.24, 1.94 -> 1.70 and 8.54 -> 8.30 ms
            const double iJi = 0.5 / a.area[gi], iJj = 0.5 / a.area[gj];
            double cw = BEM_INV4PI;
            if (!K) cw *= lami * uj[0] + lamb * s_u[t][0];
            const double along = K ? -3.0 : -1.0;
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                double jg[3], hj[3], tx[3], ty[3];
                jac_grad(vi, ni, h, jg);
                jac_grad(vj, nj, h, hj);
                if (!K) {
                    for (int c = 0; c < 3; ++c) {
                        tx[c] = jg[c] * iJi * S0;
                        ty[c] = hj[c] * iJj * S0;
                    }
                } else {
                    double g1[3], g2[3];
                    normal_grad(vi, Ni, h, g1);
                    normal_grad(vj, Nj, h, g2);
                    for (int c = 0; c < 3; ++c) {
                        tx[c] = fma(jg[c], sij, g1[c]) * iJi;
                        ty[c] = fma(hj[c], sji, g2[c]) * iJj;
                    }
                    const double hxa = h == 0 ? xa[0] - xa[1] - xa[2] : xa[h], hya = h == 0 ? ya[0] - ya[1] - ya[2] : ya[h];
                    const double hxb = h == 0 ? xb[0] - xb[1] - xb[2] : xb[h],
                                 hyb = h == 0 ? yb3[0] - yb3[1] - yb3[2] : yb3[h];
                    for (int c = 0; c < 3; ++c) {
                        tx[c] += hxa * nj[c] - hxb * ni[c];
                        ty[c] -= hya * nj[c] - hyb * ni[c];
                    }
                }
                for (int c = 0; c < 3; ++c) {
                    const double hx = h == 0 ? X[0][c] - X[1][c] - X[2][c] : X[h][c];
                    const double hy = h == 0 ? Y[0][c] - Y[1][c] - Y[2][c] : Y[h][c];
                    gx[h][c] = cw * (tx[c] + along * hx);
                    gyacc[h][c] += cw * (ty[c] - along * hy);
                }
                if (DATA) {
                    kx[h] = -BEM_INV4PI * lamb * (h == 0 ? ki[0] - ki[1] - ki[2] : ki[h]);
                    kyacc[h] += BEM_INV4PI * lami * (h == 0 ? kj[0] - kj[1] - kj[2] : kj[h]);
                }
            }
        }
        // test-vertex gradients: reduce over the warp's trial panels
        for (int b = 0; b < 3; ++b)
            for (int c = 0; c < 3; ++c) gx[b][c] = warp_sum_d(gx[b][c]);
        if (lane == 0)
            for (int b = 0; b < 3; ++b)
                for (int c = 0; c < 3; ++c)
                    if (gx[b][c] != 0.0) atomicAdd(a.grad + 3 * s_tri[t][b] + c, gx[b][c]);
        if (DATA && s_ri[t] >= 0) {  // uniform across the CTA
            for (int b = 0; b < 3; ++b) kx[b] = warp_sum_d(kx[b]);
            if (lane < 3) {
                const int col = a.trial_dof[3 * s_ri[t] + lane];
                const double v = lane == 0 ? kx[0] : lane == 1 ? kx[1] : kx[2];
                if (col >= 0 && v != 0.0) atomicAdd(a.data + col, v);
            }
        }
    }
    if (valid_j)
        for (int b = 0; b < 3; ++b)
            for (int c = 0; c < 3; ++c)
                if (gyacc[b][c] != 0.0) atomicAdd(a.grad + 3 * tri_j[b] + c, gyacc[b][c]);
    if (DATA && valid_j)
        for (int b = 0; b < 3; ++b) {
            const int col = a.trial_dof[3 * lj + b];
            if (col >= 0 && kyacc[b] != 0.0) atomicAdd(a.data + col, kyacc[b]);
        }
}

// ---- near pairs: one warp per ordered pair of the near list ----
template <int OP>
__global__ void __launch_bounds__(128) adj_near_kernel(AdjArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t pid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (pid >= a.n_near) return;
    const int4 e = a.near[pid];
    const int gi = e.x, gj = e.y, rel = e.z;
    const int li = a.test_local[gi], lj = a.trial_local[gj];
    if (li < 0 || lj < 0) return;  // warp-uniform
    const int row = a.test_dof[li];
    if (row < 0) return;
    const double lam = a.lam[row];
    if (lam == 0.0) return;
    double uj[3] = {0.0, 0.0, 0.0};
    for (int b = 0; b < a.nby; ++b) {
        const int col = a.trial_dof[lj * a.nby + b];
        uj[b] = col >= 0 ? a.u[col] : 0.0;
    }
    // slot order of the Sauter-Schwab maps (as in the assembly's near kernel)
    const int permx = a.quirk ? (0 | (1 << 2) | (2 << 4)) : (e.w & 63);
    const int permy = a.quirk ? (0 | (1 << 2) | (2 << 4)) : ((e.w >> 6) & 63);
    const int pmx[3] = {permx & 3, (permx >> 2) & 3, (permx >> 4) & 3};
    const int pmy[3] = {permy & 3, (permy >> 2) & 3, (permy >> 4) & 3};
    double vi[3][3], ni[3], vj[3][3], nj[3];
    load_tri(a, gi, vi, ni);
    load_tri(a, gj, vj, nj);
    const double Ji = 2.0 * a.area[gi], Jj = 2.0 * a.area[gj];
    double X[3][3], Y[3][3];  // slot s = stored vertex pm[s]
    int slotx[3], sloty[3];   // slot of stored vertex b
    for (int s = 0; s < 3; ++s) {
        for (int c = 0; c < 3; ++c) {
            X[s][c] = vi[pmx[s]][c];
            Y[s][c] = vj[pmy[s]][c];
        }
        slotx[pmx[s]] = s;
        sloty[pmy[s]] = s;
    }
    PairMoments M;
    M.zero();
    const bool twin = rel == REL_COINCIDE, quirk = a.quirk != 0;
    const double invJj = 1.0 / Jj;
    auto add = [&](double r1x, double r2x, double r1y, double r2y, double wj) {
        const double sx_[3] = {1.0 - r1x, r1x - r2x, r2x};
        const double sy_[3] = {1.0 - r1y, r1y - r2y, r2y};
        double d[3];
        for (int c = 0; c < 3; ++c)
            d[c] = (sx_[0] * X[0][c] + sx_[1] * X[1][c] + sx_[2] * X[2][c]) -
                   (sy_[0] * Y[0][c] + sy_[1] * Y[1][c] + sy_[2] * Y[2][c]);
        // barycentric weights per stored vertex
        const double bx[3] = {sx_[slotx[0]], sx_[slotx[1]], sx_[slotx[2]]};
        const double by[3] = {sy_[sloty[0]], sy_[sloty[1]], sy_[sloty[2]]};
        // P1 data at the trial point; the swapped twin of a coincident point has the
        // opposite normal derivative, with the data at the same point (quirk: the two
        // cancel) or at the test point's parameters, and V's same value
        double ub = 1.0, w = wj, hy[3] = {by[0], by[1], by[2]};
        if (OP == BEM_OP_K) {
            ub = by[0] * uj[0] + by[1] * uj[1] + by[2] * uj[2];
            if (twin) {
                ub -= quirk ? ub : sx_[sloty[0]] * uj[0] + sx_[sloty[1]] * uj[1] + sx_[sloty[2]] * uj[2];
                for (int b = 0; b < 3; ++b) hy[b] -= quirk ? by[b] : sx_[sloty[b]];
            }
        } else if (twin) {
            w = wj + wj;
        }
        adj_point<OP>(M, d, w, bx, by, hy, ub, 1.0, nj, invJj);
    };
    NearDigits dg;
    const int Q = a.Q, Q4 = Q * Q * Q * Q;
    dg.start(lane, Q);
    for (int p = lane; p < Q4; p += 32) {
        const double weight = (a.gw[dg.ix] * a.gw[dg.iy] * Ji) * (a.gw[dg.iz] * a.gw[dg.iw] * Jj);
        near_points(rel, a.gp[dg.ix], a.gp[dg.iy], a.gp[dg.iz], a.gp[dg.iw], weight, add);
        dg.next(Q);
    }
    M.reduce();
    if (lane != 0) return;
    double gx[3][3], gy[3][3];
    pair_grads<OP>(M, lam * (OP == BEM_OP_V ? uj[0] : 1.0), vi, ni, Ji, vj, nj, Jj, gx, gy);
    const int32_t* ti = a.tris + 3 * gi;
    const int32_t* tj = a.tris + 3 * gj;
    for (int b = 0; b < 3; ++b)
        for (int c = 0; c < 3; ++c) {
            atomicAdd(a.grad + 3 * ti[b] + c, gx[b][c]);
            atomicAdd(a.grad + 3 * tj[b] + c, gy[b][c]);
        }
    if (OP == BEM_OP_K && a.data)
        for (int b = 0; b < 3; ++b) {
            const int col = a.trial_dof[3 * lj + b];
            if (col >= 0) atomicAdd(a.data + col, lam * M.SU[b]);
        }
}

}  // namespace

int bem_launch_adjoint(bem_ctx* ctx, const bem_op_desc* op, const bem_space* test, const bem_space* trial,
                       const double* lam, const double* u, double* grad, double* data, cudaStream_t s) {
    if (int rc = bem_fill_local_map(ctx, test, ctx->test_local, s)) return rc;
    if (int rc = bem_fill_local_map(ctx, trial, ctx->trial_local, s)) return rc;
    AdjArgs a;
    a.n_test = test->n_panels;
    a.n_trial = trial->n_panels;
    a.test_panels = test->panels;
    a.test_dof = test->dof;
    a.trial_panels = trial->panels;
    a.trial_dof = trial->dof;
    a.nby = trial->nb;
    a.tris = ctx->tris;
    a.verts = ctx->verts;
    a.centroid = ctx->centroid;
    a.normal = ctx->normal;
    a.area = ctx->area;
    a.pts = ctx->pts64;
    a.phi64 = ctx->phi64;
    a.Q2 = ctx->Q2;
    a.n_near = ctx->n_near;
    a.near = ctx->near;
    a.test_local = ctx->test_local;
    a.trial_local = ctx->trial_local;
    a.gp = ctx->gp;
    a.gw = ctx->gw;
    a.Q = ctx->Q;
    a.quirk = op->quirk;
    a.lam = lam;
    a.u = u;
    a.grad = grad;
    a.data = data;
    // as in bem_launch_far64: fewer test panels per CTA where the call has too few
    // CTAs for some waves.  With few points a pair the trial vertices' atomics, one
    // set per CTA, weigh more than idle SMs (K, 320 panels, GaussQR 2: 114, 97, 86
    // and 93 us with 1, 2, 4 and 8; GaussQR 5: 403, 475, 528 and 622 us)
    a.ti = ADJ_TI;
    const int64_t cols = (a.n_trial + ADJ_THREADS - 1) / ADJ_THREADS;
    const int64_t want = (int64_t)ctx->num_sms * (ctx->Q2 <= 4 ? 1 : (ctx->Q2 <= 9 ? 3 : 16));
    while (a.ti > 1 && cols * ((a.n_test + a.ti - 1) / a.ti) < want) a.ti /= 2;
    const size_t smem = ((sizeof(double4) + sizeof(double)) * a.ti + sizeof(double2)) * ctx->Q2;
    const dim3 fgrid((unsigned)cols, (unsigned)((a.n_test + a.ti - 1) / a.ti));
    const unsigned nblocks = (unsigned)((a.n_near + 3) / 4);
    if (a.n_test > 0 && a.n_trial > 0) {
        if (op->op == BEM_OP_V) {
            adj_far_kernel<BEM_OP_V, false><<<fgrid, ADJ_THREADS, smem, s>>>(a);
            if (nblocks) adj_near_kernel<BEM_OP_V><<<nblocks, 128, 0, s>>>(a);
        } else {
            if (data)
                adj_far_kernel<BEM_OP_K, true><<<fgrid, ADJ_THREADS, smem, s>>>(a);
            else
                adj_far_kernel<BEM_OP_K, false><<<fgrid, ADJ_THREADS, smem, s>>>(a);
            if (nblocks) adj_near_kernel<BEM_OP_K><<<nblocks, 128, 0, s>>>(a);
        }
        ctx->launches += nblocks ? 2 : 1;
    }
    return bem_check_cuda(ctx, cudaGetLastError(), "adjoint kernels launch");
}
