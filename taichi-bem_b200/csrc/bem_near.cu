// Near field: coincident / common-edge / common-vertex panel pairs in FP64
// (Sauter-Schwab maps, bem_quadrature.cuh), one warp per ordered pair of the
// near list, lanes over the GaussQR^4 points.
//
// The reference integrates each operator, scope and basis pair on its own
// (single_layer_3d.py:178-367 and its twins).  The kernel's value depends on
// the point pair and the wavenumber only, so a warp evaluates r, 1/r and
// e^{ikr} once for every basis pair, for both wavenumbers of a batch and, in
// the fused passes, for V, K and W together:
//   sum w G (1, phi_1, phi_2)_x (1, phi_1, phi_2)_y        V and W (G = e^{ikr}/r)
//   sum w (d.n) F / r^3 (1, phi_1, phi_2)_x (...)_y        K and K' (F = (1 - ikr) e^{ikr})
// and phi_0 = 1 - phi_1 - phi_2 is formed at the end.  Bound: FP64 issue; per
// point 12 instructions for d (affine in the four parameters), 9 for r and
// 1/r, 13 to 24 for the phase, the rest for the moments.  The twin of each
// coincident point (swapped kernel arguments) costs no evaluation.  The lanes
// share the writes.  Measured (B200, against one kernel per operator and
// wavenumber with the library's root and sincos): the Calderon blocks of two
// wavenumbers, 5120 panels, GaussQR 4: 1.86 against 7.4 ms; V, K and W (P1) of
// eight wavenumbers, 1280 panels, GaussQR 3: 2.0 against 5.8 ms; W, 990 panels,
// GaussQR 4: 0.16 against 0.41 ms.
#include <cmath>

#include "bem_farfield.cuh"
#include "bem_quadrature.cuh"

namespace {

constexpr int NEAR_MAXK = 2;

struct NearArgs {
    int64_t n_near;
    const int4* near;
    const int32_t* test_local;
    const int32_t* trial_local;
    const int32_t* test_dof;
    const int32_t* trial_dof;
    const int32_t* tris;
    const double* verts;
    const double* area;
    const double* normal;
    const double* curl;
    const double* gp;
    const double* gw;
    int Q;
    int quirk;
    int ph;  // bound on the phase k r of a touching pair: 2 (<= 0.3), 1 (<= pi/4), 0 (any)
    int dk;  // 1: the kernel's k-derivative
    double k[NEAR_MAXK], k2[NEAR_MAXK];
    int mode;
    double* out[NEAR_MAXK];
    int64_t ld;
    double scale[NEAR_MAXK];
    double* out_t[NEAR_MAXK];
    double scale_t[NEAR_MAXK];
    const double* x;
    double* y;
    int conj_x;
    // fused passes: the second space's dofs (Calderon: P1 of both sides; Dirichlet: data), and K's scale
    const int32_t* dof2;
    const int32_t* rows;
    int nbd;
    double scale_k;
};

__device__ __forceinline__ void near_sincos(int ph, double y, double* s, double* c) {
    if (ph == 2)
        dev_sincos_poly64<true>(y, s, c);
    else if (ph == 1)
        dev_sincos_poly64<false>(y, s, c);
    else
        dev_sincos(y, s, c);
}

// One pair: panels, relation and the slot of each stored vertex in the maps' parameters
struct NearPair {
    int gi, gj, li, lj, rel;
    int sx[3], sy[3];  // slot of stored vertex b
    double B[3], a1[3], a2[3], b1[3], b2[3];  // d = B + r1x a1 + r2x a2 - r1y b1 - r2y b2
    double nx[3], ny[3];
    double JJ;  // (2 A_x)(2 A_y)
};

__device__ __forceinline__ bool near_load(const NearArgs& a, int64_t pid, NearPair& P) {
    const int4 e = a.near[pid];
    P.gi = e.x;
    P.gj = e.y;
    P.rel = e.z;
    P.li = a.test_local[P.gi];
    P.lj = a.trial_local[P.gj];
    if (P.li < 0 || P.lj < 0) return false;
    const int id = 0 | (1 << 2) | (2 << 4);
    const int px = a.quirk ? id : (e.w & 63), py = a.quirk ? id : ((e.w >> 6) & 63);
    double X[3][3], Y[3][3];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const int vx = (px >> (2 * s)) & 3, vy = (py >> (2 * s)) & 3;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            if (vx == b) P.sx[b] = s;
            if (vy == b) P.sy[b] = s;
        }
        const int tx = a.tris[3 * P.gi + vx], ty = a.tris[3 * P.gj + vy];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            X[s][c] = a.verts[3 * tx + c];
            Y[s][c] = a.verts[3 * ty + c];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        P.B[c] = X[0][c] - Y[0][c];
        P.a1[c] = X[1][c] - X[0][c];
        P.a2[c] = X[2][c] - X[1][c];
        P.b1[c] = Y[1][c] - Y[0][c];
        P.b2[c] = Y[2][c] - Y[1][c];
        P.nx[c] = a.normal[3 * P.gi + c];
        P.ny[c] = a.normal[3 * P.gj + c];
    }
    P.JJ = (2.0 * a.area[P.gi]) * (2.0 * a.area[P.gj]);
    return true;
}

// Moments of one pair: G over GX x GY and the normal derivative over KX x KY
// functions (1 or 3 a side: the constant, or (1, phi_1, phi_2)); 0 x 0 = absent.
template <int NK, int GX, int GY, int KX, int KY>
struct NearMoments {
    static constexpr int NG = GX * GY > 0 ? GX * GY : 1, ND = KX * KY > 0 ? KX * KY : 1;
    double gr[NK][NG], gi[NK][NG], kr[NK][ND], ki[NK][ND];
};

// KP: the normal derivative is K's (n_y, sign +) or K''s (n_x, sign -)
template <bool HELM, int NK, int GX, int GY, int KX, int KY, bool KP>
__device__ __forceinline__ void near_integrate(const NearArgs& a, const NearPair& P, const double* gp, const double* gw,
                                               NearMoments<NK, GX, GY, KX, KY>& M) {
    constexpr bool G = GX * GY > 0, K = KX * KY > 0;
    constexpr int FX = GX > KX ? GX : KX, FY = GY > KY ? GY : KY;
#pragma unroll
    for (int w = 0; w < NK; ++w) {
#pragma unroll
        for (int m = 0; m < M.NG; ++m) M.gr[w][m] = M.gi[w][m] = 0.0;
#pragma unroll
        for (int m = 0; m < M.ND; ++m) M.kr[w][m] = M.ki[w][m] = 0.0;
    }
    const bool twin = P.rel == REL_COINCIDE;
    const bool quirk = a.quirk != 0;
    // the reference's twin of a normal derivative cancels its own point
    const bool with_k = K && !(twin && quirk);
    const int Q = a.Q, Q4 = Q * Q * Q * Q;
    const int lane = threadIdx.x & 31;
    const int ph = a.ph;
    const bool dk = a.dk != 0;
    auto add = [&](double r1x, double r2x, double r1y, double r2y, double w) {
        double d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            d[c] = fma(r1x, P.a1[c], fma(r2x, P.a2[c], fma(-r1y, P.b1[c], fma(-r2y, P.b2[c], P.B[c]))));
        double r, rinv;
        dev_r_rinv(fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2])), r, rinv);
        // basis products, the twin's included
        const double fx[3] = {1.0, r1x - r2x, r2x}, fy[3] = {1.0, r1y - r2y, r2y};
        double cg[FX * FY > 0 ? FX * FY : 1], ck[FX * FY > 0 ? FX * FY : 1];
#pragma unroll
        for (int x = 0; x < FX; ++x)
#pragma unroll
            for (int y = 0; y < FY; ++y) {
                const double c = x == 0 ? fy[y] : (y == 0 ? fx[x] : fx[x] * fy[y]);
                double g = c, k = c;
                if (twin) {
                    const double t = quirk ? c : (x == 0 ? fx[y] : (y == 0 ? fy[x] : fy[x] * fx[y]));
                    g = c + t;
                    k = c - t;
                }
                cg[x * FY + y] = g;
                ck[x * FY + y] = k;
            }
        const double wr = w * rinv;
        double tk = 0.0, dn = 0.0;
        if (K) {
            dn = KP ? -(d[0] * P.nx[0] + d[1] * P.nx[1] + d[2] * P.nx[2])
                    : d[0] * P.ny[0] + d[1] * P.ny[1] + d[2] * P.ny[2];
            tk = wr * (rinv * rinv) * dn;
        }
#pragma unroll
        for (int q = 0; q < NK; ++q) {
            double gr = wr, gi = 0.0, kr = tk, ki = 0.0;
            if (HELM) {
                const double p = a.k[q] * r;
                double s, c;
                near_sincos(ph, p, &s, &c);
                gr = dk ? -w * s : wr * c;
                gi = dk ? w * c : wr * s;
                if (K) {
                    const double f = wr * dn * a.k[q];
                    kr = dk ? f * c : tk * fma(p, s, c);
                    ki = dk ? f * s : tk * fma(-p, c, s);
                }
            }
            if (G)
#pragma unroll
                for (int x = 0; x < GX; ++x)
#pragma unroll
                    for (int y = 0; y < GY; ++y) {
                        M.gr[q][x * GY + y] = fma(cg[x * FY + y], gr, M.gr[q][x * GY + y]);
                        if (HELM) M.gi[q][x * GY + y] = fma(cg[x * FY + y], gi, M.gi[q][x * GY + y]);
                    }
            if (with_k)
#pragma unroll
                for (int x = 0; x < KX; ++x)
#pragma unroll
                    for (int y = 0; y < KY; ++y) {
                        M.kr[q][x * KY + y] = fma(ck[x * FY + y], kr, M.kr[q][x * KY + y]);
                        if (HELM) M.ki[q][x * KY + y] = fma(ck[x * FY + y], ki, M.ki[q][x * KY + y]);
                    }
        }
    };
    NearDigits dg;
    dg.start(lane, Q);
    for (int p = lane; p < Q4; p += 32) {
        const double weight = (gw[dg.ix] * gw[dg.iy]) * (gw[dg.iz] * gw[dg.iw]) * P.JJ;
        near_points(P.rel, gp[dg.ix], gp[dg.iy], gp[dg.iz], gp[dg.iw], weight, add);
        dg.next(Q);
    }
    // the warp's sums in every lane, without 1/(4 pi)
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        if (G)
#pragma unroll
            for (int m = 0; m < M.NG; ++m) {
                M.gr[q][m] = warp_sum(M.gr[q][m]);
                if (HELM) M.gi[q][m] = warp_sum(M.gi[q][m]);
            }
        if (with_k)
#pragma unroll
            for (int m = 0; m < M.ND; ++m) {
                M.kr[q][m] = warp_sum(M.kr[q][m]);
                if (HELM) M.ki[q][m] = warp_sum(M.ki[q][m]);
            }
    }
}

// Basis pair (bx, by) of stored vertices from the moments (MX x MY, slots through
// sx / sy): a hat of slot 0 is total - phi_1 - phi_2.
template <int MX, int MY>
__device__ __forceinline__ double near_hat(const double* m, const int* sx, const int* sy, int bx, int by) {
    double row[MX];
    int qy = 0;
    if (MY == 3) qy = by == 0 ? sy[0] : (by == 1 ? sy[1] : sy[2]);
#pragma unroll
    for (int x = 0; x < MX; ++x) {
        if (MY == 1)
            row[x] = m[x];
        else
            row[x] = qy == 0 ? m[x * MY] - m[x * MY + 1] - m[x * MY + 2] : (qy == 1 ? m[x * MY + 1] : m[x * MY + 2]);
    }
    if (MX == 1) return row[0];
    const int qx = bx == 0 ? sx[0] : (bx == 1 ? sx[1] : sx[2]);
    return qx == 0 ? row[0] - row[MX > 1 ? 1 : 0] - row[MX > 2 ? 2 : 0] : (qx == 1 ? row[MX > 1 ? 1 : 0] : row[MX > 2 ? 2 : 0]);
}

__device__ __forceinline__ double curl_dot(const NearArgs& a, const NearPair& P, int bx, int by) {
    const double* cx = a.curl + 9 * (int64_t)P.gi + 3 * bx;
    const double* cy = a.curl + 9 * (int64_t)P.gj + 3 * by;
    return cx[0] * cy[0] + cx[1] * cy[1] + cx[2] * cy[2];
}

__device__ __forceinline__ void near_tables(const NearArgs& a, double* gp, double* gw) {
    if (threadIdx.x < a.Q) {
        gp[threadIdx.x] = a.gp[threadIdx.x];
        gw[threadIdx.x] = a.gw[threadIdx.x];
    }
    __syncthreads();
}

// ---- one operator, NK wavenumbers ----
template <int OP, bool HELM, int NBX, int NBY, int NK>
__global__ void __launch_bounds__(128) near_kernel(NearArgs a) {
    constexpr bool W_OP = OP == BEM_OP_W, DER = OP == BEM_OP_K || OP == BEM_OP_KP;
    // Laplace W has no mass term: its one moment is the total
    constexpr bool PHI = !(W_OP && !HELM);
    constexpr int MX = PHI ? NBX : 1, MY = PHI ? NBY : 1;
    __shared__ double s_gp[BEM_MAX_Q], s_gw[BEM_MAX_Q];
    near_tables(a, s_gp, s_gw);
    const int lane = threadIdx.x & 31;
    const int64_t pid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    NearPair P;
    if (pid >= a.n_near || !near_load(a, pid, P)) return;  // warp-uniform
    NearMoments<NK, DER ? 0 : MX, DER ? 0 : MY, DER ? MX : 0, DER ? MY : 0> M;
    near_integrate<HELM, NK, DER ? 0 : MX, DER ? 0 : MY, DER ? MX : 0, DER ? MY : 0, OP == BEM_OP_KP>(a, P, s_gp, s_gw, M);
    // lane e < NBX NBY: basis pair (e / NBY, e % NBY)
    const int bx = lane / NBY, by = lane - bx * NBY;
    if (lane >= NBX * NBY) {
        if (a.mode == 0) return;
    }
    const bool own = lane < NBX * NBY;
    const int row = own ? a.test_dof[P.li * NBX + bx] : -1;
    const int col = own ? a.trial_dof[P.lj * NBY + by] : -1;
    double cd = 0.0, nd = 0.0;
    if (W_OP && own) {
        nd = P.nx[0] * P.ny[0] + P.nx[1] * P.ny[1] + P.nx[2] * P.ny[2];
        if (NBX == 3 && NBY == 3) cd = curl_dot(a, P, bx, by);
    }
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        const double* mr = DER ? M.kr[q] : M.gr[q];
        const double* mi = DER ? M.ki[q] : M.gi[q];
        double vr, vi;
        if (W_OP) {
            // W = G curl.curl - k2 (n_x.n_y) G phi_x phi_y (hypersingular_layer_3d.py:206-211)
            vr = mr[0] * cd;
            vi = mi[0] * cd;
            if (PHI) {
                vr -= a.k2[q] * nd * near_hat<MX, MY>(mr, P.sx, P.sy, bx, by);
                if (HELM) vi -= a.k2[q] * nd * near_hat<MX, MY>(mi, P.sx, P.sy, bx, by);
            }
        } else {
            vr = near_hat<MX, MY>(mr, P.sx, P.sy, bx, by);
            vi = HELM ? near_hat<MX, MY>(mi, P.sx, P.sy, bx, by) : 0.0;
        }
        vr *= BEM_INV4PI;
        vi *= BEM_INV4PI;
        if (row < 0 || col < 0) continue;
        if (a.mode == 0) {
            if (a.out[q] == nullptr) continue;
            add_entry<HELM>(a.out[q], (int64_t)row * a.ld + col, a.scale[q] * vr, a.scale[q] * vi, true);
            if (a.out_t[q])
                add_entry<HELM>(a.out_t[q], (int64_t)col * a.ld + row, a.scale_t[q] * vr, a.scale_t[q] * vi, true);
        } else if (HELM) {
            const double xr = a.x[2 * (int64_t)col], xi = a.conj_x ? -a.x[2 * (int64_t)col + 1] : a.x[2 * (int64_t)col + 1];
            atomicAdd(a.y + 2 * (int64_t)row, a.scale[q] * (vr * xr - vi * xi));
            atomicAdd(a.y + 2 * (int64_t)row + 1, a.scale[q] * (vr * xi + vi * xr));
        } else {
            atomicAdd(a.y + row, a.scale[q] * (vr * a.x[col]));
        }
    }
}

// ---- Dirichlet pass: V (P0 x P0, dense) and K g (P0 rows, NBD data bases) ----
template <bool HELM, int NBD>
__global__ void __launch_bounds__(128) near_vkg_kernel(NearArgs a) {
    __shared__ double s_gp[BEM_MAX_Q], s_gw[BEM_MAX_Q];
    near_tables(a, s_gp, s_gw);
    const int lane = threadIdx.x & 31;
    const int64_t pid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    NearPair P;
    if (pid >= a.n_near || !near_load(a, pid, P)) return;  // warp-uniform
    NearMoments<1, 1, 1, 1, NBD> M;
    near_integrate<HELM, 1, 1, 1, 1, NBD, false>(a, P, s_gp, s_gw, M);
    if (lane == 0) {
        const int row = a.test_dof[P.li], col = a.trial_dof[P.lj];
        if (row >= 0 && col >= 0)
            add_entry<HELM>(a.out[0], (int64_t)row * a.ld + col, a.scale[0] * (BEM_INV4PI * M.gr[0][0]),
                            a.scale[0] * (BEM_INV4PI * M.gi[0][0]), true);
    } else if (lane == 1) {
        const int row = a.rows[P.li];
        if (row < 0) return;
        double cr = 0.0, ci = 0.0;
#pragma unroll
        for (int b = 0; b < NBD; ++b) {
            const int col = a.dof2[P.lj * NBD + b];
            if (col < 0) continue;
            const double vr = near_hat<1, NBD>(M.kr[0], P.sx, P.sy, 0, b);
            if (HELM) {
                const double vi = near_hat<1, NBD>(M.ki[0], P.sx, P.sy, 0, b);
                const double xr = a.x[2 * (int64_t)col],
                             xi = a.conj_x ? -a.x[2 * (int64_t)col + 1] : a.x[2 * (int64_t)col + 1];
                cr += vr * xr - vi * xi;
                ci += vr * xi + vi * xr;
            } else {
                cr += vr * a.x[col];
            }
        }
        cr *= BEM_INV4PI;
        ci *= BEM_INV4PI;
        if (HELM) {
            atomicAdd(a.y + 2 * (int64_t)row, a.scale_k * cr);
            atomicAdd(a.y + 2 * (int64_t)row + 1, a.scale_k * ci);
        } else {
            atomicAdd(a.y + row, a.scale_k * cr);
        }
    }
}

// ---- Calderon blocks: V, K, -K^T and W of NK wavenumbers (bem_calderon.cu's placement) ----
template <bool HELM, int NK>
__global__ void __launch_bounds__(128) near_calderon_kernel(NearArgs a) {
    constexpr int GX = HELM ? 3 : 1;  // Laplace W has no mass term
    __shared__ double s_gp[BEM_MAX_Q], s_gw[BEM_MAX_Q];
    near_tables(a, s_gp, s_gw);
    const int lane = threadIdx.x & 31;
    const int64_t pid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    NearPair P;
    if (pid >= a.n_near || !near_load(a, pid, P)) return;  // warp-uniform
    NearMoments<NK, GX, GX, 1, 3> M;
    near_integrate<HELM, NK, GX, GX, 1, 3, false>(a, P, s_gp, s_gw, M);
    // lane 0: V; 1..3: K; 4..6: -K^T; 7..15: W
    if (lane > 15) return;
    const int h = lane >= 7 ? 0 : (lane >= 4 ? lane - 4 : (lane >= 1 ? lane - 1 : 0));
    const int bx = lane >= 7 ? (lane - 7) / 3 : 0, by = lane >= 7 ? (lane - 7) % 3 : 0;
    const int ni = a.test_dof[P.li];
    int row, col;
    if (lane == 0) {
        row = ni;
        col = a.trial_dof[P.lj];
    } else if (lane < 7) {
        const int dj = a.dof2[P.lj * 3 + h];
        row = lane < 4 ? ni : dj;
        col = lane < 4 ? dj : ni;
    } else {
        row = a.dof2[P.li * 3 + bx];
        col = a.dof2[P.lj * 3 + by];
    }
    if (row < 0 || col < 0) return;
    double cd = 0.0, nd = 0.0;
    if (lane >= 7) {
        nd = P.nx[0] * P.ny[0] + P.nx[1] * P.ny[1] + P.nx[2] * P.ny[2];
        cd = curl_dot(a, P, bx, by);
    }
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        double vr, vi;
        if (lane == 0) {
            vr = -M.gr[q][0];
            vi = -M.gi[q][0];
        } else if (lane < 7) {
            const double s = lane < 4 ? 1.0 : -1.0;
            vr = s * near_hat<1, 3>(M.kr[q], P.sx, P.sy, 0, h);
            vi = HELM ? s * near_hat<1, 3>(M.ki[q], P.sx, P.sy, 0, h) : 0.0;
        } else {
            vr = -M.gr[q][0] * cd;
            vi = -M.gi[q][0] * cd;
            if (HELM) {
                vr += a.k2[q] * nd * near_hat<GX, GX>(M.gr[q], P.sx, P.sy, bx, by);
                vi += a.k2[q] * nd * near_hat<GX, GX>(M.gi[q], P.sx, P.sy, bx, by);
            }
        }
        add_entry<HELM>(a.out[q], (int64_t)row * a.ld + col, a.scale[q] * (BEM_INV4PI * vr),
                        a.scale[q] * (BEM_INV4PI * vi), true);
    }
}

NearArgs near_args(bem_ctx* ctx, const bem_op_desc* op, double kmax) {
    NearArgs a{};
    a.n_near = ctx->n_near;
    a.near = ctx->near;
    a.test_local = ctx->test_local;
    a.trial_local = ctx->trial_local;
    a.tris = ctx->tris;
    a.verts = ctx->verts;
    a.area = ctx->area;
    a.normal = ctx->normal;
    a.curl = ctx->curl;
    a.gp = ctx->gp;
    a.gw = ctx->gw;
    a.Q = ctx->Q;
    a.quirk = op->quirk;
    a.dk = op->deriv_k ? 1 : 0;
    // two points of touching panels are at most two panel diameters apart
    a.ph = op->kernel == BEM_KERNEL_HELMHOLTZ ? bem_phase_class(std::fabs(kmax) * 4.0 * ctx->rho_max) : 0;
    return a;
}

template <int OP, int NK>
int dispatch_near(bem_ctx* ctx, const NearArgs& a, bool helm, int nbx, int nby, cudaStream_t s) {
    const unsigned blocks = (unsigned)((a.n_near + 3) / 4);
    bool ok = true;
#define BEM_NEAR_CASE(X, Y)                                                       \
    if (nbx == X && nby == Y) {                                                   \
        if (helm)                                                                 \
            near_kernel<OP, true, X, Y, NK><<<blocks, 128, 0, s>>>(a);            \
        else if constexpr (NK == 1)                                               \
            near_kernel<OP, false, X, Y, 1><<<blocks, 128, 0, s>>>(a);            \
        else                                                                      \
            ok = false;                                                           \
    } else
    BEM_NEAR_CASE(1, 1)
    BEM_NEAR_CASE(1, 3)
    BEM_NEAR_CASE(3, 1)
    BEM_NEAR_CASE(3, 3) ok = false;
#undef BEM_NEAR_CASE
    if (!ok) return bem_fail(ctx, BEM_ERR_INVALID, "nb must be 1 (P0) or 3 (P1)");
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "near_kernel launch");
}

template <int NK>
int dispatch_near_op(bem_ctx* ctx, const NearArgs& a, int op, bool helm, int nbx, int nby, cudaStream_t s) {
    switch (op) {
        case BEM_OP_V: return dispatch_near<BEM_OP_V, NK>(ctx, a, helm, nbx, nby, s);
        case BEM_OP_K: return dispatch_near<BEM_OP_K, NK>(ctx, a, helm, nbx, nby, s);
        case BEM_OP_KP: return dispatch_near<BEM_OP_KP, NK>(ctx, a, helm, nbx, nby, s);
        case BEM_OP_W: return dispatch_near<BEM_OP_W, NK>(ctx, a, helm, nbx, nby, s);
        default: return bem_fail(ctx, BEM_ERR_INVALID, "unknown operator");
    }
}

}  // namespace

int bem_launch_near(bem_ctx* ctx, const bem_op_desc* op, const bem_space* test, const bem_space* trial, int mode,
                    void* out, int64_t ld, double scale, void* out_t, double scale_t, const void* x, void* y, int conj_x,
                    cudaStream_t s) {
    if (ctx->n_near <= 0) return BEM_OK;
    NearArgs a = near_args(ctx, op, op->k);
    a.test_dof = test->dof;
    a.trial_dof = trial->dof;
    a.k[0] = op->k;
    a.k2[0] = op->k2;
    a.mode = mode;
    a.out[0] = (double*)out;
    a.ld = ld;
    a.scale[0] = scale;
    a.out_t[0] = (double*)out_t;
    a.scale_t[0] = scale_t;
    a.x = (const double*)x;
    a.y = (double*)y;
    a.conj_x = conj_x;
    return dispatch_near_op<1>(ctx, a, op->op, op->kernel == BEM_KERNEL_HELMHOLTZ, test->nb, trial->nb, s);
}

int bem_launch_near_batch(bem_ctx* ctx, const bem_op_desc* op, const bem_space* test, const bem_space* trial, int nk,
                          const double* k, const double* k2, void* const* out, int64_t ld, const double* scale,
                          void* const* out_t, const double* scale_t, cudaStream_t s) {
    if (ctx->n_near <= 0) return BEM_OK;
    double kmax = 0.0;
    for (int w = 0; w < nk; ++w) kmax = std::fmax(kmax, std::fabs(k[w]));
    for (int w0 = 0; w0 < nk; w0 += NEAR_MAXK) {
        const int m = nk - w0 < NEAR_MAXK ? nk - w0 : NEAR_MAXK;
        NearArgs a = near_args(ctx, op, kmax);
        a.test_dof = test->dof;
        a.trial_dof = trial->dof;
        a.ld = ld;
        for (int w = 0; w < m; ++w) {
            a.k[w] = k[w0 + w];
            a.k2[w] = k2[w0 + w];
            a.out[w] = (double*)out[w0 + w];
            a.scale[w] = scale[w0 + w];
            a.out_t[w] = out_t ? (double*)out_t[w0 + w] : nullptr;
            a.scale_t[w] = a.out_t[w] ? scale_t[w0 + w] : 0.0;
        }
        const int rc = m == 2 ? dispatch_near_op<2>(ctx, a, op->op, true, test->nb, trial->nb, s)
                              : dispatch_near_op<1>(ctx, a, op->op, true, test->nb, trial->nb, s);
        if (rc) return rc;
    }
    return BEM_OK;
}

int bem_launch_near_dirichlet(bem_ctx* ctx, const bem_op_desc* op, const bem_space* test, const bem_space* trial,
                              void* out, int64_t ld, double scale, const bem_space* rows, const bem_space* data,
                              const void* g, void* y, double scale_k, int conj_g, cudaStream_t s) {
    if (ctx->n_near <= 0) return BEM_OK;
    NearArgs a = near_args(ctx, op, op->k);
    a.test_dof = test->dof;
    a.trial_dof = trial->dof;
    a.rows = rows->dof;
    a.dof2 = data->dof;
    a.k[0] = op->k;
    a.out[0] = (double*)out;
    a.ld = ld;
    a.scale[0] = scale;
    a.x = (const double*)g;
    a.y = (double*)y;
    a.scale_k = scale_k;
    a.conj_x = conj_g;
    const unsigned blocks = (unsigned)((a.n_near + 3) / 4);
    const bool helm = op->kernel == BEM_KERNEL_HELMHOLTZ;
    if (helm && data->nb == 3)
        near_vkg_kernel<true, 3><<<blocks, 128, 0, s>>>(a);
    else if (helm)
        near_vkg_kernel<true, 1><<<blocks, 128, 0, s>>>(a);
    else if (data->nb == 3)
        near_vkg_kernel<false, 3><<<blocks, 128, 0, s>>>(a);
    else
        near_vkg_kernel<false, 1><<<blocks, 128, 0, s>>>(a);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "near_vkg_kernel launch");
}

int bem_launch_near_calderon(bem_ctx* ctx, const bem_op_desc* op, int nk, const double* k, const double* k2,
                             const bem_space* neu, const bem_space* dir, void* const* out, const double* coef, int64_t ld,
                             cudaStream_t s) {
    if (ctx->n_near <= 0) return BEM_OK;
    double kmax = 0.0;
    for (int w = 0; w < nk; ++w) kmax = std::fmax(kmax, std::fabs(k[w]));
    NearArgs a = near_args(ctx, op, kmax);
    a.test_dof = a.trial_dof = neu->dof;
    a.dof2 = dir->dof;
    a.ld = ld;
    for (int w = 0; w < nk; ++w) {
        a.k[w] = k[w];
        a.k2[w] = k2[w];
        a.out[w] = (double*)out[w];
        a.scale[w] = coef[w];
    }
    const unsigned blocks = (unsigned)((a.n_near + 3) / 4);
    const bool helm = op->kernel == BEM_KERNEL_HELMHOLTZ;
    if (helm && nk == 2)
        near_calderon_kernel<true, 2><<<blocks, 128, 0, s>>>(a);
    else if (helm)
        near_calderon_kernel<true, 1><<<blocks, 128, 0, s>>>(a);
    else if (nk == 2)
        near_calderon_kernel<false, 2><<<blocks, 128, 0, s>>>(a);
    else
        near_calderon_kernel<false, 1><<<blocks, 128, 0, s>>>(a);
    ctx->launches++;
    return bem_check_cuda(ctx, cudaGetLastError(), "near_calderon_kernel launch");
}
