// Sauter-Schwab quadrature points of the near-field panel pairs (coincident,
// common-edge, common-vertex), shared by the assembly kernels and the shape
// adjoint.  For one 4D Gauss point (xsi, eta1, eta2, eta3) of the collapsed
// 4-cube with product weight `weight` (Gauss weights x 2A_x x 2A_y), every
// region of the relation calls
//   add(r1x, r2x, r1y, r2y, w)
// with the reference-triangle parameters of the point on each panel and the
// region's weight (Duffy Jacobian included).  The maps follow
// single_layer_3d.py:178-367 and m_mats_coincide (BEM_manager.py:141-165).
// The coincide rule evaluates each of its three regions a second time with the
// kernel's arguments swapped; that twin is left to the caller, since it needs
// no new evaluation: the same value for a kernel of r alone and the opposite
// one for a normal derivative, with the bases of both sides exchanged
// (corrected rule) or, as the reference has them, at the same parameters
// (`quirk`).
#pragma once

#include "bem_internal.cuh"

template <class F>
__device__ __forceinline__ void near_points(int rel, double xsi, double eta1, double eta2, double eta3, double weight,
                                            F&& add) {
    if (rel == REL_COINCIDE) {
        const double w = weight * (xsi * xsi * xsi * eta1 * eta1 * eta2);
        const double w0 = xsi, w1 = xsi * eta1, w2 = xsi * eta1 * eta2, w3 = xsi * eta1 * eta2 * eta3;
        // m_mats_coincide (BEM_manager.py:141-165) applied to w
#pragma unroll 1
        for (int m = 0; m < 3; ++m) {
            const double z0 = m == 2 ? w0 - w3 : w0;
            const double z1 = m == 0 ? w0 - w1 + w2 : (m == 1 ? w1 - w2 + w3 : w1 - w3);
            const double z2 = m == 0 ? w3 : (m == 1 ? w2 : -w3);
            const double z3 = m == 0 ? w2 : (m == 1 ? w3 : w2 - w3);
            add(z0, z1, z0 - z2, z1 - z3, w);
        }
    } else if (rel == REL_VERTEX) {
        const double w = weight * (xsi * xsi * xsi * eta2);
        const double p1 = xsi, p2 = xsi * eta1, q1 = xsi * eta2, q2 = xsi * eta2 * eta3;
#pragma unroll 1
        for (int m = 0; m < 2; ++m) add(m ? q1 : p1, m ? q2 : p2, m ? p1 : q1, m ? p2 : q2, w);
    } else {  // REL_EDGE
        const double jac1 = xsi * xsi * xsi * eta1 * eta1;
        const double jac = jac1 * eta2;
#pragma unroll 1
        for (int m = 0; m < 5; ++m) {
            double w0, w1, w2, w3;
            if (m == 0) {
                w0 = xsi; w1 = -xsi * eta1 * eta2; w2 = xsi * eta1 * (1.0 - eta2); w3 = xsi * eta1 * eta3;
            } else if (m == 1) {
                w0 = xsi; w1 = -xsi * eta1 * eta2 * eta3; w2 = xsi * eta1 * eta2 * (1.0 - eta3); w3 = xsi * eta1;
            } else if (m == 2) {
                w0 = xsi * (1.0 - eta1 * eta2); w1 = xsi * eta1 * eta2; w2 = xsi * eta1 * eta2 * eta3;
                w3 = xsi * eta1 * (1.0 - eta2);
            } else if (m == 3) {
                w0 = xsi * (1.0 - eta1 * eta2 * eta3); w1 = xsi * eta1 * eta2 * eta3; w2 = xsi * eta1;
                w3 = xsi * eta1 * eta2 * (1.0 - eta3);
            } else {
                w0 = xsi * (1.0 - eta1 * eta2 * eta3); w1 = xsi * eta1 * eta2 * eta3; w2 = xsi * eta1 * eta2;
                w3 = xsi * eta1 * (1.0 - eta2 * eta3);
            }
            add(w0, w3, w0 + w1, w2, weight * (m == 0 ? jac1 : jac));
        }
    }
}

// The Gauss points p = lane, lane + 32, ... of Q^4, as base-Q digits advanced
// without divisions.
struct NearDigits {
    int ix, iy, iz, iw, s0, s1, s2, s3;
    __device__ __forceinline__ void start(int lane, int Q) {
        iw = lane % Q;
        iz = (lane / Q) % Q;
        iy = (lane / (Q * Q)) % Q;
        ix = lane / (Q * Q * Q);
        s0 = 32 % Q;
        s1 = (32 / Q) % Q;
        s2 = (32 / (Q * Q)) % Q;
        s3 = 32 / (Q * Q * Q);
    }
    __device__ __forceinline__ void next(int Q) {
        iw += s0;
        int c = iw >= Q;
        iw -= c ? Q : 0;
        iz += s1 + c;
        c = iz >= Q;
        iz -= c ? Q : 0;
        iy += s2 + c;
        c = iy >= Q;
        iy -= c ? Q : 0;
        ix += s3 + c;
    }
};
