// mf_point.cuh -- the matrix-free tangent at one quadrature point, in FP32 (the mixed-precision
// PCG) or FP64.
#pragma once

#include <cfloat>

#include "nb2_internal.cuh"

namespace nb2 {

// r = m^-1; returns det m
template <typename R>
__device__ __forceinline__ R inv3r(const R* m, R* r) {
    const R c00 = m[4] * m[8] - m[5] * m[7];
    const R c10 = m[7] * m[2] - m[8] * m[1];
    const R c20 = m[1] * m[5] - m[2] * m[4];
    const R det = c00 * m[0] + c10 * m[3] + c20 * m[6];
    const R id = (R)1 / det;
    r[0] = c00 * id;
    r[1] = c10 * id;
    r[2] = c20 * id;
    r[3] = (m[5] * m[6] - m[3] * m[8]) * id;
    r[4] = (m[8] * m[0] - m[6] * m[2]) * id;
    r[5] = (m[2] * m[3] - m[0] * m[5]) * id;
    r[6] = (m[3] * m[7] - m[4] * m[6]) * id;
    r[7] = (m[6] * m[1] - m[7] * m[0]) * id;
    r[8] = (m[0] * m[4] - m[1] * m[3]) * id;
    return det;
}

// sigma_a = Da eps with eps the engineering strain of the gradient G (row-major 3x3); returns
// the symmetric stress in kinetic Voigt order
template <typename Real, typename DaT>
__device__ __forceinline__ void aniso_stress(const DaT* Da, const Real* G, Real* sa) {
    const Real eps[6] = {G[0], G[4], G[8], G[5] + G[7], G[2] + G[6], G[1] + G[3]};
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        Real t = (Real)0;
#pragma unroll
        for (int w = 0; w < 6; ++w) t += (Real)Da[sym6(v, w)] * eps[w];
        sa[v] = t;
    }
}

// J2 as the product sees it where a point may leave the hardening range (k_mf_setup).  FP64 always runs
// this variant.  In FP32, where eight unrolled points more of code cost 1.8% of the product (142.4 ->
// 144.9 us per iteration at 100^3), it runs only when the setup met such a point.
constexpr int MODEL_J2S = 6;
constexpr bool model_j2(int model) { return model == MODEL_J2 || model == MODEL_J2S; }

// Coefficients of a quadrature point: KC numbers, of which the product always reads the first NEAR;
// those of an element's points lie together, [element][point][NEAR], and the others (J2: only a
// plastic point has them, and the last two only one outside the hardening range; the anisotropic
// tangent) behind all of these, [coefficient][element][point].
template <int MODEL>
struct MfCoef {
    static constexpr int KC =
        model_j2(MODEL) ? 8 : ((MODEL == MODEL_LE) ? 2 : (model_aniso(MODEL) ? 8 + 21 : 8));
    static constexpr int NEAR = model_j2(MODEL) ? 1 : ((MODEL == MODEL_LE) ? 2 : 8);
};

// Marks a J2 point whose mu' and b stand behind its other coefficients: the smallest normal number, so
// that as mu' it adds nothing and only the branch of the plastic points has to look for it (an infinity,
// looked for at every point, cost 2.4% of an FP64 J2 solve at 100^3; this costs nothing there)
template <typename R>
constexpr R kOddPoint = sizeof(R) == 4 ? (R)FLT_MIN : (R)DBL_MIN;

// P = S J^-T at one point (J and Gx: gradients of the positions and the input in the reference
// element, in the same scaling; near: the point's first NEAR coefficients; far: its others, st
// apart).  J2 only: kdet turns
// det J into the point weight s (w times the determinant of the true Jacobian), Kb is the bulk
// modulus.
template <int MODEL, typename R>
__device__ __forceinline__ void point_flux(const R* J, const R* Gx, const R* near,
                                           const R* __restrict__ far, long long st, R kdet, R Kb, R* Pm) {
    constexpr bool kFinite = (MODEL == MODEL_NH || MODEL == MODEL_MS || model_aniso(MODEL));
    constexpr bool kJ2 = model_j2(MODEL);
    R Ji[9];
    const R det = inv3r(J, Ji);
    R G[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            G[i * 3 + k] = Gx[i * 3 + 0] * Ji[0 * 3 + k] + Gx[i * 3 + 1] * Ji[1 * 3 + k] +
                           Gx[i * 3 + 2] * Ji[2 * 3 + k];
    R cl, cm, c0 = (R)0, sw = (R)0;
    if constexpr (kJ2) {
        c0 = near[0];
        const R mu = (c0 < (R)0 ? -c0 : c0);
        sw = det * kdet;
        cm = sw * mu;
        cl = sw * (Kb - ((R)2 / (R)3) * mu);
    } else {
        cl = near[0];
        cm = near[1];
    }
    const R ltr = cl * (G[0] + G[4] + G[8]);
    R S[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            S[i * 3 + k] = cm * (G[i * 3 + k] + G[k * 3 + i]) + (i == k ? ltr : (R)0);
    if constexpr (kJ2) {
        if (c0 < (R)0) {  // plastic point: S -= s (m:G) m, or += s b (N:G) N
            R bw = -sw;
            // softening: the terms of mu', which are not in S yet, and b
            if (MODEL == MODEL_J2S && __builtin_expect(c0 == -kOddPoint<R>, 0)) {
                const R mw = sw * far[5 * st];
                const R mtr = (R)(-2.0 / 3.0) * mw * (G[0] + G[4] + G[8]);
                bw = sw * far[6 * st];
                S[0] += (R)2 * mw * G[0] + mtr;
                S[4] += (R)2 * mw * G[4] + mtr;
                S[8] += (R)2 * mw * G[8] + mtr;
                const R s3 = mw * (G[5] + G[7]), s4 = mw * (G[2] + G[6]), s5 = mw * (G[1] + G[3]);
                S[5] += s3; S[7] += s3;
                S[2] += s4; S[6] += s4;
                S[1] += s5; S[3] += s5;
            }
            const R m0 = far[0], m1 = far[st], m3 = far[2 * st], m4 = far[3 * st],
                    m5 = far[4 * st];
            const R m2 = -(m0 + m1);
            const R bN = bw * (m0 * G[0] + m1 * G[4] + m2 * G[8] + m3 * (G[5] + G[7]) +
                                    m4 * (G[2] + G[6]) + m5 * (G[1] + G[3]));
            // m symmetric (11 22 33 23 13 12)
            S[0] += bN * m0; S[4] += bN * m1; S[8] += bN * m2;
            S[5] += bN * m3; S[7] += bN * m3;
            S[2] += bN * m4; S[6] += bN * m4;
            S[1] += bN * m5; S[3] += bN * m5;
        }
    }
    if constexpr (model_aniso(MODEL)) {
        R Da[21], sa[6];
#pragma unroll
        for (int c = 0; c < 21; ++c) Da[c] = far[c * st];
        aniso_stress(Da, G, sa);
        S[0] += sa[0]; S[4] += sa[1]; S[8] += sa[2];
        S[5] += sa[3]; S[7] += sa[3];
        S[2] += sa[4]; S[6] += sa[4];
        S[1] += sa[5]; S[3] += sa[5];
    }
    if constexpr (kFinite) {
        R sg[9];
        sg[0] = near[2]; sg[4] = near[3]; sg[8] = near[4];
        sg[5] = sg[7] = near[5];
        sg[2] = sg[6] = near[6];
        sg[1] = sg[3] = near[7];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                S[i * 3 + k] += G[i * 3 + 0] * sg[0 * 3 + k] + G[i * 3 + 1] * sg[1 * 3 + k] +
                                G[i * 3 + 2] * sg[2 * 3 + k];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            Pm[i * 3 + k] = S[i * 3 + 0] * Ji[k * 3 + 0] + S[i * 3 + 1] * Ji[k * 3 + 1] +
                            S[i * 3 + 2] * Ji[k * 3 + 2];
}

}  // namespace nb2
