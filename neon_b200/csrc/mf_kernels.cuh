// mf_kernels.cuh -- the setup of the matrix-free tangent product (included by elements.cu, which
// owns the shape-function tables); the product itself and the PCG around it are in mf_cg.cu.
//
// With G = sum_b v_b (x) L_b the element force of node a is (the product the assembled blocks
//   K_ab = s[lam' La(x)Lb + mu'((La.Lb) I + Lb(x)La) + b (N La)(x)(N Lb)] + s (La.sigma.Lb) I
// give) y_a = s [lam' tr(G) La + mu' (G + G^T) La + b (N:G) N La + (Da eps(G)) La + G sigma La].
#pragma once

// Setup from the stored FP64 outputs of the last MODE_STORE pass (A.u = its displacement):
//   md[c/4][e][c%4]  = (float)(x_a - x_0)_k, c = 3a + k (FP32 operator only; null for FP64)
//   mc (MfCoef)      = s lam', s mu' | finite strain: then s sigma (6)
//                  | Langevin / non-affine microsphere: then s Da (21, packed upper triangle)
//                  | J2: mu', elastic; -mu' and m = sqrt(-b) N (its 11 22 23 13 12 components: N is
//                    deviatoric, so m_33 = -m_11 - m_22), plastic.  The J2 tangent is
//                    lam' I(x)I + 2 mu' I + b N(x)N with lam' = K - 2 mu'/3, and at a plastic point
//                    of a hardening material b < 0 < mu', so b N(x)N = -m(x)m.  The point weight
//                    s = w det J comes from the element's own geometry at apply time.  Six numbers
//                    per point instead of nine, one at an elastic point.  A softening material
//                    leaves that range (b > 0 where the yield stress of the last state is
//                    negative, mu' < 0 where the present one is): such a point stores
//                    -kOddPoint, N, mu' and b, and leaves this setup's number in *odd_setup.
//   de[3a+i][e]      = element contribution to K_(3a+i, 3a+i)
template <int NPE, int MODEL, typename R>
__global__ void __launch_bounds__(64) k_mf_setup(ElementArgs A, float* __restrict__ md,
                                                 R* __restrict__ mc, double* __restrict__ de,
                                                 unsigned* odd_setup, unsigned setup) {
    using T = Topo<NPE>;
    constexpr int NQ = T::NQ, G = T::G, EPC = T::EPC;
    constexpr bool kFinite = (MODEL == MODEL_NH || MODEL == MODEL_MS || model_aniso(MODEL));
    constexpr bool kJ2 = (MODEL == MODEL_J2);
    constexpr bool kAniso = model_aniso(MODEL);
    __shared__ double sx[EPC][NPE][3];
    __shared__ double sdN[NQ][NPE][3];
    __shared__ double sD[EPC][NQ][NPE * 3];
    const int tid = threadIdx.x;
    const int le = tid / G;
    const int lane = tid % G;
    const long long e = (long long)blockIdx.x * EPC + le, E = A.E;
    const bool valid = e < E;
    for (int i = tid; i < NQ * NPE * 3; i += blockDim.x)
        (&sdN[0][0][0])[i] = (NPE == 8) ? c_dN_hex8[i] : c_dN_tet4[i];
#pragma unroll
    for (int j = 0; j < (NPE + G - 1) / G; ++j) {
        const int a = lane + j * G;
        if (a < NPE && valid) {
            const int nd = A.conn[e * NPE + a];
#pragma unroll
            for (int k = 0; k < 3; ++k) sx[le][a][k] = A.u[3ll * nd + k] + A.X[3ll * nd + k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < (NPE + G - 1) / G; ++j) {
        const int a = lane + j * G;
        if (a < NPE && valid && md)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int c = 3 * a + k;
                md[((c / 4) * E + e) * 4 + c % 4] = (float)(sx[le][a][k] - sx[le][0][k]);
            }
    }
    for (int l = lane; l < NQ; l += G) {
        if (!valid) break;
        const double w = (NPE == 8) ? c_w_hex8[l] : (1.0 / 6.0);
        const long long q = e * NQ + l;
        const long long n = A.nqp;
        constexpr int NEAR = MfCoef<MODEL>::NEAR;
        R* near = mc + q * NEAR;
        [[maybe_unused]] R* far = mc + n * NEAR + q;
        double Fc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int a = 0; a < NPE; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int k = 0; k < 3; ++k) Fc[i * 3 + k] += sx[le][a][i] * sdN[l][a][k];
        double Ji[9];
        inv3(Fc, Ji);
        const double s = w * det3(Fc);
        const double lam = A.dpar[0 * n + q], mu = A.dpar[1 * n + q];
        double b = 0.0, N6[6] = {0, 0, 0, 0, 0, 0}, sg[6] = {0, 0, 0, 0, 0, 0};
        if constexpr (kJ2) {
            b = A.dpar[2 * n + q];
#pragma unroll
            for (int c = 0; c < 6; ++c) N6[c] = A.dpar[(3 + c) * n + q];
            const R mu_r = (R)mu;
            const bool plastic = b != 0.0;
            // what the short form cannot hold: signs of their own, NaN at a plastic point
            const bool odd = plastic ? !(b < 0.0 && mu_r > kOddPoint<R>) : mu_r < (R)0;
            const double f = odd ? 1.0 : (plastic ? sqrt(-b) : 0.0);
            near[0] = odd ? -kOddPoint<R> : (plastic ? -mu_r : mu_r);
            far[0 * n] = (R)(f * N6[0]);
            far[1 * n] = (R)(f * N6[1]);
            far[2 * n] = (R)(f * N6[3]);
            far[3 * n] = (R)(f * N6[4]);
            far[4 * n] = (R)(f * N6[5]);
            if (odd) {
                far[5 * n] = mu_r;
                far[6 * n] = (R)b;
                *(volatile unsigned*)odd_setup = setup;
            }
        } else {
            near[0] = (R)(s * lam);
            near[1] = (R)(s * mu);
        }
        if constexpr (kFinite) {
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                sg[c] = A.sig[c * n + q];
                near[2 + c] = (R)(s * sg[c]);
            }
        }
        double Da[kAniso ? 21 : 1];
        if constexpr (kAniso) {
#pragma unroll
            for (int c = 0; c < 21; ++c) {
                Da[c] = A.dpar[(3 + c) * n + q];
                far[c * n] = (R)(s * Da[c]);
            }
        }
#pragma unroll
        for (int a = 0; a < NPE; ++a) {
            double La[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                La[k] = sdN[l][a][0] * Ji[0 * 3 + k] + sdN[l][a][1] * Ji[1 * 3 + k] +
                        sdN[l][a][2] * Ji[2 * 3 + k];
            const double LL = La[0] * La[0] + La[1] * La[1] + La[2] * La[2];
            double nl[3] = {0, 0, 0};
            if constexpr (kJ2) {
                nl[0] = N6[0] * La[0] + N6[5] * La[1] + N6[4] * La[2];
                nl[1] = N6[5] * La[0] + N6[1] * La[1] + N6[3] * La[2];
                nl[2] = N6[4] * La[0] + N6[3] * La[1] + N6[2] * La[2];
            }
            double geo = 0.0;
            if constexpr (kFinite)
                geo = sg[0] * La[0] * La[0] + sg[1] * La[1] * La[1] + sg[2] * La[2] * La[2] +
                      2.0 * (sg[3] * La[1] * La[2] + sg[4] * La[0] * La[2] + sg[5] * La[0] * La[1]);
            double ka[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            if constexpr (kAniso) aniso_block(Da, La, La, ka);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                sD[le][l][3 * a + i] = s * (lam * La[i] * La[i] + mu * (LL + La[i] * La[i]) +
                                            b * nl[i] * nl[i] + geo + ka[4 * i]);
        }
    }
    __syncthreads();
    if (!valid) return;
#pragma unroll
    for (int j = 0; j < (NPE + G - 1) / G; ++j) {
        const int a = lane + j * G;
        if (a < NPE)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                double t = 0.0;
#pragma unroll
                for (int l = 0; l < NQ; ++l) t += sD[le][l][3 * a + i];
                de[(3 * a + i) * E + e] = t;
            }
    }
}

