// mf_cg.cu -- the matrix-free tangent product in FP32 and FP64 and the Jacobi-PCG on it.
//
// Reference: conjugate_gradient::solve (linear_solver.cpp:67-109) on the assembled matrix.  The
// assembled K of a hex8 mesh costs 27 blocks x 76 B = 2.1 KB per node and SpMV in FP64, and large
// solves are bound by reading it (0.45 ms per iteration at 100^3, 0.84 of the HBM rate).  Applied
// element by element the same operator needs per element: the connectivity, node positions (FP64:
// gathered; FP32: 84 B relative to the element's first node, differences taken in FP64), per
// quadrature point the tangent coefficients (J2: 1 at an elastic point, 6 at a
// plastic one; linear elasticity 2; finite strain 8), and the input and output vectors.
//
// One CG iteration is three kernels, each started early by programmatic dependent launch (hex8):
//   k_mf_apply   one thread per element, everything in registers: gathers p = z + beta p of its nodes,
//                forms y_e = K_e p_e, adds the half of it that belongs to the next element's nodes
//                there (neighbouring lanes, where the connectivity says they are neighbours: all of a
//                structured mesh) and writes one product per remaining element node;
//   k_mf_gather  per node: q = sum of its products (4 instead of 8 inside a structured mesh), p updated
//                in place, p.q -> alpha;
//   k_mf_xr      x += alpha p, r -= alpha q, z = D^-1 r, r.r and r.z -> stop test, beta.
// (A variant in which a CTA adds the products of 128 elements in shared memory, one partial sum per
// node it touches, halved the products again but took 142 us against 82 for k_mf_apply at 100^3 in
// FP32: its barriers and list reads leave too little in flight at 16 warps per SM.)
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <string>

#include <thrust/device_ptr.h>
#include <thrust/execution_policy.h>
#include <thrust/sort.h>

#include "mf_cg.cuh"
#include "mf_point.cuh"
#include "reduce.cuh"

namespace nb2 {

namespace {

// threads of an element block: a hex8 thread runs long, so small blocks fill the last wave better
template <int NPE>
constexpr int kThreads = NPE == 8 ? 64 : 128;
constexpr int kIterations = 32;  // CG iterations per captured graph

// ---------------------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------------------
// Whether hex8 lane t's face nodes 1, 2, 5, 6 are the nodes 0, 3, 4, 7 of lane t + 1 (one bit each):
// their products are then added there
__device__ __forceinline__ unsigned merged_faces(const int (&nd)[8], bool valid) {
    const unsigned on = __ballot_sync(0xffffffffu, valid);
    const int lane = threadIdx.x & 31;
    const int n0 = __shfl_down_sync(0xffffffffu, nd[0], 1), n3 = __shfl_down_sync(0xffffffffu, nd[3], 1);
    const int n4 = __shfl_down_sync(0xffffffffu, nd[4], 1), n7 = __shfl_down_sync(0xffffffffu, nd[7], 1);
    if (!valid || lane == 31 || !((on >> (lane + 1)) & 1u)) return 0u;
    return (nd[1] == n0 ? 1u : 0u) | (nd[2] == n3 ? 2u : 0u) | (nd[5] == n4 ? 4u : 0u) |
           (nd[6] == n7 ? 8u : 0u);
}

// key[a E + e] = the node that product (a, e) is added to, N where it is merged into the next lane's
template <int NPE>
__global__ void k_product_nodes(int E, int N, const int* __restrict__ conn, int* __restrict__ key,
                                int* __restrict__ idx) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = e < E;
    int nd[NPE];
#pragma unroll
    for (int a = 0; a < NPE; ++a) nd[a] = valid ? conn[e * NPE + a] : -1;
    unsigned gone = 0;
    if constexpr (NPE == 8) {
        const unsigned m = merged_faces(nd, valid);
        gone = ((m & 1u) << 1) | ((m & 2u) << 1) | ((m & 4u) << 3) | ((m & 8u) << 3);
    }
    if (!valid) return;
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
        key[(long long)a * E + e] = (gone >> a) & 1u ? N : nd[a];
        idx[(long long)a * E + e] = (int)(a * (long long)E + e);
    }
}

// products of every node, in ascending order: the first four (-1 where there are fewer), and the
// place in the sorted list, from which a node with more reads on
__global__ void k_node_products(const int* __restrict__ keys, const int* __restrict__ idx,
                                long long m, int N, int4* __restrict__ first,
                                int* __restrict__ ptr) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a > N) return;
    long long lo = 0, hi = m;
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (keys[mid] < a) lo = mid + 1; else hi = mid;
    }
    ptr[a] = (int)lo;
    if (a == N) return;
    int f[4];
    for (int k = 0; k < 4; ++k) f[k] = lo + k < m && keys[lo + k] == a ? idx[lo + k] : -1;
    first[a] = make_int4(f[0], f[1], f[2], f[3]);
}

// ---------------------------------------------------------------------------------------
// operator
// ---------------------------------------------------------------------------------------
// z and p, the vectors every element gathers: three numbers per node, in FP32 padded to four so that
// one 16-byte load brings a node (16 loads per element in place of 48)
template <typename R>
constexpr int kNode = sizeof(R) == 4 ? 4 : 3;
// place of unknown i in a node vector
template <typename R>
__device__ __forceinline__ long long node_at(long long i) {
    return kNode<R> == 3 ? i : i + i / 3;
}
__device__ __forceinline__ void load_node(const float* v, int a, float (&t)[3]) {
    const float4 f = reinterpret_cast<const float4*>(v)[a];
    t[0] = f.x;
    t[1] = f.y;
    t[2] = f.z;
}
__device__ __forceinline__ void load_node(const double* v, int a, double (&t)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) t[k] = v[3ll * a + k];
}
// the same, in program order: a load that the compiler may not move behind the test of `done`
__device__ __forceinline__ void load_node_now(const float* v, int a, float (&t)[3]) {
    [[maybe_unused]] float pad;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(t[0]), "=f"(t[1]), "=f"(t[2]), "=f"(pad)
                 : "l"(v + 4ll * a)
                 : "memory");
}
__device__ __forceinline__ void load_node_now(const double* v, int a, double (&t)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(t[k]) : "l"(v + 3ll * a + k) : "memory");
}
__device__ __forceinline__ void store_node(float* v, int a, const float (&t)[3]) {
    reinterpret_cast<float4*>(v)[a] = make_float4(t[0], t[1], t[2], 0.0f);
}
__device__ __forceinline__ void store_node(double* v, int a, const double (&t)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[3ll * a + k] = t[k];
}

template <typename R>
struct MfView {
    int E;
    const int* conn;
    const float* md;   // FP32: [3 NPE / 4][E][4], the coordinates of the nodes one after another
    const R* mc;       // see k_mf_setup
    const double* x;   // FP64: [N][3]
    R* ye;             // [NPE][E][3]
};

// modal coefficients (sum_a s_a(m) u_a) of a hex8 nodal 3-vector field, nodes in the reference's
// corner order; M[0..6] = xi, eta, zeta, xi eta, xi zeta, eta zeta, xi eta zeta (mode 1 unused)
template <typename R>
__device__ __forceinline__ void hex8_modes(const R (&u)[8][3], R (&M)[7][3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const R p0 = u[1][c] + u[0][c], m0 = u[1][c] - u[0][c];
        const R p1 = u[2][c] + u[3][c], m1 = u[2][c] - u[3][c];
        const R p2 = u[5][c] + u[4][c], m2 = u[5][c] - u[4][c];
        const R p3 = u[6][c] + u[7][c], m3 = u[6][c] - u[7][c];
        const R q0 = p1 + p0, q1 = p1 - p0, q2 = p3 + p2, q3 = p3 - p2;
        const R r0 = m1 + m0, r1 = m1 - m0, r2 = m3 + m2, r3 = m3 - m2;
        M[0][c] = r2 + r0;  // xi
        M[1][c] = q3 + q1;  // eta
        M[2][c] = q2 - q0;  // zeta
        M[3][c] = r3 + r1;  // xi eta
        M[4][c] = r2 - r0;  // xi zeta
        M[5][c] = q3 - q1;  // eta zeta
        M[6][c] = r3 - r1;  // xi eta zeta
    }
}

// y = K_e v for one element with node positions (or positions relative to the first node) d.  hex8
// works in the element's trilinear modes (1, xi, eta, zeta, xi eta, xi zeta, eta zeta, xi eta zeta):
// a +/- butterfly turns the 8 nodal vectors into modal coefficients, the reference gradient at a
// point is then 4 terms per entry, and the outputs are accumulated per mode and turned back into
// nodal forces once -- about 30% fewer FMAs than nodal sums at every point.  (The factor 1/8 of
// the trilinear shape functions cancels: J and Gx carry it alike, and P dN_a carries 8 * 1/8.)
// Per point, with J = sum_a d_a (x) dN_a, Gx = sum_a v_a (x) dN_a:
//   G = Gx J^-1,  S = s[lam' tr(G) I + mu' (G + G^T) + b (N:G) N + G sigma],  P = S J^-T,
//   y_a += P dN_a                     (y_a = S L_a with L_a = J^-T dN_a, never formed)
// mc: the element's near coefficients, far: its first point's others (MfCoef)
template <int NEAR>
__device__ __forceinline__ void load_near(const float* __restrict__ p, float (&c)[NEAR]) {
    if constexpr (NEAR % 4 == 0) {
#pragma unroll
        for (int k = 0; k < NEAR; k += 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + k);
            c[k] = t.x;
            c[k + 1] = t.y;
            c[k + 2] = t.z;
            c[k + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < NEAR; ++k) c[k] = p[k];
    }
}
template <int NEAR>
__device__ __forceinline__ void load_near(const double* __restrict__ p, double (&c)[NEAR]) {
    if constexpr (NEAR % 2 == 0) {
#pragma unroll
        for (int k = 0; k < NEAR; k += 2) {
            const double2 t = *reinterpret_cast<const double2*>(p + k);
            c[k] = t.x;
            c[k + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < NEAR; ++k) c[k] = p[k];
    }
}

template <int NPE, int MODEL, typename R>
__device__ __forceinline__ void element_product(const R (&d)[NPE][3], const R (&v)[NPE][3],
                                                const R* __restrict__ mc,
                                                const R* __restrict__ far, long long nqp, R Kb,
                                                R (&y)[NPE][3]) {
    using C = MfCoef<MODEL>;
    if constexpr (NPE == 8) {
        R Md[7][3], Mv[7][3], Y[7][3];
        hex8_modes(d, Md);
        hex8_modes(v, Mv);
#pragma unroll
        for (int m = 0; m < 7; ++m) Y[m][0] = Y[m][1] = Y[m][2] = (R)0;
        constexpr R g = (R)0.57735026918962576;  // 1/sqrt(3): the 2-point Gauss abscissa
        // Points in z, x, eta order.  With u = sum_m u_m m the reference gradient is
        //   d/dxi = (M0 + z M4) + eta (M3 + z M6),  d/deta = (M1 + z M5) + xi (M3 + z M6),
        //   d/dzeta = (M2 + x M4) + eta (M5 + x M6),
        // whose brackets are shared by the points of a layer or of an edge: 90 FMAs a field instead
        // of 216; the outputs are summed the same way, transposed
#pragma unroll
        for (int iz = 0; iz < 2; ++iz) {
            const R z = iz ? g : -g;
            R Jx[2][3], Gx0[2][3], ja[3], jb[3], ga[3], gb[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const R j0 = Md[0][c] + z * Md[4][c], g0 = Mv[0][c] + z * Mv[4][c];
                ja[c] = Md[1][c] + z * Md[5][c];
                jb[c] = Md[3][c] + z * Md[6][c];
                ga[c] = Mv[1][c] + z * Mv[5][c];
                gb[c] = Mv[3][c] + z * Mv[6][c];
                Jx[0][c] = j0 - g * jb[c];
                Jx[1][c] = j0 + g * jb[c];
                Gx0[0][c] = g0 - g * gb[c];
                Gx0[1][c] = g0 + g * gb[c];
            }
            R S0[2][3], S1[3], S1x[3];
#pragma unroll
            for (int ix = 0; ix < 2; ++ix) {
                const R x = ix ? g : -g;
                R J[9], G[9], jc[3], jd[3], gc[3], gd[3], P0[9], P1[9];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    J[3 * c + 1] = ja[c] + x * jb[c];
                    G[3 * c + 1] = ga[c] + x * gb[c];
                    jc[c] = Md[2][c] + x * Md[4][c];
                    jd[c] = Md[5][c] + x * Md[6][c];
                    gc[c] = Mv[2][c] + x * Mv[4][c];
                    gd[c] = Mv[5][c] + x * Mv[6][c];
                }
#pragma unroll
                for (int ie = 0; ie < 2; ++ie) {
                    const R e = ie ? g : -g;
                    // the reference's point numbers (hexahedron_quadrature.cpp order)
                    const int l = 4 * iz + (ie ? (ix ? 2 : 3) : (ix ? 1 : 0));
                    R near[C::NEAR];
                    load_near<C::NEAR>(mc + l * C::NEAR, near);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        J[3 * c] = Jx[ie][c];
                        G[3 * c] = Gx0[ie][c];
                        J[3 * c + 2] = jc[c] + e * jd[c];
                        G[3 * c + 2] = gc[c] + e * gd[c];
                    }
                    point_flux<MODEL>(J, G, near, far + l, nqp, (R)(1.0 / 512.0), Kb,
                                      ie ? P1 : P0);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const R t1 = P0[3 * c + 1] + P1[3 * c + 1];
                    const R u = P0[3 * c + 2] + P1[3 * c + 2], w = P1[3 * c + 2] - P0[3 * c + 2];
                    if (ix == 0) {
                        S0[0][c] = P0[3 * c];
                        S0[1][c] = P1[3 * c];
                        S1[c] = t1;
                        S1x[c] = -t1;
                    } else {
                        S0[0][c] += P0[3 * c];
                        S0[1][c] += P1[3 * c];
                        S1[c] += t1;
                        S1x[c] += t1;
                    }
                    Y[2][c] += u;
                    Y[4][c] += x * u;
                    Y[5][c] += g * w;
                    Y[6][c] += (x * g) * w;
                }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const R s0 = S0[0][c] + S0[1][c];
                const R t = g * ((S0[1][c] - S0[0][c]) + S1x[c]);
                Y[0][c] += s0;
                Y[4][c] += z * s0;
                Y[3][c] += t;
                Y[6][c] += z * t;
                Y[1][c] += S1[c];
                Y[5][c] += z * S1[c];
            }
        }
        // back to nodes: y_a = sum_m s_a(m) Y_m (transposed butterfly; mode 1 carries nothing)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const R a0_1 = -Y[2][c], a1_1 = Y[2][c];           // 1 -/+ zeta
            const R a0_e = Y[1][c] - Y[5][c], a1_e = Y[1][c] + Y[5][c];
            const R a0_x = Y[0][c] - Y[4][c], a1_x = Y[0][c] + Y[4][c];
            const R a0_xe = Y[3][c] - Y[6][c], a1_xe = Y[3][c] + Y[6][c];
            // z = 0 corners 0..3, z = 1 corners 4..7
            const R b00_1 = a0_1 - a0_e, b01_1 = a0_1 + a0_e;   // (y=0 / y=1, z=0)
            const R b00_x = a0_x - a0_xe, b01_x = a0_x + a0_xe;
            const R b10_1 = a1_1 - a1_e, b11_1 = a1_1 + a1_e;   // (y=0 / y=1, z=1)
            const R b10_x = a1_x - a1_xe, b11_x = a1_x + a1_xe;
            y[0][c] = b00_1 - b00_x;  // (x0 y0 z0)
            y[1][c] = b00_1 + b00_x;  // (x1 y0 z0)
            y[2][c] = b01_1 + b01_x;  // (x1 y1 z0)
            y[3][c] = b01_1 - b01_x;  // (x0 y1 z0)
            y[4][c] = b10_1 - b10_x;  // (x0 y0 z1)
            y[5][c] = b10_1 + b10_x;  // (x1 y0 z1)
            y[6][c] = b11_1 + b11_x;  // (x1 y1 z1)
            y[7][c] = b11_1 - b11_x;  // (x0 y1 z1)
        }
    } else {
        // tet4: dN = (e_x, e_y, e_z, -1 -1 -1)
        R J[9], Gx[9], P[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                J[i * 3 + k] = d[k][i] - d[3][i];
                Gx[i * 3 + k] = v[k][i] - v[3][i];
            }
        R near[C::NEAR];
        load_near<C::NEAR>(mc, near);
        point_flux<MODEL>(J, Gx, near, far, nqp, (R)(1.0 / 6.0), Kb, P);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int k = 0; k < 3; ++k) y[k][i] = P[i * 3 + k];
            y[3][i] = -(P[i * 3 + 0] + P[i * 3 + 1] + P[i * 3 + 2]);
        }
    }
}

// CTAs per SM that the registers are cut for (hex8: 64 threads each).  FP32: 8 (128 registers); J2, which
// needs the fewest, 10 (96, a few spilled): 141 against 145 us per iteration at 100^3, and 163 with 6;
// finite strain at 64^3 56 us with 8, 59 with 6, 61 with 10.  tet4 (128 threads each) waits for memory, so
// warps count: 10 (48 registers), 8 for the anisotropic models.  72^3 x 6 linear, neo-Hooke, Langevin: 113,
// 114, 140 us per iteration; 116, 117, 144 with 4 of 256 threads (56 to 72 registers).
template <int NPE, int MODEL, typename R>
constexpr int apply_blocks() {
    if (NPE == 4) return sizeof(R) == 8 ? 4 : (model_aniso(MODEL) ? 8 : 10);
    return sizeof(R) == 8 || model_aniso(MODEL) ? 4 : (MODEL == MODEL_J2 ? 10 : 8);
}

// ye = the element products of K (z + beta p) (p null: of K z); skipped once the CG scalars say done.
// What does not change between iterations is requested before the wait for the kernel ahead.  FP32
// is held by its 1.7 k instructions per element at 16 to 20 warps per SM, FP64 by the FP64 pipe
// (1.4 k operations per element, 64 per cycle and SM) at 8 warps.  Per iteration of J2 at 100^3:
// FP64 450 (assembled K) -> 216 us, FP32 156 -> 141 us.
template <int NPE, int MODEL, typename R>
__global__ void __launch_bounds__(kThreads<NPE>, apply_blocks<NPE, MODEL, R>())
    k_mf_apply(MfView<R> M, R Kb, const R* z, const R* p, const CgScalars* s) {
    pdl_next();
    const long long e = (long long)blockIdx.x * kThreads<NPE> + threadIdx.x, E = M.E;
    const bool valid = e < E;
    const long long el = valid ? e : E - 1;  // lanes past the end repeat the last element
    int nd[NPE];
    {
        const int4* c4 = reinterpret_cast<const int4*>(M.conn + el * NPE);
#pragma unroll
        for (int j = 0; j < NPE / 4; ++j) {
            const int4 t = c4[j];
            nd[4 * j] = t.x;
            nd[4 * j + 1] = t.y;
            nd[4 * j + 2] = t.z;
            nd[4 * j + 3] = t.w;
        }
    }
    R d[NPE][3];
    if constexpr (sizeof(R) == 4) {
        const float4* m4 = reinterpret_cast<const float4*>(M.md);
#pragma unroll
        for (int j = 0; j < 3 * NPE / 4; ++j) {
            const float4 t = m4[j * E + el];
            (&d[0][0])[4 * j] = t.x;
            (&d[0][0])[4 * j + 1] = t.y;
            (&d[0][0])[4 * j + 2] = t.z;
            (&d[0][0])[4 * j + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int a = 0; a < NPE; ++a)
#pragma unroll
            for (int k = 0; k < 3; ++k) d[a][k] = M.x[3ll * nd[a] + k];
    }
    pdl_wait();
    R v[NPE][3], y[NPE][3], beta = (R)0;
    int done = 0;
    if (s) {
        // through L1 (a volatile load is not): every warp reads this one line, and 50,000 of them
        // at one L2 slice took 9 of 42 us for tet4 at 64^3
        double b;
        asm volatile("ld.global.s32 %0, [%1];" : "=r"(done) : "l"(&s->done) : "memory");
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(b) : "l"(&s->beta) : "memory");
        beta = (R)b;
    }
#pragma unroll
    for (int a = 0; a < NPE; ++a) load_node_now(z, nd[a], v[a]);
    if (p) {
        R t[NPE][3];
#pragma unroll
        for (int a = 0; a < NPE; ++a) load_node_now(p, nd[a], t[a]);
        if (done) return;
#pragma unroll
        for (int a = 0; a < NPE; ++a)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[a][k] += beta * t[a][k];
    } else if (done) {
        return;
    }
    unsigned gone = 0;
    if constexpr (NPE == 8) gone = merged_faces(nd, valid);
    constexpr int NQ = NPE == 8 ? 8 : 1, NEAR = MfCoef<MODEL>::NEAR;
    element_product<NPE, MODEL>(d, v, M.mc + el * (NQ * NEAR), M.mc + E * (NQ * NEAR) + el * NQ,
                                E * NQ, Kb, y);
    if constexpr (NPE == 8) {
        // the products of the face shared with the previous lane arrive here
        constexpr int from[4] = {1, 2, 5, 6}, to[4] = {0, 3, 4, 7};
        const unsigned mine = __shfl_up_sync(0xffffffffu, gone, 1);
        const unsigned take = (threadIdx.x & 31) ? mine : 0u;
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const R got = __shfl_up_sync(0xffffffffu, y[from[f]][k], 1);
                if ((take >> f) & 1u) y[to[f]][k] += got;
            }
    }
    if (!valid) return;
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
        if constexpr (NPE == 8) {
            const int f = a == 1 ? 0 : (a == 2 ? 1 : (a == 5 ? 2 : (a == 6 ? 3 : -1)));
            if (f >= 0 && ((gone >> f) & 1u)) continue;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) M.ye[((long long)a * E + e) * 3 + k] = y[a][k];
    }
}

// ye = the element contributions to diag(K), added over merged faces like the products
template <int NPE>
__global__ void __launch_bounds__(kThreads<NPE>) k_mf_diag_products(int E, const int* __restrict__ conn,
                                                               const double* __restrict__ de,
                                                               double* __restrict__ ye) {
    const long long e = (long long)blockIdx.x * kThreads<NPE> + threadIdx.x;
    const bool valid = e < E;
    int nd[NPE];
    double y[NPE][3];
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
        nd[a] = valid ? conn[e * NPE + a] : -1;
#pragma unroll
        for (int k = 0; k < 3; ++k) y[a][k] = valid ? de[(long long)(3 * a + k) * E + e] : 0.0;
    }
    if constexpr (NPE == 8) {
        constexpr int from[4] = {1, 2, 5, 6}, to[4] = {0, 3, 4, 7};
        const unsigned gone = merged_faces(nd, valid);
        const unsigned mine = __shfl_up_sync(0xffffffffu, gone, 1);
        const unsigned take = (threadIdx.x & 31) ? mine : 0u;
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double got = __shfl_up_sync(0xffffffffu, y[from[f]][k], 1);
                if ((take >> f) & 1u) y[to[f]][k] += got;
            }
    }
    if (!valid) return;
#pragma unroll
    for (int a = 0; a < NPE; ++a)
#pragma unroll
        for (int k = 0; k < 3; ++k) ye[((long long)a * E + e) * 3 + k] = y[a][k];
}

// products of the nodes (MfPlan)
struct NodeSums {
    const int4* first;
    const int *ptr, *idx;
};

// hex8: the first four from one 16-byte load (all there are inside a structured mesh); tet4, with about
// 24 products a node, straight from the list
template <int NPE, typename R>
__device__ __forceinline__ void node_sum(int a, const NodeSums& S, const R* ye, R (&y)[3]) {
    if constexpr (NPE == 8) {
        const int4 f = S.first[a];
        const int j[4] = {f.x, f.y, f.z, f.w};
        R t[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) t[k][i] = j[k] >= 0 ? ye[3ll * j[k] + i] : (R)0;
#pragma unroll
        for (int i = 0; i < 3; ++i) y[i] = ((t[0][i] + t[1][i]) + t[2][i]) + t[3][i];
        if (f.w < 0) return;
    } else {
        y[0] = y[1] = y[2] = (R)0;
    }
    const int k1 = S.ptr[a + 1];
#pragma unroll 4
    for (int k = S.ptr[a] + (NPE == 8 ? 4 : 0); k < k1; ++k) {
        const long long j = 3ll * S.idx[k];
#pragma unroll
        for (int i = 0; i < 3; ++i) y[i] += ye[j + i];
    }
}

// Jacobi inverse (1 for a zero diagonal)
template <int NPE, typename X>
__global__ void k_mf_inv(int N, NodeSums S, const double* __restrict__ ye,
                         X* __restrict__ inv) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= N) return;
    double d[3];
    node_sum<NPE>(a, S, ye, d);
#pragma unroll
    for (int k = 0; k < 3; ++k) inv[3ll * a + k] = d[k] != 0.0 ? (X)(1.0 / d[k]) : (X)1;
}

// y = the node sums
template <int NPE, typename R>
__global__ void k_mf_sum(int N, NodeSums S, const R* __restrict__ ye, double* __restrict__ y) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= N) return;
    R t[3];
    node_sum<NPE>(a, S, ye, t);
#pragma unroll
    for (int k = 0; k < 3; ++k) y[3ll * a + k] = (double)t[k];
}

__global__ void k_mf_positions(long long n, const double* __restrict__ X,
                               const double* __restrict__ u, double* __restrict__ x) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        x[i] = u[i] + X[i];
}

// ---------------------------------------------------------------------------------------
// CG kernels
// ---------------------------------------------------------------------------------------
// tet4: p = z + beta p on its own.  A node has about 24 elements, each of which would gather z and p
// (hex8: 8; there the extra kernel costs more, 9 us at 100^3 in FP32)
__global__ void __launch_bounds__(kRedThreads) k_mf_p(int N, const float* z, float* p,
                                                      const CgScalars* s) {
    pdl_next();
    pdl_wait();
    if (s->done) return;
    const float beta = (float)s->beta;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += gridDim.x * blockDim.x) {
        float zn[3], pn[3];
        load_node(z, a, zn);
        load_node(p, a, pn);
#pragma unroll
        for (int k = 0; k < 3; ++k) pn[k] = zn[k] + beta * pn[k];
        store_node(p, a, pn);
    }
}

// q = K p (masked rows 0), p = z + beta p in place (hex8), p.q; the last block forms
// alpha = (r.z)/(p.q)
template <int NPE, typename R>
__global__ void __launch_bounds__(kRedThreads, NPE == 8 && sizeof(R) == 4 ? 8 : 4)
    k_mf_gather(int N, NodeSums S, const R* ye, const R* z, R* p, R* q,
                const unsigned char* __restrict__ mask, CgScalars* s, double* partials) {
    pdl_next();
    pdl_wait();
    if (s->done) return;
    const R beta = (R)s->beta;
    double dot[1] = {0.0};
    const int stride = gridDim.x * blockDim.x;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += stride) {
        const long long i = 3ll * a;
        R zn[3], pn[3], y[3];
        unsigned char m[3];
        load_node(p, a, pn);
        if constexpr (NPE == 8) {
            load_node(z, a, zn);
#pragma unroll
            for (int k = 0; k < 3; ++k) pn[k] = zn[k] + beta * pn[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) m[k] = mask[i + k];
        node_sum<NPE>(a, S, ye, y);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const R v = m[k] ? (R)0 : y[k];
            q[i + k] = v;
            dot[0] += (double)pn[k] * (double)v;
        }
        if constexpr (NPE == 8) store_node(p, a, pn);
    }
    if (block_partials<1>(dot, partials, &s->counter[0])) {
        double tot[1];
        final_sum<1>(partials, tot);
        if (threadIdx.x == 0) {
            s->pq = tot[0];
            s->alpha = s->abs_new / tot[0];
            // Eigen's CG carries on through p.Ap <= 0 (an indefinite tangent); only a
            // non-finite step size is a failure (neon: FE_INVALID -> computational_error)
            if (!isfinite(s->alpha)) {
                s->status = NB2_E_NAN;
                s->done = 1;
            }
            s->counter[0] = 0;
        }
    }
}

template <typename R>
__device__ __forceinline__ void xrz_one(R& x, R& r, R& z, R p, R q, R inv, R alpha,
                                        double (&acc)[2]) {
    x += alpha * p;
    r -= alpha * q;
    z = inv * r;
    acc[0] += (double)r * (double)r;
    acc[1] += (double)r * (double)z;
}

template <typename R>
__global__ void __launch_bounds__(kRedThreads) k_mf_xr(long long n, R* x, R* r, R* z, const R* p,
                                                       const R* q, const R* __restrict__ inv,
                                                       CgScalars* s, double* partials) {
    using V = typename Vec16<R>::T;
    constexpr int W = Vec16<R>::W;
    pdl_next();
    pdl_wait();
    if (s->done) return;
    const R alpha = (R)s->alpha;
    double acc[2] = {0.0, 0.0};
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long st = (long long)gridDim.x * blockDim.x;
    const long long nv = n / W;  // the context's own buffers: aligned
    for (long long j = t0; j < nv; j += st) {
        R xv[W], rv[W], zv[W], pv[W], qv[W], iv[W];
        *reinterpret_cast<V*>(xv) = reinterpret_cast<const V*>(x)[j];
        *reinterpret_cast<V*>(rv) = reinterpret_cast<const V*>(r)[j];
        *reinterpret_cast<V*>(qv) = reinterpret_cast<const V*>(q)[j];
        *reinterpret_cast<V*>(iv) = reinterpret_cast<const V*>(inv)[j];
        if constexpr (kNode<R> == 3) {
            *reinterpret_cast<V*>(pv) = reinterpret_cast<const V*>(p)[j];
        } else {
#pragma unroll
            for (int w = 0; w < W; ++w) pv[w] = p[node_at<R>(W * j + w)];
        }
#pragma unroll
        for (int w = 0; w < W; ++w) xrz_one(xv[w], rv[w], zv[w], pv[w], qv[w], iv[w], alpha, acc);
        reinterpret_cast<V*>(x)[j] = *reinterpret_cast<V*>(xv);
        reinterpret_cast<V*>(r)[j] = *reinterpret_cast<V*>(rv);
        if constexpr (kNode<R> == 3) {
            reinterpret_cast<V*>(z)[j] = *reinterpret_cast<V*>(zv);
        } else {
#pragma unroll
            for (int w = 0; w < W; ++w) z[node_at<R>(W * j + w)] = zv[w];
        }
    }
    for (long long i = nv * W + t0; i < n; i += st)
        xrz_one(x[i], r[i], z[node_at<R>(i)], p[node_at<R>(i)], q[i], inv[i], alpha, acc);
    if (block_partials<2>(acc, partials, &s->counter[1])) {
        double tot[2];
        final_sum<2>(partials, tot);
        if (threadIdx.x == 0) {
            s->rr = tot[0];
            if (tot[0] < s->threshold) {
                s->done = 1;
            } else if (tot[0] > s->rr_cap) {
                s->done = 1;
                s->status = NB2_E_CG_BREAKDOWN;
            } else {
                s->beta = tot[1] / s->abs_new;
                s->abs_new = tot[1];
                s->rz = tot[1];
                s->iterations += 1;
                if (s->iterations >= s->max_iterations) {
                    s->done = 1;
                    s->status = NB2_E_CG_MAXIT;
                }
            }
            if (!isfinite(tot[0])) {
                s->done = 1;
                s->status = NB2_E_NAN;
            }
            s->counter[1] = 0;
        }
    }
}

// x = 0, r = b, z = D^-1 r, p = 0 (the first direction is z + 0 p); b.b, r.r, r.z
template <typename R>
__global__ void __launch_bounds__(kRedThreads) k_mf_init(long long n, const double* __restrict__ b,
                                                         R* x, R* r, R* z, R* p, const R* inv,
                                                         CgScalars* s, double* partials,
                                                         double tol, int maxit) {
    double acc[3] = {0, 0, 0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const R bi = (R)b[i], zi = inv[i] * bi;
        const long long at = node_at<R>(i);
        x[i] = (R)0;
        r[i] = bi;
        z[at] = zi;
        p[at] = (R)0;
        acc[0] += b[i] * b[i];
        acc[1] += (double)bi * (double)bi;
        acc[2] += (double)bi * (double)zi;
    }
    if (block_partials<3>(acc, partials, &s->counter[2])) {
        double tot[3];
        final_sum<3>(partials, tot);
        if (threadIdx.x == 0) {
            s->rhs_norm2 = tot[0];
            s->threshold = fmax(tol * tol * tot[0], DBL_MIN);
            s->rr = tot[1];
            s->abs_new = tot[2];
            s->rz = tot[2];
            s->beta = 0.0;
            s->rr_cap = INFINITY;
            s->iterations = 0;
            s->max_iterations = maxit;
            s->status = 0;
            s->done = 0;
            if (tot[0] == 0.0) {
                s->done = 1;
                s->rr = 0.0;
            } else if (tot[1] < s->threshold) {
                s->done = 1;
            }
            s->counter[2] = 0;
        }
    }
}

// x64[i] += xs[i]; xs[i] = 0 (fold the FP32 increment into the FP64 iterate)
__global__ void k_fold(long long n, float* __restrict__ xs, double* __restrict__ x64) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        x64[i] += (double)xs[i];
        xs[i] = 0.0f;
    }
}

// r = b - y on free rows, 0 on masked rows; rs = (float) r, zs = D^-1 rs; r.r (FP64), rs.zs.  The
// cycle goes on with the replaced residual until it has fallen by delta (fresh: with p = zs): the
// last block sets the scalars, or leaves `done` set where the solve has ended.
__global__ void __launch_bounds__(kRedThreads) k_true_residual(
    long long n, const double* __restrict__ b, const double* __restrict__ y,
    const unsigned char* __restrict__ mask, const float* __restrict__ inv, float* __restrict__ rs,
    float* __restrict__ zs, CgScalars* s, double* partials, double thr, double delta, int fresh) {
    double acc[2] = {0.0, 0.0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double ri = mask[i] ? 0.0 : b[i] - y[i];
        const float rf = (float)ri, zf = inv[i] * rf;
        rs[i] = rf;
        zs[node_at<float>(i)] = zf;
        acc[0] += ri * ri;
        acc[1] += (double)rf * (double)zf;
    }
    if (block_partials<2>(acc, partials, &s->counter[3])) {
        double tot[2];
        final_sum<2>(partials, tot);
        if (threadIdx.x == 0) {
            // continue the recurrence with the replaced residual: beta = rz_new / rz_old
            s->beta = fresh ? 0.0 : tot[1] / s->abs_new;
            s->abs_new = tot[1];
            s->rz = tot[1];
            s->rr = tot[0];
            // a cycle whose FP32 recurrence r.r grows to this multiple of the replaced one has
            // diverged (CG residual norms are not monotone: a factor 1000 in the norm)
            s->rr_cap = 1e6 * tot[0];
            const bool stop = !isfinite(tot[0]) || tot[0] < thr ||
                              s->status == NB2_E_CG_MAXIT || s->iterations >= s->max_iterations;
            if (!stop) {
                s->threshold = fmax(thr, delta * delta * tot[0]);
                s->done = 0;
                s->status = 0;
            }
            s->counter[3] = 0;
        }
    }
}

// an FP32 node vector
__global__ void k_to_float(long long n, const double* __restrict__ a, float* __restrict__ b) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        b[node_at<float>(i)] = (float)a[i];
}

__global__ void k_copy_double(long long n, const double* __restrict__ a, double* __restrict__ b) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        b[i] = a[i];
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
unsigned vec_grid(long long n) { return (unsigned)std::min<long long>((n + 255) / 256, 148 * 8); }

template <typename R>
MfView<R> view(const nb2_ctx* c) {
    const MfPlan* P = c->mf;
    MfView<R> M;
    M.E = c->E;
    M.conn = c->conn;
    M.md = P->md;
    if constexpr (sizeof(R) == 4)
        M.mc = P->mc32;
    else
        M.mc = P->mc64;
    M.x = P->x;
    M.ye = reinterpret_cast<R*>(P->ye);
    return M;
}

NodeSums sums(const nb2_ctx* c) { return NodeSums{c->mf->first, c->mf->nptr, c->mf->nidx}; }

unsigned element_threads(const nb2_ctx* c) {
    return (unsigned)(c->npe == 8 ? kThreads<8> : kThreads<4>);
}
unsigned element_grid(const nb2_ctx* c) {
    return (c->E + element_threads(c) - 1) / element_threads(c);
}

template <int NPE, int MODEL, typename R>
cudaError_t apply_t(nb2_ctx* c, bool pdl, const R* z, const R* p, const CgScalars* s) {
    return launch_early(pdl, c->stream, element_grid(c), element_threads(c), 0, k_mf_apply<NPE, MODEL, R>,
                  view<R>(c), (R)c->mat.bulk_modulus, z, p, s);
}

template <int NPE, typename R>
cudaError_t apply_model(nb2_ctx* c, bool pdl, const R* z, const R* p, const CgScalars* s) {
    switch (c->mat.model) {
        case MODEL_LE: return apply_t<NPE, MODEL_LE>(c, pdl, z, p, s);
        case MODEL_NH: return apply_t<NPE, MODEL_NH>(c, pdl, z, p, s);
        case MODEL_J2:
            if constexpr (sizeof(R) == 4)
                if (!c->mf->odd32) return apply_t<NPE, MODEL_J2>(c, pdl, z, p, s);
            return apply_t<NPE, MODEL_J2S>(c, pdl, z, p, s);
        case MODEL_MS: return apply_t<NPE, MODEL_MS>(c, pdl, z, p, s);
        default:
            if constexpr (sizeof(R) == 4)
                return c->mat.model == MODEL_ML ? apply_t<NPE, MODEL_ML>(c, pdl, z, p, s)
                                                : apply_t<NPE, MODEL_MN>(c, pdl, z, p, s);
            else
                return cudaErrorInvalidValue;
    }
}

// the element products of K (z + beta p) into ye
template <typename R>
cudaError_t apply(nb2_ctx* c, bool pdl, const R* z, const R* p, const CgScalars* s) {
    c->launches++;
    return c->npe == 8 ? apply_model<8>(c, pdl, z, p, s) : apply_model<4>(c, pdl, z, p, s);
}

template <typename T>
int allocate(nb2_ctx* c, T** p, long long count) {
    if (*p) return NB2_OK;
    if (cudaMalloc((void**)p, sizeof(T) * std::max<long long>(count, 1)) != cudaSuccess) {
        *p = nullptr;
        return cuda_fail(c, cudaGetLastError(), "cudaMalloc (matrix-free operator)");
    }
    return NB2_OK;
}

int coefficients(int model) {
    return model == MODEL_J2 ? 8 : (model == MODEL_LE ? 2 : (model_aniso(model) ? 8 + 21 : 8));
}

struct Scratch {  // freed on every way out
    void* p = nullptr;
    ~Scratch() {
        if (p) cudaFree(p);
    }
};

int build_plan(nb2_ctx* c, MfPlan* P) {
    const int E = c->E, N = c->N, npe = c->npe;
    const long long m = (long long)E * npe;
    NB2_TRY(allocate(c, &P->nptr, N + 1));
    NB2_TRY(allocate(c, &P->first, N));
    NB2_TRY(allocate(c, &P->nidx, m));
    NB2_TRY(allocate(c, &P->ye, 3 * m));
    NB2_TRY(allocate(c, &P->de, 3 * m));
    // node -> its products, ascending (a stable sort keeps it)
    Scratch keys;
    int* kp = nullptr;
    NB2_TRY(allocate(c, &kp, m));
    keys.p = kp;
    auto product_nodes = npe == 8 ? k_product_nodes<8> : k_product_nodes<4>;
    product_nodes<<<element_grid(c), element_threads(c), 0, c->stream>>>(E, N, c->conn, kp,
                                                                          P->nidx);
    try {  // its scratch may not fit; no exception may pass the C interface
        thrust::stable_sort_by_key(thrust::cuda::par.on(c->stream), thrust::device_pointer_cast(kp),
                                   thrust::device_pointer_cast(kp + m),
                                   thrust::device_pointer_cast(P->nidx));
    } catch (const std::exception& e) {
        cudaGetLastError();
        c->error = std::string("matrix-free operator: ") + e.what();
        return NB2_E_CUDA;
    }
    k_node_products<<<(N + 1 + 255) / 256, 256, 0, c->stream>>>(kp, P->nidx, m, N, P->first,
                                                               P->nptr);
    c->launches += 2;
    NB2_CUDA(c, cudaGetLastError());
    NB2_CUDA(c, cudaStreamSynchronize(c->stream));
    return NB2_OK;
}

// the Jacobi inverse of the last setup's contributions
template <typename X>
int jacobi(nb2_ctx* c, X* inv) {
    MfPlan* P = c->mf;
    if (c->npe == 8)
        k_mf_diag_products<8><<<element_grid(c), element_threads(c), 0, c->stream>>>(c->E, c->conn, P->de,
                                                                         P->ye);
    else
        k_mf_diag_products<4><<<element_grid(c), element_threads(c), 0, c->stream>>>(c->E, c->conn, P->de,
                                                                         P->ye);
    auto kernel = c->npe == 8 ? k_mf_inv<8, X> : k_mf_inv<4, X>;
    kernel<<<(c->N + 255) / 256, 256, 0, c->stream>>>(c->N, sums(c), P->ye, inv);
    c->launches += 2;
    NB2_CUDA(c, cudaGetLastError());
    return NB2_OK;
}

// one thread per node, up to 8 blocks an SM (the partial sums have room for 8 per block of the other
// reductions)
unsigned gather_grid(const nb2_ctx* c) {
    return (unsigned)std::min((c->N + kRedThreads - 1) / kRedThreads,
                              (c->npe == 8 ? 2 : 1) * reduction_blocks(c));
}

// Iterations in captured blocks until the device scalars say done.
template <typename R>
struct MfRunner {
    nb2_ctx* c;
    R *x, *r, *z, *p, *q, *inv;
    bool use_graphs;
    cudaGraphExec_t* cache;

    cudaError_t enqueue() {
        const int RB = reduction_blocks(c);
        const MfPlan* P = c->mf;
        const R* ye = reinterpret_cast<const R*>(P->ye);
        // early starts gain 1-3% on hex8; on tet4 they lose 8% (waiting blocks take the place of working
        // ones)
        const bool pdl = c->npe == 8;
        for (int it = 0; it < kIterations; ++it) {
            cudaError_t e;
            if constexpr (sizeof(R) == 4) {
                if (c->npe == 4) {
                    e = launch_early(pdl, c->stream, gather_grid(c), (unsigned)kRedThreads, 0, k_mf_p,
                               c->N, (const float*)z, p, (const CgScalars*)c->cgs);
                    if (e == cudaSuccess)
                        e = apply<R>(c, pdl, (const R*)p, (const R*)nullptr, c->cgs);
                } else {
                    e = apply<R>(c, pdl, z, p, c->cgs);
                }
            } else {
                e = apply<R>(c, pdl, z, p, c->cgs);  // hex8 only
            }
            if (e == cudaSuccess)
                e = launch_early(pdl, c->stream, gather_grid(c), (unsigned)kRedThreads, 0,
                           c->npe == 8 ? k_mf_gather<8, R> : k_mf_gather<4, R>, c->N, sums(c), ye,
                           (const R*)z, p, q, (const unsigned char*)c->mask, c->cgs, c->partials);
            if (e == cudaSuccess)
                e = launch_early(pdl, c->stream, (unsigned)RB, (unsigned)kRedThreads, 0, k_mf_xr<R>,
                           (long long)c->n, x, r, z, (const R*)p, (const R*)q, (const R*)inv,
                           c->cgs, c->partials);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    int run(int maxit) {
        if (use_graphs && *cache == nullptr) {
            // plain launches if the stream cannot be captured (e.g. the legacy default stream)
            cudaGraph_t g = nullptr;
            if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) ==
                cudaSuccess) {
                const long long before = c->launches;
                const cudaError_t e = enqueue();
                c->launches = before;
                if (cudaStreamEndCapture(c->stream, &g) == cudaSuccess && g) {
                    if (e != cudaSuccess || cudaGraphInstantiate(cache, g, 0) != cudaSuccess)
                        *cache = nullptr;
                    cudaGraphDestroy(g);
                }
            }
            cudaGetLastError();
            if (*cache == nullptr) use_graphs = false;
        }
        int guard = 0;
        for (;;) {
            if (use_graphs)
                NB2_CUDA(c, cudaGraphLaunch(*cache, c->stream));
            else
                NB2_CUDA(c, enqueue());
            c->launches += 3 * kIterations;
            NB2_TRY(wait_scalars(c));
            if (c->h_cgs->done) break;
            if (++guard > (maxit / kIterations) + 4) break;  // scalars say not done: cannot happen
        }
        NB2_CUDA(c, cudaGetLastError());
        return NB2_OK;
    }
};

}  // namespace

void mf_release(MfPlan* P) {
    if (!P) return;
    for (auto g : {P->graph32[0], P->graph32[1], P->graph64})
        if (g) cudaGraphExecDestroy(g);
    void* ptrs[] = {P->first, P->nptr, P->nidx, P->ye,  P->de, P->md,
                    P->mc32,  P->mc64, P->x,    P->z32, P->p32,
                    P->z64};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete P;
}

bool mf64_applies(const nb2_ctx* c) { return !model_aniso(c->mat.model); }

bool mf64_ready(const nb2_ctx* c) {
    return c->mf && c->mf->mc64 && c->mf->x && c->mf->z64;
}

int ensure_mf(nb2_ctx* c, bool fp32, bool fp64) {
    if (!c->mf) {
        auto* P = new MfPlan();
        const int st = build_plan(c, P);
        if (st != NB2_OK) {
            mf_release(P);
            return st;
        }
        c->mf = P;
    }
    MfPlan* P = c->mf;
    const long long points = (long long)c->nqp * coefficients(c->mat.model);
    if (fp32) {
        NB2_TRY(allocate(c, &P->md, 3ll * c->npe * c->E));
        NB2_TRY(allocate(c, &P->mc32, points));
        NB2_TRY(allocate(c, &P->z32, 4ll * c->N));
        NB2_TRY(allocate(c, &P->p32, 4ll * c->N));
    }
    if (fp64 && mf64_applies(c) && !mf64_ready(c)) {
        int st = allocate(c, &P->mc64, points);
        if (st == NB2_OK) st = allocate(c, &P->x, (long long)c->n);
        if (st == NB2_OK) st = allocate(c, &P->z64, (long long)c->n);
        if (st != NB2_OK) {  // its callers go without it: leave them the room
            for (double** p : {&P->mc64, &P->x, &P->z64}) {
                if (*p) cudaFree(*p);
                *p = nullptr;
            }
            if (!P->p32) {
                mf_release(P);
                c->mf = nullptr;
            }
            return st;
        }
    }
    return NB2_OK;
}

int mf_setup(nb2_ctx* c, bool fp32, bool fp64) {
    MfPlan* P = c->mf;
    if (fp64) {
        NB2_TRY(launch_mf_setup64(c, P->mc64, P->de));
        k_mf_positions<<<vec_grid(c->n), 256, 0, c->stream>>>(c->n, c->X, c->u_tan, P->x);
        c->launches++;
    }
    if (fp32) NB2_TRY(launch_mf_setup32(c, P->md, P->mc32, P->de));
    NB2_CUDA(c, cudaGetLastError());
    return NB2_OK;
}

// which FP32 product the last setup asks for; waits for it
static int choose_product32(nb2_ctx* c) {
    NB2_TRY(wait_scalars(c));
    c->mf->odd32 = c->h_cgs->mf_odd_setup == c->mf_setups;
    return NB2_OK;
}

int mf_apply64(nb2_ctx* c, const double* v, double* y) {
    const double* none = nullptr;
    NB2_CUDA(c, apply<double>(c, false, v, none, nullptr));
    auto kernel = c->npe == 8 ? k_mf_sum<8, double> : k_mf_sum<4, double>;
    kernel<<<(c->N + 255) / 256, 256, 0, c->stream>>>(c->N, sums(c), c->mf->ye, y);
    c->launches++;
    NB2_CUDA(c, cudaGetLastError());
    return NB2_OK;
}

int mf_apply(nb2_ctx* c, const double* v, double* y) {
    NB2_TRY(ensure_mf(c, true, false));
    NB2_TRY(mf_setup(c, true, false));
    NB2_TRY(choose_product32(c));
    k_to_float<<<vec_grid(c->n), 256, 0, c->stream>>>(c->n, v, c->mf->z32);
    const float* none = nullptr;
    NB2_CUDA(c, apply<float>(c, false, (const float*)c->mf->z32, none, nullptr));
    auto kernel = c->npe == 8 ? k_mf_sum<8, float> : k_mf_sum<4, float>;
    kernel<<<(c->N + 255) / 256, 256, 0, c->stream>>>(
        c->N, sums(c), reinterpret_cast<const float*>(c->mf->ye), y);
    c->launches += 2;
    NB2_CUDA(c, cudaGetLastError());
    return NB2_OK;
}

int pcg_mf64(nb2_ctx* c, const double* b, double* x, double tol, int maxit, int* iterations,
             double* error, bool use_graphs) {
    NB2_TRY(ensure_mf(c, false, true));
    MfPlan* P = c->mf;
    NB2_TRY(mf_setup(c, false, true));
    NB2_TRY(jacobi(c, c->cg_inv));
    MfRunner<double> cg{c,       c->cg_x,   c->cg_r,    P->z64,     c->cg_p,
                        c->cg_q, c->cg_inv, use_graphs, &P->graph64};
    k_mf_init<double><<<reduction_blocks(c), kRedThreads, 0, c->stream>>>(
        c->n, b, cg.x, cg.r, cg.z, cg.p, cg.inv, c->cgs, c->partials, tol, maxit);
    c->launches++;
    NB2_TRY(cg.run(maxit));
    k_copy_double<<<vec_grid(c->n), 256, 0, c->stream>>>(c->n, cg.x, x);
    c->launches++;
    const CgScalars& h = *c->h_cgs;
    *iterations = h.iterations;
    *error = h.rhs_norm2 > 0 ? std::sqrt(h.rr / h.rhs_norm2) : 0.0;
    if (h.status) return h.status;
    if (!h.done) return NB2_E_TIMEOUT;
    return NB2_OK;
}

// Mixed-precision PCG with reliable updates (residual replacement): the iterations run in FP32
// (FP64 dot products); whenever the FP32 residual has dropped by `delta` since the last replacement
// (or below the final threshold), the FP32 increment is folded into the FP64 iterate x, the true
// residual b - K x is formed with the FP64 operator, and the FP32 residual is replaced by it; the
// search direction is kept, so the Krylov space is not thrown away as a restarted defect correction
// does.  Stops when the true residual meets ||r|| < tol ||b|| (the PCG's stop test,
// linear_solver.cpp:67-109).
int pcg_reliable_mixed(nb2_ctx* c, const double* b, double* x, double tol, double delta,
                       int maxit, double* work, int* iterations, bool use_graphs) {
    const bool mf64 = mf64_ready(c);  // else the element kernels' product
    NB2_TRY(ensure_mf(c, true, false));
    MfPlan* P = c->mf;
    NB2_TRY(mf_setup(c, true, mf64));
    NB2_TRY(jacobi(c, c->cg32_inv));
    MfRunner<float> cg{c,         c->cg32_x,   c->cg32_r,  P->z32,     P->p32,
                       c->cg32_q, c->cg32_inv, use_graphs, nullptr};
    const long long n = c->n;
    const int RB = reduction_blocks(c);
    NB2_CUDA(c, cudaMemsetAsync(x, 0, sizeof(double) * n, c->stream));
    // the first pause comes after a delta reduction of ||b|| (threshold max(tol, delta)^2 b.b)
    k_mf_init<float><<<RB, kRedThreads, 0, c->stream>>>(n, b, cg.x, cg.r, cg.z, cg.p, cg.inv,
                                                        c->cgs, c->partials, std::max(tol, delta),
                                                        maxit);
    c->launches++;
    NB2_TRY(choose_product32(c));
    cg.cache = &P->graph32[P->odd32];
    const double b2 = c->h_cgs->rhs_norm2;
    const double thr = std::max(tol * tol * b2, 2.2250738585072014e-308);
    *iterations = 0;
    if (b2 == 0.0) return NB2_OK;
    int resets = 0;
    for (int update = 0;; ++update) {
        if (!c->h_cgs->done) NB2_TRY(cg.run(maxit));
        const CgScalars h = *c->h_cgs;
        *iterations = h.iterations;
        // a diverged cycle (its kept search direction no longer fits the replaced residual,
        // near the FP32 operator's accuracy floor): replace the residual again and restart the
        // cycle with p = D^-1 r, at most three times per solve
        const bool fresh = h.status == NB2_E_CG_BREAKDOWN && resets < 3;
        if (fresh) ++resets;
        if (h.status && h.status != NB2_E_CG_MAXIT && !fresh) return h.status;
        // reliable update: x += xs; r = b - K x in FP64
        k_fold<<<vec_grid(n), 256, 0, c->stream>>>(n, cg.x, x);
        NB2_TRY(mf64 ? mf_apply64(c, x, work) : launch_apply(c, x, work));
        k_true_residual<<<RB, kRedThreads, 0, c->stream>>>(n, b, work, c->mask, cg.inv, cg.r, cg.z,
                                                           c->cgs, c->partials, thr, delta,
                                                           fresh ? 1 : 0);
        c->launches += 2;
        NB2_TRY(wait_scalars(c));
        const double rr = c->h_cgs->rr;
        if (std::getenv("NB2_DEBUG"))
            std::fprintf(stderr, "[nb2] reliable update %d: its %d true |r|^2 %.6e thr %.6e\n",
                         update, h.iterations, rr, thr);
        if (!std::isfinite(rr)) return NB2_E_NAN;
        if (rr < thr) return NB2_OK;
        if (h.status == NB2_E_CG_MAXIT || h.iterations >= maxit || update > 1000)
            return NB2_E_CG_MAXIT;
    }
}

}  // namespace nb2
