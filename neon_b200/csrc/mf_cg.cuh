// mf_cg.cuh -- the matrix-free tangent product and its PCG: interface of mf_cg.cu.
#pragma once

#include "nb2_internal.cuh"

namespace nb2 {

// Element products and the lists that sum them per node; everything is fixed by the mesh and all
// sums run in a fixed order.
struct MfPlan {
    int4* first = nullptr;                 // [N] the first four products of a node
    int *nptr = nullptr, *nidx = nullptr;  // all of them, sorted by node
    double* ye = nullptr;                  // [npe][E][3] products (FP32: half of it)
    double* de = nullptr;                  // [3 npe][E] element contributions to diag(K)
    float* md = nullptr;                   // FP32 operator (k_mf_setup)
    float* mc32 = nullptr;
    double* mc64 = nullptr;                // FP64 operator: coefficients and node positions X + u
    double* x = nullptr;
    float *z32 = nullptr, *p32 = nullptr;  // D^-1 r and p of the PCG ([N][4]; FP64: [N][3])
    double* z64 = nullptr;
    cudaGraphExec_t graph32[2] = {nullptr, nullptr}, graph64 = nullptr;  // FP32: by odd32
    bool odd32 = false;                    // the last FP32 setup needs MODEL_J2S
};

void mf_release(MfPlan* p);

// Build the plan (once per context) and the buffers of the FP32 and / or FP64 operator.  Where the
// memory does not suffice nothing of the FP64 operator is left allocated: solves go without it.
int ensure_mf(nb2_ctx* c, bool fp32, bool fp64);
bool mf64_ready(const nb2_ctx* c);  // the FP64 operator's buffers are there
// whether the FP64 operator exists for the context's model (the anisotropic microspheres keep
// the assembled K: 29 FP64 coefficients per point are as many bytes)
bool mf64_applies(const nb2_ctx* c);

// operator data of the tangent stored by the last MODE_STORE pass
int mf_setup(nb2_ctx* c, bool fp32, bool fp64);
// y = K v with the FP64 operator of the last mf_setup (y unmasked)
int mf_apply64(nb2_ctx* c, const double* v, double* y);
// y = K v with the FP32 operator (sets it up; v, y device FP64; y unmasked)
int mf_apply(nb2_ctx* c, const double* v, double* y);

// Jacobi-PCG on the FP64 operator (sets it up)
int pcg_mf64(nb2_ctx* c, const double* b, double* x, double tol, int maxit, int* iterations,
             double* error, bool use_graphs);
// mixed precision with reliable updates: FP32 iterations, FP64 true residual every `delta`
// reduction (on the FP64 operator where it is ready); work: n doubles
int pcg_reliable_mixed(nb2_ctx* c, const double* b, double* x, double tol, double delta,
                       int maxit, double* work, int* iterations, bool use_graphs);

}  // namespace nb2
