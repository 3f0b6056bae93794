// hydro_train.h -- parameters of the fused training step (hydro_train.cu).
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace sfh {

// Rows forward and back: x0 [batch][64] inputs, target [batch][n_out]; the
// BF16 layer inputs x and gradients dz are outputs; z[3] [batch][64] receives
// the network's outputs (first n_out columns) or, where a step keeps them,
// every z [batch][n_l] its layer's pre-activations.
struct RowsParams {
    const __nv_bfloat16* x0;
    const float* target;
    const float* tmean;
    const float* tistd;
    const __nv_bfloat16* w16[4];
    const __nv_bfloat16* wt16[4];
    const float* bias[4];
    __nv_bfloat16* x[3];
    __nv_bfloat16* dz[4];
    float* z[4];
    int batch;
    int n_out;
};

// One layer's gradients: part receives `splits` partial products [k][n] over
// slice_rows batch rows each, col `slabs` column sums [n] over slab_rows rows.
struct GradLayer {
    const __nv_bfloat16* in;
    const __nv_bfloat16* dz;
    float* part;
    float* col;
    int k, n;
    int splits, slice_rows;
    int slabs, slab_rows;
};

struct GradsParams {
    GradLayer layer[4];
    const float* target;
    const float* tmean;
    const float* tistd;
    const float* z3;
    double* loss;
    int batch;
    int n_out;
};

struct UpdateLayer {
    const float* part;
    const float* col;
    float *w, *mw, *vw, *gw;
    float *b, *mb, *vb, *gb;
    __nv_bfloat16* w16;
    __nv_bfloat16* wt16;
    int k, n;
    int splits, slabs;
};

struct UpdateParams {
    UpdateLayer layer[4];
    float lr, b1, b2, eps, wd, bc1, bc2;
};

// keep: leave the pre-activations in R.z
cudaError_t launch_train_step(const RowsParams& R, const GradsParams& G, const UpdateParams& U, bool keep,
                              cudaStream_t s);

}  // namespace sfh
