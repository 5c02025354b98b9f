// Backward pass of the layer (backward.cu) and the tensor-core products it adds to the forward's.
#pragma once

#include "common.cuh"

namespace omoe {

int bw_set_training(omoe_handle *h, int on);
bool bw_training(const omoe_handle *h);
void bw_forward_invalidate(omoe_handle *h);
// A training-mode forward of no rows on one GPU launches nothing and still counts as the forward a backward follows.
void bw_forward_empty(omoe_handle *h);
// Expert stage of a training-mode forward: g and u kept, then h = silu(g) * u, then the down product.
cudaError_t bw_forward_experts(omoe_handle *h, int T, cudaStream_t s, int *n);
// x_is_compute: x has the layer's compute dtype (the normalised rows of the block form) instead of io_dtype
int bw_backward(omoe_handle *h, const void *x, bool x_is_compute, const void *dy, void *dx, int T, int io_dtype,
                cudaStream_t s, int *launches);
int bw_backward_block(omoe_handle *h, const void *x, const float *gamma, float eps, const void *dy, void *dx,
                      float *dgamma, int T, int io_dtype, cudaStream_t s, int *launches);
int bw_get_grads(omoe_handle *h, float *d_router, float *d_bias, float *d_gate, float *d_up, float *d_down,
                 cudaStream_t s);
int bw_set_aux(omoe_handle *h, float coef);
// counts_host: picks per expert, or null to take them from the device.
int bw_aux_loss(omoe_handle *h, float *loss_host, cudaStream_t s, const int32_t *counts_host);
void bw_destroy(omoe_handle *h);

// 2-D bf16 tensor map: [rows, cols] with `ld` elements between rows, box box_rows x 64 columns, 128-byte swizzle.
bool encode_map_bf16(CUtensorMap *m, void *ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
// Per matrix z < n_mat (1 or 2) and local expert e: C_z,e [M, N] (fp32) = A_z[seg_e]^T * B[seg_e], seg_e = the expert's rows
// rounded up to 64.  a*, b: row-major activations [rows_cap, M or N] bf16 with a box of 64 rows; o*: [e_local, M, N] fp32 with
// a box of 32 x 32.  Rows past an expert's count must be zero in A and finite in B.  (experts_sm100_wgrad.cu)
struct alignas(64) WgradMaps {
    CUtensorMap a0, a1, b, o0, o1;
};
cudaError_t launch_wgrad(omoe_handle *h, cudaStream_t s, const WgradMaps &maps, int n_mat, int M, int N);

// fp32 layers (experts_f32.cu); rows as for launch_experts_f32.  Forward products: h = silu(g) * u and yp, keeping g | u in gu unless null.
cudaError_t f32_forward_experts(omoe_handle *h, cudaStream_t s, long rows, void *gu, int *n);
// dgu = dg | du and dxp from the gradient dyp of the expert outputs.
cudaError_t f32_grad_rows(omoe_handle *h, cudaStream_t s, long rows, const void *dyp, void *gu, void *dgu, void *dxp, int *n);
// out_z [e_local, M, N] = (a + z*a_next)^T * b over each expert's rows, z < n_mat; a has lda floats between rows.
cudaError_t f32_wgrad(omoe_handle *h, cudaStream_t s, const void *a, int lda, int a_next, const void *b, int n_mat, int M,
                      int N, float *out0, float *out1);

}  // namespace omoe
