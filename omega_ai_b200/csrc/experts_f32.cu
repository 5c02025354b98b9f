// fp32 expert products on CUDA cores (compute_dtype = OMOE_F32).  This is the
// arithmetic the reference's FullyLayer performs (cublasSgemm, fp32 in and out;
// src/main/java/com/omega/engine/nn/layer/FullyLayer.java:235 ->
// src/main/java/com/omega/engine/gpu/GPUOP.java:405-417) in the order of
// LlamaMLPLayer.output() (LlamaMLPLayer.java:117-123), with SiLU
// (src/main/resources/cu/activeFunction.cu:172-180) and the element-wise
// product (src/main/resources/cu/OPKernel.cu:1040) fused into the first
// product's epilogue instead of being three more passes over [rows, d_ff]; the backward's SwiGLU pass is the epilogue
// of the product in front of it likewise.
//
// These layers are small (the engine's own precision, sized for a host-side reference run), so what bounds a product is
// latency: a few hundred rows over 4 to 16 experts, a reduction of a few hundred.  Hence small tiles that skip
// padding rows (32 rows x 64 columns, 128 threads, 4 x 4 outputs each), operands brought by 16-byte asynchronous
// copies into a ring of three stages so that the loads of two steps are always under way, and both halves of a
// gate/up pair in one block.  Measured against 64 x 64 tiles that loaded, waited and multiplied in turn and walked the padding
// rows in the backward: forward of 64 tokens, d 128, d_ff 256, 8 experts 44.4 -> 27.5 us; training step of 300 tokens,
// d 256, d_ff 384 497 -> 181 us.  Every output is one chain of fused multiply-adds over ascending k.
//
// Blocks are numbered over the row tiles that hold rows, as many as the step's rows can give: a grid over the buffers' rows made
// blocks without rows hold their slots until the product before was done, and had the real ones share the SMs that were left
// (256 tokens, d 512, d_ff 1024, 8 experts top-2: 158 us, now 109; 48 tiles of which 20 hold rows).
#include "backward.cuh"
#include "common.cuh"

namespace omoe {

namespace {

constexpr int BM = 32, BN = 64, BK = 16, ST = 3;
constexpr int LDK = BK + 4;  // words between rows of a tile stored [row][k]: 8 rows of 16-byte reads hit 32 banks
constexpr int LDN = BN + 4;  // words between rows of a tile stored [k][column]

__device__ __forceinline__ void cp16(float *dst, const float *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float silu_f32(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_grad_f32(float x) {
    const float sg = 1.0f / (1.0f + expf(-x));
    return sg * (1.0f + x * (1.0f - sg));
}

enum Epi {
    kStore,       // c = A B0
    kSwiglu,      // c = silu(A B0) * (A B1)
    kSwigluKeep,  // the same, and gu[r] = A B0 | A B1
    kSwigluBack,  // with dh = A B0 and g, u from gu: c[r] = (dh * u) * silu'(g) | dh * silu(g), 2 N columns
    kSum,         // c = A B0 + A1 B1
};

// Rows grouped by expert, row tiles numbered over the experts in order, column tiles fastest.  B is [expert][n][k] (B_KN false) or
// [expert][k][n]; A1 starts a_next floats after A.
template <bool B_KN, Epi EPI>
__global__ void __launch_bounds__(128)
rows_sgemm_kernel(const float *__restrict__ A, int lda, int a_next, const float *__restrict__ B0,
                  const float *__restrict__ B1, float *__restrict__ C, float *__restrict__ gu, int N, int K,
                  const int32_t *__restrict__ poffsets, const int32_t *__restrict__ counts, int E) {
    constexpr int NS = (EPI == kStore || EPI == kSwigluBack) ? 1 : 2;  // accumulator sets
    constexpr int NA = EPI == kSum ? 2 : 1;
    constexpr int B_WORDS = B_KN ? BK * LDN : BN * LDK;
    __shared__ __align__(16) float sa[ST][NA][BM * LDK];
    __shared__ __align__(16) float sb[ST][NS][B_WORDS];
    pdl_wait();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int n_ct = (N + BN - 1) / BN, rt = blockIdx.x / n_ct, n0 = (blockIdx.x - rt * n_ct) * BN;
    // the expert of row tile rt, ceil(count / BM) tiles each; every warp works it out for itself
    int e = -1, tile = 0, cnt = 0, before = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
        const int lane = tid & 31;
        const int c = e0 + lane < E ? counts[e0 + lane] : 0, own = (c + BM - 1) / BM;
        int upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        upto += before;
        const uint32_t hit = __ballot_sync(0xffffffffu, rt >= upto - own && rt < upto);
        if (hit != 0) {
            const int src = __ffs(hit) - 1;
            e = e0 + src;
            tile = rt - __shfl_sync(0xffffffffu, upto - own, src);
            cnt = __shfl_sync(0xffffffffu, c, src);
            break;
        }
        before = __shfl_sync(0xffffffffu, upto, 31);
    }
    if (e < 0) return;
    const int row0 = poffsets[e] + tile * BM, valid = cnt - tile * BM;  // rows of this tile that carry tokens: > 0
    const float *Bs[2] = {B0 + (size_t)e * N * K, NS == 2 ? B1 + (size_t)e * N * K : nullptr};

    auto issue = [&](int step) {
        const int st = step % ST, k0 = step * BK;
        {
            const int r = tid >> 2, c = (tid & 3) * 4;  // 32 rows x 4 pieces
            const bool ok = r < valid && k0 + c < K;   // K is a multiple of 8: a piece is whole or absent
#pragma unroll
            for (int a = 0; a < NA; a++)
                cp16(&sa[st][a][r * LDK + c], ok ? A + (size_t)(row0 + r) * lda + a * a_next + k0 + c : A, ok);
        }
#pragma unroll
        for (int b = 0; b < NS; b++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int p = tid + i * 128;
                if constexpr (B_KN) {
                    const int kk = p >> 4, c = (p & 15) * 4;
                    const bool ok = k0 + kk < K && n0 + c < N;
                    cp16(&sb[st][b][kk * LDN + c], ok ? Bs[b] + (size_t)(k0 + kk) * N + n0 + c : B0, ok);
                } else {
                    const int n = p >> 2, c = (p & 3) * 4;
                    const bool ok = n0 + n < N && k0 + c < K;
                    cp16(&sb[st][b][n * LDK + c], ok ? Bs[b] + (size_t)(n0 + n) * K + k0 + c : B0, ok);
                }
            }
        cp_commit();
    };

    float acc[NS][4][4] = {};
    const int steps = (K + BK - 1) / BK;
    issue(0);
    if (steps > 1) issue(1);
    else cp_commit();
    for (int s = 0; s < steps; s++) {
        cp_wait<1>();
        __syncthreads();  // the step's tiles are in for everyone, and everyone is done with the stage refilled next
        if (s + 2 < steps) issue(s + 2);
        else cp_commit();
        const int st = s % ST;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float4 a[NA][4];
#pragma unroll
            for (int q = 0; q < NA; q++)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    a[q][i] = *reinterpret_cast<const float4 *>(&sa[st][q][(ty * 4 + i) * LDK + kk]);
#pragma unroll
            for (int b = 0; b < NS; b++) {
                float4 w[4];  // B_KN: w[k] holds columns 4tx..4tx+3; else w[j] holds four k of column tx + 16j
#pragma unroll
                for (int j = 0; j < 4; j++)
                    w[j] = *reinterpret_cast<const float4 *>(B_KN ? &sb[st][b][(kk + j) * LDN + tx * 4]
                                                                 : &sb[st][b][(tx + 16 * j) * LDK + kk]);
                const float4 *av = a[NA == 2 ? b : 0];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float v = acc[b][i][j];
                        if constexpr (B_KN) {
                            v = fmaf(av[i].x, (&w[0].x)[j], v);
                            v = fmaf(av[i].y, (&w[1].x)[j], v);
                            v = fmaf(av[i].z, (&w[2].x)[j], v);
                            v = fmaf(av[i].w, (&w[3].x)[j], v);
                        } else {
                            v = fmaf(av[i].x, w[j].x, v);
                            v = fmaf(av[i].y, w[j].y, v);
                            v = fmaf(av[i].z, w[j].z, v);
                            v = fmaf(av[i].w, w[j].w, v);
                        }
                        acc[b][i][j] = v;
                    }
            }
        }
    }
    pdl_trigger();  // not before: a block of the next product that waits here takes this one's place
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = ty * 4 + i;
        if (r >= valid) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + (B_KN ? tx * 4 + j : tx + 16 * j);
            if (n >= N) continue;
            const size_t row = (size_t)(row0 + r);
            const float v = acc[0][i][j];
            if constexpr (EPI == kStore) {
                C[row * N + n] = v;
            } else if constexpr (EPI == kSum) {
                C[row * N + n] = v + acc[1][i][j];
            } else if constexpr (EPI == kSwigluBack) {
                const float g = gu[row * 2 * N + n], u = gu[row * 2 * N + N + n];
                C[row * 2 * N + n] = (v * u) * silu_grad_f32(g);
                C[row * 2 * N + N + n] = v * silu_f32(g);
            } else {
                const float u = acc[NS - 1][i][j];
                if constexpr (EPI == kSwigluKeep) {
                    gu[row * 2 * N + n] = v;
                    gu[row * 2 * N + N + n] = u;
                }
                C[row * N + n] = silu_f32(v) * u;
            }
        }
    }
}

// Weight gradients: matrix z (blockIdx.z / E) and expert (blockIdx.z % E): C_z,e[m, n] = sum over the expert's rows r,
// ascending, of A[r, z*a_next + m] * B[r, n].  64 x 64 tiles, 256 threads.
__global__ void __launch_bounds__(256)
wgrad_sgemm_kernel(const float *__restrict__ A, int lda, int a_next, const float *__restrict__ B, int ldb,
                   float *__restrict__ C0, float *__restrict__ C1, int M, int N, const int32_t *__restrict__ poffsets,
                   const int32_t *__restrict__ counts, int E) {
    __shared__ __align__(16) float sa[ST][BK * LDN], sb[ST][BK * LDN];
    const int z = blockIdx.z / E, e = blockIdx.z - z * E, m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    pdl_trigger();
    pdl_wait();
    const int row0 = poffsets[e], cnt = counts[e];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int kk0 = tid >> 4, c0 = (tid & 15) * 4;  // this thread's 16-byte piece of a step: row, column
    auto issue = [&](int step) {
        const int st = step % ST, r = step * BK + kk0;
        const bool in = r < cnt, oka = in && m0 + c0 < M, okb = in && n0 + c0 < N;
        cp16(&sa[st][kk0 * LDN + c0], oka ? A + (size_t)(row0 + r) * lda + (size_t)z * a_next + m0 + c0 : A, oka);
        cp16(&sb[st][kk0 * LDN + c0], okb ? B + (size_t)(row0 + r) * ldb + n0 + c0 : B, okb);
        cp_commit();
    };
    float acc[4][4] = {};
    const int steps = (cnt + BK - 1) / BK;
    if (steps > 0) issue(0);
    if (steps > 1) issue(1);
    else cp_commit();
    for (int s = 0; s < steps; s++) {
        cp_wait<1>();
        __syncthreads();
        if (s + 2 < steps) issue(s + 2);
        else cp_commit();
        const int st = s % ST;
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a = *reinterpret_cast<const float4 *>(&sa[st][kk * LDN + ty * 4]);
            const float4 b = *reinterpret_cast<const float4 *>(&sb[st][kk * LDN + tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
    float *C = z ? C1 : C0;
    const int n = n0 + tx * 4;
    if (n >= N) return;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty * 4 + i;
        if (m < M)
            *reinterpret_cast<float4 *>(&C[((size_t)e * M + m) * N + n]) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// Most row tiles any placement of a step's rows on the local experts can give; `rows` is negative where only the capacity of
// the buffers bounds them.
long row_tiles(const omoe_handle *h, long rows) {
    if (rows < 0) return h->rows_cap / BM;
    const long some = rows < h->e_local ? rows : h->e_local;  // experts that can have a row
    return some + (rows - some) / BM;
}

// Dependent launch hides about 3.5 us per forward, but the blocks of the next product then settle, several to an SM, wherever
// the product before them finishes first, and stay there while the other SMs go idle.  That costs nothing while all blocks are
// fewer than the SMs by a margin: it is used up to two thirds of the SMs.  Forward with it and without: 44 blocks (256 tokens, d 128,
// d_ff 256, 4 experts top-1) 27.9 us against 31.0; 92 (8 experts top-2) 31.8 against 31.7; 140 (1024 tokens, 4 experts) 40.6 against 33.0;
// 368 (256 tokens, d 512, d_ff 1024, 8 experts top-2) 121 against 110.
bool dependent_launch(const omoe_handle *h, long rows) {
    const int widest = h->cfg.d_model > h->cfg.d_ff ? h->cfg.d_model : h->cfg.d_ff;
    return h->pdl && h->cfg.world == 1 && row_tiles(h, rows) * ceil_div(widest, BN) * 3 <= 2 * (long)h->sm_count;
}

template <bool B_KN, Epi EPI>
cudaError_t launch_rows(omoe_handle *h, cudaStream_t s, long rows, const void *A, int lda, int a_next, const void *B0,
                        const void *B1, void *C, void *gu, int N, int K) {
    return launch_ex(rows_sgemm_kernel<B_KN, EPI>, dim3((unsigned)(row_tiles(h, rows) * ceil_div(N, BN))), dim3(128), 0, s,
                     dependent_launch(h, rows), static_cast<const float *>(A), lda, a_next, static_cast<const float *>(B0),
                     static_cast<const float *>(B1), static_cast<float *>(C), static_cast<float *>(gu), N, K,
                     h->ex_poffsets, h->ex_counts, h->e_local);
}

}  // namespace

cudaError_t f32_forward_experts(omoe_handle *h, cudaStream_t s, long rows, void *gu, int *n) {
    const int d = h->cfg.d_model, dff = h->cfg.d_ff;
    cudaError_t e = gu ? launch_rows<false, kSwigluKeep>(h, s, rows, h->xp, d, 0, h->w_gate, h->w_up, h->hbuf, gu, dff, d)
                       : launch_rows<false, kSwiglu>(h, s, rows, h->xp, d, 0, h->w_gate, h->w_up, h->hbuf, nullptr, dff, d);
    if (e != cudaSuccess) return e;
    (*n)++;
    e = launch_rows<false, kStore>(h, s, rows, h->hbuf, dff, 0, h->w_down, nullptr, h->yp, nullptr, d, dff);
    if (e == cudaSuccess) (*n)++;
    return e;
}

cudaError_t launch_experts_f32(omoe_handle *h, cudaStream_t s, int *n, long rows) { return f32_forward_experts(h, s, rows, nullptr, n); }

cudaError_t f32_grad_rows(omoe_handle *h, cudaStream_t s, long rows, const void *dyp, void *gu, void *dgu, void *dxp, int *n) {
    const int d = h->cfg.d_model, dff = h->cfg.d_ff;
    cudaError_t e = launch_rows<true, kSwigluBack>(h, s, rows, dyp, d, 0, h->w_down, nullptr, dgu, gu, dff, d);
    if (e != cudaSuccess) return e;
    (*n)++;
    e = launch_rows<true, kSum>(h, s, rows, dgu, 2 * dff, dff, h->w_gate, h->w_up, dxp, nullptr, d, dff);
    if (e == cudaSuccess) (*n)++;
    return e;
}

cudaError_t f32_wgrad(omoe_handle *h, cudaStream_t s, const void *a, int lda, int a_next, const void *b, int n_mat, int M,
                      int N, float *out0, float *out1) {
    const int El = h->e_local;
    return launch_ex(wgrad_sgemm_kernel, dim3(ceil_div(N, 64), ceil_div(M, 64), n_mat * El), dim3(256), 0, s,
                     h->pdl && h->cfg.world == 1, static_cast<const float *>(a), lda, a_next, static_cast<const float *>(b), N, out0, out1, M, N,
                     h->ex_poffsets, h->ex_counts, El);
}

}  // namespace omoe
