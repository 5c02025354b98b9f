// Backward of the MoE layer: gradients with respect to the input rows and to every weight, for a
// given gradient of the output.
//
// The chain is the reference's, applied per expert to the rows that expert received:
//   LlamaMLPLayer.diff() (src/main/java/com/omega/engine/nn/layer/llama/LlamaMLPLayer.java:139-158):
//     linear2.back(delta); d_up = d_h * silu(g); d_gate = silu_backward(g, d_h * u); diff = linear1.diff + linear3.diff
//   FullyLayer.diff() (src/main/java/com/omega/engine/nn/layer/FullyLayer.java:292-334):
//     diffW = delta^T * input (overwritten each call), diff = delta * W, diffB = column sums of delta
//   silu_backward (src/main/resources/cu/activeFunction.cu:182-190), softmax_back
//   (src/main/resources/cu/SoftmaxKernel.cu:100-112) for the router's probabilities.
// What the reference does not have is fixed here: the picks are constants; with renormalised gates
// w_j = p_j / s the probabilities get d p_j = (d w_j - sum_i d w_i w_i) / s; d w_j = <dy[t], yp_j>;
// dx[t] = sum of the picks' dxp rows in pick order plus the router's term, added last.
//
// A forward in training mode keeps what this needs: the pre-activation rows g and u (one buffer
// [rows, 2*d_ff], g in the left half), h, yp and the routing.
//
// bf16 layers: every product runs on pairs of SMs (experts_sm100_pair.cu, experts_sm100_wgrad.cu).  The training
// forward's up/gate product stores g and u beside h from one accumulator.  The first product of the
// backward turns dh into dg and du in its epilogue; it and dxp read the
// forward's weights as they lie, as MN-major operands (dxp = dg * W_gate + du * W_up is ONE product with two sources), so
// there are no transposed copies to refresh when the weights change: on the Mixtral-shaped layer those were 2.8 GB of
// memory and three passes over the weights after every omoe_set_weights.  The weight-gradient products reduce over an
// expert's rows and read the activations in place; padding rows are zeroed in xp and dyp, hence zero in everything
// derived from them.
// fp32 layers: the CUDA-core products of experts_f32.cu, which skip padding rows.
#include <stdlib.h>
#include <string.h>

#include <new>
#include <type_traits>

#include "backward.cuh"
#include "common.cuh"
#include "ep.cuh"

namespace omoe {

struct BwState {
    bool training;
    bool fwd_valid;   // the last forward ran in training mode and its saved rows are intact
    int fwd_T;
    float aux_coef;   // weight of the auxiliary load-balancing loss in the objective (0: none)
    float *aux_ps;    // [E] column sums of the router probabilities (omoe_get_aux_loss)
    void *dxn;        // [t_max, d] gradient of the normalised rows (block form), io dtype
    float *inv_rms;   // [t_max] 1/rms of every row (block form)
    void *gu;         // [rows_cap, 2*dff] g | u (compute dtype)
    void *dyp;        // [rows_cap, d]
    void *dgu;        // [rows_cap, 2*dff] dg | du
    void *dxp;        // [rows_cap, d]
    float *dgw;       // [t_max*k] gradient of the gate weights
    void **dyp_table, **dxp_table;  // device [world]: every rank's dyp / dxp buffer (entry `rank` is this GPU's)
    bool own_grad_rows;  // dyp, dxp and the tables were allocated here (one GPU); else they belong to the transport
    float *dl;        // [t_max, E] gradient of the logits
    float *dwr_part;  // [slices][E][d] partial sums of d W_router
    int dwr_slices;
    // gradients (fp32)
    float *d_router, *d_bias, *d_gate, *d_up, *d_down;
    // tensor maps of the bf16 products
    PairMaps up, back, dxp_maps;  // up/gate keeping g and u; dyp * W_down and SwiGLU's backward; dg * W_gate + du * W_up
    WgradMaps w_down, w_gu;
};

namespace {

// ---- combine backward + router backward: one warp per token ---------------------------------------
// dyp[pos_j] = w_j * dy[t];  d w_j = <dy[t], yp[pos_j]>;  then lane 0 turns the k values d w into the
// E values d logits (gate renormalisation, softmax_back), serially and in index order like softmax_back itself.
// With expert parallelism the yp row is read from, and the dyp row written to, the buffers of the rank that
// owns the pick's expert (peer loads and stores); the last block to finish raises "rows have landed" on
// every rank, as the forward's dispatch does.
template <typename YT, typename OT>
__global__ void __launch_bounds__(256)
combine_bwd_kernel(const OT *__restrict__ dy, void *const *__restrict__ yp_table, void *const *__restrict__ dyp_table,
                   int e_local, EpSignal sig, int32_t *ticket, const int32_t *__restrict__ pos, const int32_t *__restrict__ topk_idx,
                   const float *__restrict__ topk_w, const float *__restrict__ logits, float *__restrict__ dgw,
                   float *__restrict__ dl, int T, int d, int k, int E, int renorm, float aux_c,
                   const int32_t *__restrict__ counts) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t < T) {
    float dw[kMaxTopK];
    for (int j = 0; j < k; j++) {
        const int r = pos[(size_t)t * k + j];
        const int q = topk_idx[(size_t)t * k + j] / e_local;  // rank that owns the pick's expert
        const YT *yp = static_cast<const YT *>(yp_table[q]);
        YT *dyp = static_cast<YT *>(dyp_table[q]);
        const float w = topk_w[(size_t)t * k + j];
        float acc = 0.f;
        // r < 0: the pick has no row (a refused expert-parallel step); nothing is read or written for it
        for (int c = lane * 8; r >= 0 && c < d; c += 256) {
            float a[8], y[8], o[8];
            load8(dy + (size_t)t * d + c, a);
            load8(yp + (size_t)r * d + c, y);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                acc = fmaf(a[i], y[i], acc);
                o[i] = w * a[i];
            }
            store8(dyp + (size_t)r * d + c, o);
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        dw[j] = acc;
    }
    if (lane == 0) {
        const float *lg = logits + (size_t)t * E;
        float *out = dl + (size_t)t * E;
        // softmax of the row, three passes (SoftmaxKernel.cu:5-24)
        float mx = lg[0];
        for (int e = 1; e < E; e++) mx = fmaxf(mx, lg[e]);
        float sum = 0.f;
        for (int e = 0; e < E; e++) sum += expf(lg[e] - mx);
        float ssum = 0.f, dot = 0.f;
        for (int j = 0; j < k; j++) {
            dgw[(size_t)t * k + j] = dw[j];
            ssum += expf(lg[topk_idx[(size_t)t * k + j]] - mx) / sum;
            dot += dw[j] * topk_w[(size_t)t * k + j];
        }
        // d p: the picks' terms, plus aux_c * f_e on every expert when the auxiliary loss is on (f_e = share
        // of the step's picks that went to e; aux_c = coef * E / T).  softmax_back: sum_i p_i dp_i, then
        // (dp_i - sum) * p_i.
        const float inv_picks = 1.0f / ((float)T * (float)k);
        float pd = 0.f;
        if (aux_c != 0.f)
            for (int e = 0; e < E; e++) pd += (expf(lg[e] - mx) / sum) * (aux_c * ((float)counts[e] * inv_picks));
        for (int j = 0; j < k; j++) {
            const float p = expf(lg[topk_idx[(size_t)t * k + j]] - mx) / sum;
            const float dp = renorm ? (dw[j] - dot) / ssum : dw[j];
            pd += p * dp;
        }
        for (int e = 0; e < E; e++) {
            const float a = aux_c != 0.f ? aux_c * ((float)counts[e] * inv_picks) : 0.f;
            out[e] = (a - pd) * (expf(lg[e] - mx) / sum);
        }
        for (int j = 0; j < k; j++) {
            const int e = topk_idx[(size_t)t * k + j];
            const float p = expf(lg[e] - mx) / sum;
            const float a = aux_c != 0.f ? aux_c * ((float)counts[e] * inv_picks) : 0.f;
            const float dp = (renorm ? (dw[j] - dot) / ssum : dw[j]) + a;
            out[e] = (dp - pd) * p;
        }
    }
    }  // t < T
    if (sig.flags != nullptr) {
        // make this block's rows visible system-wide, take a ticket, and let the last block tell every rank
        __threadfence_system();
        __syncthreads();
        __shared__ int s_last;
        if (threadIdx.x == 0) s_last = (atomicAdd(ticket, 1) == (int)gridDim.x - 1);
        __syncthreads();
        if (s_last && (int)threadIdx.x < sig.world) {
            __threadfence_system();
            uint32_t *f = sig.flags[threadIdx.x] + sig.rank;
            asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(f), "r"(*sig.seq) : "memory");
        }
        if (s_last && threadIdx.x == 0) *ticket = 0;  // every block has arrived: zero for the next user
    }
}

// ps[e] = sum_t softmax(logits[t, :])[e]: one block per expert, threads stride the tokens, fixed tree at the end.
__global__ void __launch_bounds__(256)
prob_colsum_kernel(const float *__restrict__ logits, float *__restrict__ ps, int T, int E) {
    __shared__ float s[256];
    const int e = blockIdx.x;
    float acc = 0.f;
    for (int t = threadIdx.x; t < T; t += 256) {
        const float *lg = logits + (size_t)t * E;
        float mx = lg[0];
        for (int i = 1; i < E; i++) mx = fmaxf(mx, lg[i]);
        float sum = 0.f;
        for (int i = 0; i < E; i++) sum += expf(lg[i] - mx);
        acc += expf(lg[e] - mx) / sum;
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o >= 1; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) ps[e] = s[0];
}

// dx[t] = ((dxp[pos_0] + dxp[pos_1]) + ...) + sum_e dl[t,e] * W_r[e,:]   (one warp per token)
// With expert parallelism the dxp rows are read from their owners' buffers once every owner has raised
// "outputs ready" for this step (bounded wait).
template <typename YT, typename OT>
__global__ void __launch_bounds__(256)
dx_kernel(void *const *__restrict__ dxp_table, int e_local, const int32_t *__restrict__ topk_idx, EpWait wait,
          int32_t *dev_err, const int32_t *__restrict__ pos, const float *__restrict__ dl,
          const float *__restrict__ w_r, OT *__restrict__ dx, int T, int d, int k, int E) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float s_dl[];  // [warps][E]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (wait.flags != nullptr) {
        if ((int)threadIdx.x < wait.world) ep_wait_flag(wait.flags + threadIdx.x, *wait.seq, wait.timeout_ns, dev_err);
        __syncthreads();
    }
    if (t >= T) return;
    float *my = s_dl + warp * E;
    for (int e = lane; e < E; e += 32) my[e] = dl[(size_t)t * E + e];
    __syncwarp();
    for (int c = lane * 8; c < d; c += 256) {
        float acc[8];
        for (int j = 0; j < k; j++) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            const YT *dxp = static_cast<const YT *>(dxp_table[topk_idx[(size_t)t * k + j] / e_local]);
            const int r = pos[(size_t)t * k + j];
            if (r >= 0) load8(dxp + (size_t)r * d + c, v);  // r < 0: no row (a refused expert-parallel step)
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = (j == 0) ? v[i] : acc[i] + v[i];
        }
        float r[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int e = 0; e < E; e++) {
            float w[8];
            load8(w_r + (size_t)e * d + c, w);
            const float g = my[e];
#pragma unroll
            for (int i = 0; i < 8; i++) r[i] = fmaf(g, w[i], r[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] += r[i];
        store8(dx + (size_t)t * d + c, acc);
    }
}

__device__ __forceinline__ void ld_pair(const float *p, float &a, float &b) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    a = v.x;
    b = v.y;
}
__device__ __forceinline__ void ld_pair(const __nv_bfloat16 *p, float &a, float &b) {
    const uint32_t v = *reinterpret_cast<const uint32_t *>(p);
    a = __uint_as_float(v << 16);
    b = __uint_as_float(v & 0xffff0000u);
}

// d W_router[e, c] = sum_t dl[t, e] * x[t, c].  A block owns 512 columns (two per thread), one slice of the tokens and
// eight experts, whose dl values it keeps in shared memory; the kernel is all load latency, so a thread requests the x
// values of 16 tokens before it uses the first (4096 tokens, d 1024, 8 experts: 30 -> 11 us against one column and one token at
// a time).  Partials go to part[slice][E][d]; a second kernel adds
// the slices in order, so the sum has one fixed order.
constexpr int kDwrExperts = 8, kDwrTokens = 64;
template <typename XT>
__global__ void __launch_bounds__(256)
dwr_partial_kernel(const XT *__restrict__ x, const float *__restrict__ dl, float *__restrict__ part, int T, int d,
                   int E, int slices) {
    pdl_trigger();
    pdl_wait();
    __shared__ float s_dl[kDwrTokens][kDwrExperts];
    const int c = blockIdx.x * 512 + threadIdx.x * 2;
    const int e0 = blockIdx.z * kDwrExperts;
    const int per = (T + slices - 1) / slices;
    const int t0 = blockIdx.y * per, t1 = min(T, t0 + per);
    float a0[kDwrExperts] = {}, a1[kDwrExperts] = {};
    for (int tb = t0; tb < t1; tb += kDwrTokens) {
        __syncthreads();
        for (int i = threadIdx.x; i < kDwrTokens * kDwrExperts; i += 256) {
            const int t = tb + i / kDwrExperts, e = e0 + i % kDwrExperts;
            s_dl[i / kDwrExperts][i % kDwrExperts] = (t < t1 && e < E) ? dl[(size_t)t * E + e] : 0.f;
        }
        __syncthreads();
        if (c >= d) continue;  // d is a multiple of 8: a pair of columns is whole or absent
        const int nt = min(kDwrTokens, t1 - tb);
        for (int q = 0; q < nt; q += 16) {
            float x0[16], x1[16];
#pragma unroll
            for (int u = 0; u < 16; u++)
                if (q + u < nt) ld_pair(x + (size_t)(tb + q + u) * d + c, x0[u], x1[u]);
#pragma unroll
            for (int u = 0; u < 16; u++)
                if (q + u < nt) {
#pragma unroll
                    for (int i = 0; i < kDwrExperts; i++) {
                        const float g = s_dl[q + u][i];
                        a0[i] = fmaf(g, x0[u], a0[i]);
                        a1[i] = fmaf(g, x1[u], a1[i]);
                    }
                }
        }
    }
    if (c < d) {
#pragma unroll
        for (int i = 0; i < kDwrExperts; i++)
            if (e0 + i < E)
                *reinterpret_cast<float2 *>(part + ((size_t)blockIdx.y * E + e0 + i) * d + c) = make_float2(a0[i], a1[i]);
    }
}

__global__ void __launch_bounds__(256)
dwr_reduce_kernel(const float *__restrict__ part, float *__restrict__ out, int n, int slices) {
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float acc = 0.f;
#pragma unroll 8
    for (int s = 0; s < slices; s++) acc += part[(size_t)s * n + i];
    out[i] = acc;
}

// d bias[e] = sum_t dl[t, e]: one block per expert, threads stride the tokens, fixed tree at the end.
__global__ void __launch_bounds__(256) dbias_kernel(const float *__restrict__ dl, float *__restrict__ out, int T, int E) {
    pdl_trigger();
    pdl_wait();
    __shared__ float s[256];
    const int e = blockIdx.x;
    float acc = 0.f;
    for (int t = threadIdx.x; t < T; t += 256) acc += dl[(size_t)t * E + e];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o >= 1; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[e] = s[0];
}

// Zero the padding rows of every expert's segment (rows [poffsets[e] + counts[e], poffsets[e+1])) of buf
// [rows, ld] (16-byte vectors; ld is a multiple of 8).  blockIdx.x = expert.
__global__ void __launch_bounds__(256)
zero_pad_rows_kernel(__nv_bfloat16 *__restrict__ buf, int ld, const int32_t *__restrict__ poffsets,
                     const int32_t *__restrict__ counts) {
    pdl_trigger();
    pdl_wait();
    const int e = blockIdx.x;
    const int r0 = poffsets[e] + counts[e], r1 = poffsets[e + 1];
    const int vec_per_row = ld / 8;
    const int64_t total = (int64_t)(r1 - r0) * vec_per_row;
    uint4 *base = reinterpret_cast<uint4 *>(buf + (size_t)r0 * ld);
    for (int64_t i = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.y * blockDim.x)
        base[i] = make_uint4(0u, 0u, 0u, 0u);
}

#define BW_TRY(expr)                                  \
    do {                                              \
        cudaError_t _e = (expr);                      \
        if (_e != cudaSuccess) return _e;             \
    } while (0)

// Programmatic dependent launch along the training step, as along the forward (pdl.cuh): every kernel of it waits before its
// first access.  One GPU only: with expert parallelism kernels without the instructions stand in between.
bool bw_pdl(const omoe_handle *h) { return h->pdl && h->cfg.world == 1; }

// Rows of the step, where this rank alone decides them.
long step_rows(const omoe_handle *h, int T) { return h->cfg.world == 1 ? (long)T * h->cfg.top_k : -1; }

cudaError_t forward_experts(omoe_handle *h, BwState *b, int T, cudaStream_t s, int *n) {
    const int d = h->cfg.d_model, dff = h->cfg.d_ff;
    if (h->cfg.compute_dtype != OMOE_BF16) return f32_forward_experts(h, s, step_rows(h, T), b->gu, n);
    // padding rows hold rows of earlier steps: zero them, so that g, u and h are zero there too and a
    // reduction over blocks of 64 rows (the weight gradients) adds nothing
    const bool pdl = bw_pdl(h);
    BW_TRY(launch_ex(zero_pad_rows_kernel, dim3(h->e_local, 8), dim3(256), 0, s, pdl, static_cast<__nv_bfloat16 *>(h->xp), d,
                     h->ex_poffsets, h->ex_counts));
    BW_TRY(launch_pair(h, s, pdl, PairKind::kUpGateKeep, b->up, dff, d, 64));
    BW_TRY(launch_pair(h, s, pdl, PairKind::kPlain, h->maps.down, d, dff, 32));
    *n += 3;
    return cudaSuccess;
}

template <typename CT, typename OT>
cudaError_t backward_t(omoe_handle *h, BwState *b, const void *x, bool x_is_compute, const void *dy, void *dx, int T,
                       cudaStream_t s, int *n) {
    const int d = h->cfg.d_model, dff = h->cfg.d_ff, El = h->e_local, E = h->cfg.n_experts, k = h->cfg.top_k;
    const int warps = 8, tblocks = ceil_div(T, warps);
    const bool ep = h->cfg.world > 1, pdl = bw_pdl(h);
    EpSignal sig{nullptr, 1, 0, nullptr};
    if (ep) {
        BW_TRY(ep_bw_advance(h, s));  // the backward is a step of its own for the flags
        (*n)++;
        sig = ep_rows_signal(h);
    }
    if (T > 0) {
        BW_TRY(launch_ex(combine_bwd_kernel<CT, OT>, dim3(tblocks), dim3(256), 0, s, pdl, static_cast<const OT *>(dy), h->d_out_table, b->dyp_table, El, sig, h->ticket, h->pos, h->topk_idx,
            h->topk_w, h->logits, b->dgw, b->dl, T, d, k, E, h->cfg.renormalize,
            b->aux_coef != 0.f ? b->aux_coef * (float)E / (float)T : 0.f, h->counts));
    } else {
        BW_TRY(ep_signal_rows(h, s));  // no tokens here: nothing to send, but the owners wait for every rank
    }
    (*n)++;
    if (ep) {
        BW_TRY(ep_wait_rows(h, s));  // every rank's gradient rows for my experts have landed
        (*n)++;
    }
    if constexpr (sizeof(CT) == 2) {
        BW_TRY(launch_ex(zero_pad_rows_kernel, dim3(El, 8), dim3(256), 0, s, pdl, static_cast<CT *>(b->dyp), d, h->ex_poffsets,
                         h->ex_counts));
        (*n)++;
        // dg | du from dh = dyp * W_down; rows up to a multiple of 64, because the weight gradients reduce over blocks of 64 rows
        BW_TRY(launch_pair(h, s, pdl, PairKind::kSwigluBack, b->back, dff, d, 64));
        (*n)++;
        BW_TRY(launch_pair(h, s, pdl, PairKind::kPlainMN2, b->dxp_maps, d, dff, 32));
        (*n)++;
        if (ep) {
            // the input-gradient rows are complete: the token ranks may fetch them while the weight gradients run
            BW_TRY(ep_signal_out(h, s));
            (*n)++;
        }
        // d W_down[e] [d, dff] = dyp_e^T * h_e;  d W_gate[e], d W_up[e] [dff, d] = dg_e^T * xp_e, du_e^T * xp_e
        BW_TRY(launch_wgrad(h, s, b->w_down, 1, d, dff));
        BW_TRY(launch_wgrad(h, s, b->w_gu, 2, dff, d));
        *n += 2;
    } else {
        // dg | du from dyp * W_down, then dxp = dg * W_gate + du * W_up
        BW_TRY(f32_grad_rows(h, s, step_rows(h, T), b->dyp, b->gu, b->dgu, b->dxp, n));
        if (ep) {
            BW_TRY(ep_signal_out(h, s));
            (*n)++;
        }
        // d W_down[e][c][f] = sum_r dyp[r, c] * h[r, f];  d W_gate[e][f][c], d W_up = sum_r dg[r, f], du[r, f] * xp[r, c]
        BW_TRY(f32_wgrad(h, s, b->dyp, d, 0, h->hbuf, 1, d, dff, b->d_down, nullptr));
        BW_TRY(f32_wgrad(h, s, b->dgu, 2 * dff, dff, h->xp, 2, dff, d, b->d_gate, b->d_up));
        *n += 2;
    }
    // router: d W_router = dl^T * x, d bias = column sums of dl
    {
        const int slices = b->dwr_slices;
        dim3 grid((unsigned)ceil_div(d, 512), (unsigned)slices, (unsigned)ceil_div(E, kDwrExperts));
        auto run = [&](auto *xr) {
            using XT = typename std::remove_cv<typename std::remove_pointer<decltype(xr)>::type>::type;
            return launch_ex(dwr_partial_kernel<XT>, grid, dim3(256), 0, s, pdl, xr, b->dl, b->dwr_part, T, d, E, slices);
        };
        // x: the rows the router saw (the caller's rows, or the normalised rows of the block form)
        BW_TRY(x_is_compute ? run(static_cast<const CT *>(x)) : run(static_cast<const OT *>(x)));
        BW_TRY(launch_ex(dwr_reduce_kernel, dim3(ceil_div(E * d, 256)), dim3(256), 0, s, pdl, b->dwr_part, b->d_router, E * d,
                         slices));
        BW_TRY(launch_ex(dbias_kernel, dim3(E), dim3(256), 0, s, pdl, b->dl, b->d_bias, T, E));
        *n += 3;
    }
    if (T > 0) {
        const EpWait wt = ep ? ep_out_wait(h) : EpWait{nullptr, 1, nullptr, 0};
        BW_TRY(launch_ex(dx_kernel<CT, OT>, dim3(tblocks), dim3(256), warps * E * sizeof(float), s, pdl, b->dxp_table, El,
                         h->topk_idx, wt, h->dev_err, h->pos, b->dl, h->w_router, static_cast<OT *>(dx), T, d, k, E));
        (*n)++;
    }
    return cudaSuccess;
}

void free_state(BwState *b) {
    if (!b->own_grad_rows) b->dyp = b->dxp = nullptr, b->dyp_table = b->dxp_table = nullptr;
    void *ptrs[] = {b->dyp_table, b->dxp_table, b->gu, b->dyp, b->dgu, b->dxp, b->dgw, b->dl, b->dwr_part, b->d_router, b->d_bias, b->d_gate, b->d_up, b->d_down, b->aux_ps, b->dxn, b->inv_rms};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete b;
}

}  // namespace

int bw_set_training(omoe_handle *h, int on) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!on) {
        if (b) { b->training = false; b->fwd_valid = false; }
        return OMOE_OK;
    }
    if (b) { b->training = true; return OMOE_OK; }
    b = new (std::nothrow) BwState();
    if (!b) return OMOE_ERR_NOMEM;
    memset(b, 0, sizeof(*b));
    const size_t cs = h->cfg.compute_dtype == OMOE_BF16 ? 2 : 4;
    const size_t rows = (size_t)h->rows_cap, d = h->cfg.d_model, dff = h->cfg.d_ff, El = h->e_local;
    const size_t E = h->cfg.n_experts, tm = h->cfg.t_max, k = h->cfg.top_k;
    b->dwr_slices = (int)(tm >= 4096 ? 64 : (tm >= 256 ? 8 : 1));
    struct { void **p; size_t bytes; } bufs[] = {
        {&b->gu, rows * 2 * dff * cs}, {&b->dgu, rows * 2 * dff * cs}, {(void **)&b->dgw, tm * k * 4},
        {(void **)&b->dl, tm * E * 4}, {(void **)&b->dwr_part, (size_t)b->dwr_slices * E * d * 4},
        {(void **)&b->d_router, E * d * 4}, {(void **)&b->d_bias, E * 4}, {(void **)&b->aux_ps, E * 4}, {(void **)&b->d_gate, El * dff * d * 4},
        {(void **)&b->d_up, El * dff * d * 4}, {(void **)&b->d_down, El * dff * d * 4}};
    bool ok = true;
    for (auto &x : bufs) ok = ok && cudaMalloc(x.p, x.bytes ? x.bytes : 1) == cudaSuccess;
    if (h->cfg.world > 1) {
        // gradient rows cross GPUs: the buffers the peers can reach belong to the transport
        ep_grad_buffers(h, &b->dyp, &b->dxp, &b->dyp_table, &b->dxp_table);
        b->own_grad_rows = false;
    } else {
        b->own_grad_rows = true;
        ok = ok && cudaMalloc(&b->dyp, rows * d * cs) == cudaSuccess && cudaMalloc(&b->dxp, rows * d * cs) == cudaSuccess &&
             cudaMalloc(&b->dyp_table, sizeof(void *)) == cudaSuccess &&
             cudaMalloc(&b->dxp_table, sizeof(void *)) == cudaSuccess;
        if (ok) {
            cudaMemcpy(b->dyp_table, &b->dyp, sizeof(void *), cudaMemcpyHostToDevice);
            cudaMemcpy(b->dxp_table, &b->dxp, sizeof(void *), cudaMemcpyHostToDevice);
        }
    }
    if (!ok) {
        cudaGetLastError();
        free_state(b);
        snprintf(h->err, sizeof(h->err), "omoe_set_training: device allocation of the backward buffers failed");
        return OMOE_ERR_NOMEM;
    }
    // padding rows are read by the row-wise products (their results are never used): keep them finite
    cudaMemset(b->gu, 0, rows * 2 * dff * cs);
    if (b->own_grad_rows) cudaMemset(b->dyp, 0, rows * d * cs);
    cudaMemset(b->dgu, 0, rows * 2 * dff * cs);
    if (cs == 2) {
        typedef __nv_bfloat16 bf;
        bf *gu = static_cast<bf *>(b->gu), *dgu = static_cast<bf *>(b->dgu);
        // weights as [expert][reduction][output feature]: the boxes end with the expert's matrix
        auto weights = [&](CUtensorMap *mp, void *w, uint64_t red, uint64_t out) {
            const uint64_t dims[3] = {out, red, El}, strides[2] = {out, out * red};
            const uint32_t box[3] = {64, 64, 1};
            return encode_map_nd(mp, w, 3, dims, strides, box);
        };
        auto grads = [&](CUtensorMap *mp, float *g, uint64_t M, uint64_t N) {
            const uint64_t dims[3] = {N, M, El}, strides[2] = {N, N * M};
            const uint32_t box[3] = {32, 32, 1};
            return encode_map_nd(mp, g, 3, dims, strides, box, true);
        };
        b->up = h->maps.up;
        bool m = encode_map_bf16(&b->up.o1, gu, rows, dff, 2 * dff, 32) &&
                 encode_map_bf16(&b->up.o2, gu + dff, rows, dff, 2 * dff, 32) &&
                 weights(&b->back.a0, h->w_down, d, dff) &&
                 encode_map_bf16(&b->back.b0, b->dyp, rows, d, d, 128) &&
                 encode_map_bf16(&b->back.b0_32, b->dyp, rows, d, d, 32) &&
                 weights(&b->dxp_maps.a0, h->w_gate, dff, d) && weights(&b->dxp_maps.a1, h->w_up, dff, d) &&
                 encode_map_bf16(&b->dxp_maps.b0, dgu, rows, dff, 2 * dff, 128) &&
                 encode_map_bf16(&b->dxp_maps.b0_32, dgu, rows, dff, 2 * dff, 32) &&
                 encode_map_bf16(&b->dxp_maps.b1, dgu + dff, rows, dff, 2 * dff, 128) &&
                 encode_map_bf16(&b->dxp_maps.b1_32, dgu + dff, rows, dff, 2 * dff, 32) &&
                 encode_map_bf16(&b->dxp_maps.o0, b->dxp, rows, d, d, 32) &&
                 encode_map_bf16(&b->w_down.a0, b->dyp, rows, d, d, 64) &&
                 encode_map_bf16(&b->w_down.b, h->hbuf, rows, dff, dff, 64) && grads(&b->w_down.o0, b->d_down, d, dff) &&
                 encode_map_bf16(&b->w_gu.a0, dgu, rows, dff, 2 * dff, 64) &&
                 encode_map_bf16(&b->w_gu.a1, dgu + dff, rows, dff, 2 * dff, 64) &&
                 encode_map_bf16(&b->w_gu.b, h->xp, rows, d, d, 64) && grads(&b->w_gu.o0, b->d_gate, dff, d) &&
                 grads(&b->w_gu.o1, b->d_up, dff, d);
        b->back.s0 = b->up.o1;  // g, u in; dg, du out
        b->back.s1 = b->up.o2;
        b->back.o0 = b->dxp_maps.b0_32;
        b->back.o1 = b->dxp_maps.b1_32;
        if (!m) {
            free_state(b);
            snprintf(h->err, sizeof(h->err), "omoe_set_training: cuTensorMapEncodeTiled failed");
            return OMOE_ERR_CUDA;
        }
    }
    if (cudaDeviceSynchronize() != cudaSuccess) {
        free_state(b);
        return OMOE_ERR_CUDA;
    }
    b->training = true;
    h->bw = b;
    return OMOE_OK;
}

bool bw_training(const omoe_handle *h) { return h->bw && static_cast<BwState *>(h->bw)->training; }

void bw_forward_invalidate(omoe_handle *h) {
    if (h->bw) static_cast<BwState *>(h->bw)->fwd_valid = false;
}

void bw_forward_empty(omoe_handle *h) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (b && b->training) {
        b->fwd_valid = true;
        b->fwd_T = 0;
    }
}

cudaError_t bw_forward_experts(omoe_handle *h, int T, cudaStream_t s, int *n) {
    BwState *b = static_cast<BwState *>(h->bw);
    cudaError_t e = forward_experts(h, b, T, s, n);
    b->fwd_valid = e == cudaSuccess;
    b->fwd_T = T;
    return e;
}

int bw_backward(omoe_handle *h, const void *x, bool x_is_compute, const void *dy, void *dx, int T, int io_dtype,
                cudaStream_t s, int *launches) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!b || !b->training) {
        snprintf(h->err, sizeof(h->err), "omoe_backward: call omoe_set_training(h, 1) and a forward first");
        return OMOE_ERR_STATE;
    }
    if (h->cfg.world > 1 && !ep_ready(h)) {
        snprintf(h->err, sizeof(h->err), "omoe_backward: call omoe_ep_export / omoe_ep_import on every rank first");
        return OMOE_ERR_STATE;
    }
    if (!b->fwd_valid || b->fwd_T != T) {
        snprintf(h->err, sizeof(h->err), "omoe_backward: no training-mode forward of T=%d rows precedes this call", T);
        return OMOE_ERR_STATE;
    }
    if (T == 0 && h->cfg.world == 1) {  // no rows: every gradient is zero
        const size_t E = h->cfg.n_experts, d = h->cfg.d_model, dff = h->cfg.d_ff, El = h->e_local;
        cudaMemsetAsync(b->d_router, 0, E * d * 4, s);
        cudaMemsetAsync(b->d_bias, 0, E * 4, s);
        cudaMemsetAsync(b->d_gate, 0, El * dff * d * 4, s);
        cudaMemsetAsync(b->d_up, 0, El * dff * d * 4, s);
        cudaMemsetAsync(b->d_down, 0, El * dff * d * 4, s);
        return OMOE_OK;
    }
    cudaError_t e;
    if (h->cfg.compute_dtype == OMOE_BF16)
        e = io_dtype == OMOE_BF16 ? backward_t<__nv_bfloat16, __nv_bfloat16>(h, b, x, x_is_compute, dy, dx, T, s, launches)
                                  : backward_t<__nv_bfloat16, float>(h, b, x, x_is_compute, dy, dx, T, s, launches);
    else
        e = backward_t<float, float>(h, b, x, x_is_compute, dy, dx, T, s, launches);
    if (e != cudaSuccess) {
        snprintf(h->err, sizeof(h->err), "omoe_backward: %s", cudaGetErrorString(e));
        return OMOE_ERR_CUDA;
    }
    // Expert parallel: one backward per forward.  The owners raise "outputs ready" before their weight-gradient
    // kernels, which still read the gradient rows; only the next forward's count exchange orders the peers
    // behind those kernels, so a second backward could overwrite rows that are still being read.
    if (h->cfg.world > 1) b->fwd_valid = false;
    return OMOE_OK;
}

int bw_get_grads(omoe_handle *h, float *d_router, float *d_bias, float *d_gate, float *d_up, float *d_down,
                 cudaStream_t s) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!b) {
        snprintf(h->err, sizeof(h->err), "omoe_get_weight_grads: no backward has run");
        return OMOE_ERR_STATE;
    }
    const size_t E = h->cfg.n_experts, d = h->cfg.d_model, dff = h->cfg.d_ff, El = h->e_local;
    struct { float *dst; const float *src; size_t n; } cp[] = {
        {d_router, b->d_router, E * d}, {d_bias, b->d_bias, E}, {d_gate, b->d_gate, El * dff * d},
        {d_up, b->d_up, El * dff * d}, {d_down, b->d_down, El * dff * d}};
    for (auto &c : cp)
        if (c.dst && cudaMemcpyAsync(c.dst, c.src, c.n * 4, cudaMemcpyDefault, s) != cudaSuccess) {
            snprintf(h->err, sizeof(h->err), "omoe_get_weight_grads: copy failed");
            return OMOE_ERR_CUDA;
        }
    if (cudaStreamSynchronize(s) != cudaSuccess) return OMOE_ERR_CUDA;
    return OMOE_OK;
}

namespace {

// RMSNorm backward of one row per warp, after rmsnorm_backward_kernel2 (src/main/resources/cu/RMSKernel.cu:225-275):
//   rms = sqrtf(sum(x^2)/C + eps);  drms = sum(x * dout * w) * (-1 / (rms^3 * C));
//   dinp = dout * w / rms + drms * x.
// Here dx = dy + dinp (the residual branch of the block adds dy itself) and 1/rms is kept per row for the
// weight gradient, which the reference accumulates with atomics and this build sums in a fixed order.
template <typename OT>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_kernel(const OT *__restrict__ x, const float *__restrict__ gamma, const OT *__restrict__ dxn,
                   const OT *__restrict__ dy, OT *__restrict__ dx, float *__restrict__ inv_rms, float eps, int T,
                   int d) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= T) return;
    const OT *xr = x + (size_t)t * d, *gr = dxn + (size_t)t * d;
    float ss = 0.f, dot = 0.f;
    for (int c = lane * 8; c < d; c += 256) {
        float xv[8], gv[8], wv[8];
        load8(xr + c, xv);
        load8(gr + c, gv);
        load8(gamma + c, wv);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            ss = fmaf(xv[i], xv[i], ss);
            dot = fmaf(xv[i] * gv[i], wv[i], dot);
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        dot += __shfl_xor_sync(0xffffffffu, dot, o);
    }
    const float rms = sqrtf(ss / (float)d + eps);
    const float drms = dot * (-1.0f / (rms * rms * rms * (float)d));
    if (lane == 0) inv_rms[t] = 1.0f / rms;
    for (int c = lane * 8; c < d; c += 256) {
        float xv[8], gv[8], wv[8], dv[8], o[8];
        load8(xr + c, xv);
        load8(gr + c, gv);
        load8(gamma + c, wv);
        load8(dy + (size_t)t * d + c, dv);
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = dv[i] + (gv[i] * wv[i] / rms + drms * xv[i]);
        store8(dx + (size_t)t * d + c, o);
    }
}

// d gamma[c] = sum_t (x[t,c] / rms_t) * dxn[t,c]: a block takes 64 columns (two per lane) of one slice of the tokens, warp w
// every eighth token from w on; the warps' sums are added in order, the partials [slices][d] by dwr_reduce_kernel.
template <typename OT>
__global__ void __launch_bounds__(256)
dgamma_partial_kernel(const OT *__restrict__ x, const OT *__restrict__ dxn, const float *__restrict__ inv_rms,
                      float *__restrict__ part, int T, int d, int slices) {
    __shared__ float s_sum[8][64];
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 64 + lane * 2;
    const int per = (T + slices - 1) / slices;
    const int t0 = blockIdx.y * per, t1 = min(T, t0 + per);
    float a0 = 0.f, a1 = 0.f;
    if (c < d) {  // d is a multiple of 8: a pair of columns is whole or absent
#pragma unroll 4
        for (int t = t0 + warp; t < t1; t += 8) {
            float x0, x1, g0, g1;
            ld_pair(x + (size_t)t * d + c, x0, x1);
            ld_pair(dxn + (size_t)t * d + c, g0, g1);
            const float r = inv_rms[t];
            a0 = fmaf(x0 * r, g0, a0);
            a1 = fmaf(x1 * r, g1, a1);
        }
    }
    s_sum[warp][lane * 2] = a0;
    s_sum[warp][lane * 2 + 1] = a1;
    __syncthreads();
    const int col = blockIdx.x * 64 + threadIdx.x;
    if (threadIdx.x < 64 && col < d) {
        float acc = s_sum[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < 8; w++) acc += s_sum[w][threadIdx.x];
        part[(size_t)blockIdx.y * d + col] = acc;
    }
}

template <typename OT>
cudaError_t block_tail_t(omoe_handle *h, BwState *b, const void *x, const float *gamma, float eps, const void *dy,
                         void *dx, float *dgamma, int T, cudaStream_t s, int *n) {
    const int d = h->cfg.d_model, slices = b->dwr_slices;
    const bool pdl = bw_pdl(h);
    const OT *xr = static_cast<const OT *>(x), *dxn = static_cast<const OT *>(b->dxn);
    if (T > 0)
        BW_TRY(launch_ex(rmsnorm_bwd_kernel<OT>, dim3(ceil_div(T, 8)), dim3(256), 0, s, pdl, xr, gamma, dxn,
                         static_cast<const OT *>(dy), static_cast<OT *>(dx), b->inv_rms, eps, T, d));
    // the partial buffer of the router's weight gradient is free again by now ([slices][E][d] >= [slices][d])
    BW_TRY(launch_ex(dgamma_partial_kernel<OT>, dim3(ceil_div(d, 64), slices), dim3(256), 0, s, pdl, xr, dxn, b->inv_rms,
                     b->dwr_part, T, d, slices));
    BW_TRY(launch_ex(dwr_reduce_kernel, dim3(ceil_div(d, 256)), dim3(256), 0, s, pdl, b->dwr_part, dgamma, d, slices));
    *n += 3;
    return cudaSuccess;
}

}  // namespace

// Backward of y = x + MoE(rmsnorm(x) * gamma): the layer's backward on the normalised rows the forward kept,
// then the RMSNorm backward, with the residual branch's dy added in the same pass.
int bw_backward_block(omoe_handle *h, const void *x, const float *gamma, float eps, const void *dy, void *dx,
                      float *dgamma, int T, int io_dtype, cudaStream_t s, int *launches) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!b || !b->training) {
        snprintf(h->err, sizeof(h->err), "omoe_backward_block: call omoe_set_training(h, 1) and a forward first");
        return OMOE_ERR_STATE;
    }
    if (!b->dxn) {
        const size_t bytes = (size_t)h->cfg.t_max * h->cfg.d_model * 4;
        if (cudaMalloc(&b->dxn, bytes) != cudaSuccess || cudaMalloc(&b->inv_rms, (size_t)h->cfg.t_max * 4) != cudaSuccess) {
            cudaGetLastError();
            snprintf(h->err, sizeof(h->err), "omoe_backward_block: device allocation failed");
            return OMOE_ERR_NOMEM;
        }
    }
    int rc = bw_backward(h, h->xn, true, dy, b->dxn, T, io_dtype, s, launches);
    if (rc != OMOE_OK) return rc;
    cudaError_t e = io_dtype == OMOE_BF16
                        ? block_tail_t<__nv_bfloat16>(h, b, x, gamma, eps, dy, dx, dgamma, T, s, launches)
                        : block_tail_t<float>(h, b, x, gamma, eps, dy, dx, dgamma, T, s, launches);
    if (e != cudaSuccess) {
        snprintf(h->err, sizeof(h->err), "omoe_backward_block: %s", cudaGetErrorString(e));
        return OMOE_ERR_CUDA;
    }
    return OMOE_OK;
}

int bw_set_aux(omoe_handle *h, float coef) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!b) {
        snprintf(h->err, sizeof(h->err), "omoe_set_aux_loss: switch training mode on first");
        return OMOE_ERR_STATE;
    }
    b->aux_coef = coef;
    return OMOE_OK;
}

int bw_aux_loss(omoe_handle *h, float *loss_host, cudaStream_t s, const int32_t *counts_host) {
    BwState *b = static_cast<BwState *>(h->bw);
    if (!b) {
        snprintf(h->err, sizeof(h->err), "omoe_get_aux_loss: switch training mode on first");
        return OMOE_ERR_STATE;
    }
    const int T = h->last_T, E = h->cfg.n_experts, k = h->cfg.top_k;
    *loss_host = 0.f;
    if (T == 0) return OMOE_OK;
    prob_colsum_kernel<<<E, 256, 0, s>>>(h->logits, b->aux_ps, T, E);
    float ps[kMaxExperts];
    int32_t cnt[kMaxExperts];
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(ps, b->aux_ps, sizeof(float) * E, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        (!counts_host && cudaMemcpyAsync(cnt, h->counts, sizeof(int32_t) * E, cudaMemcpyDeviceToHost, s) != cudaSuccess) ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        snprintf(h->err, sizeof(h->err), "omoe_get_aux_loss: CUDA error");
        return OMOE_ERR_CUDA;
    }
    if (!counts_host) counts_host = cnt;
    float loss = 0.f;
    for (int e = 0; e < E; e++) loss += ((float)counts_host[e] / ((float)T * (float)k)) * (ps[e] / (float)T);
    *loss_host = (float)E * loss;
    return OMOE_OK;
}

void bw_destroy(omoe_handle *h) {
    if (h->bw) free_state(static_cast<BwState *>(h->bw));
    h->bw = nullptr;
}

}  // namespace omoe
