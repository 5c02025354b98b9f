// Routing and dispatch of a decode step (a handful of tokens) in ONE launch.
//
// With T <= 8 the separate router, scan and dispatch kernels are pure launch and
// dependent-load latency (about 40 us for work that takes a few).  Here a block owns
// one expert: all its threads bring the router row into shared memory, warp t folds it against token t.  The rows of the
// router are cold (the expert weights of the step before have passed through L2) and the step is too short to hide it, so
// what counts is round trips to memory: every SM fetches one row, all of it at once, and every load of a thread is
// requested before the first is used.  The block that finishes last picks the experts, turns the
// picks into counts, offsets, row positions and the tile table, and copies the token rows into the dispatch buffer.
// A step of one token on few experts and narrow rows runs in one block instead, a warp per expert: there is nothing to join then
// (launch_pl).
// Measured against a block per token whose warps walked the experts (loads inside a bounds branch, each waited for before
// the next): step of 8 tokens, d 2048, 64 experts 144.5 -> 124 us (this kernel 33 -> 14 us), of one token, d 4096, 8 experts
// 132 -> 126 us.
// Outputs are the same arrays, with the same contents, as the
// three-kernel path; the logits follow the same fixed reduction tree, so the
// routing stays bit-exact.  Single GPU only (expert-parallel steps need the
// count exchange between the two halves).
#include "route_small.cuh"

namespace omoe {

namespace {

using namespace small;

// Eight row elements as they lie in memory: the load and its use are apart.
template <typename XT>
struct Raw8;
template <>
struct Raw8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float *p) {
        a = __ldg(reinterpret_cast<const float4 *>(p));
        b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    }
    __device__ __forceinline__ void get(float (&v)[8]) const {
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
};
template <>
struct Raw8<__nv_bfloat16> {
    uint4 a;
    __device__ __forceinline__ void load(const __nv_bfloat16 *p) { a = __ldg(reinterpret_cast<const uint4 *>(p)); }
    __device__ __forceinline__ void get(float (&v)[8]) const { unpack8(a, v); }
};

constexpr int kRowChunk = 4096;  // columns of a router row in shared memory at a time
constexpr int kAhead = 8;        // 256-column pieces of a token row requested together

// PL: experts per lane of a warp (ceil(E/32)).
template <int PL, typename XT>
__global__ void __launch_bounds__(256)
route_small_kernel(const XT *__restrict__ x, const float *__restrict__ w_r, const float *__restrict__ bias, int T, int d,
                   int E, int k, int renorm, float *__restrict__ logits, int32_t *__restrict__ topk_idx,
                   float *__restrict__ topk_w, int32_t *__restrict__ counts, int32_t *__restrict__ offsets,
                   int32_t *__restrict__ poffsets, int32_t *__restrict__ tile_expert, int max_tiles,
                   int32_t *__restrict__ pos, __nv_bfloat16 *__restrict__ xp, int32_t *ticket) {
    __shared__ float sl[kSmallMaxTokens][kMaxExperts];
    __shared__ int32_t s_idx[kSmallMaxPicks], s_rank[kSmallMaxPicks], s_pos[kSmallMaxPicks];
    __shared__ int32_t s_cnt[kMaxExperts], s_poff[kMaxExperts + 1];
    __shared__ __align__(16) float s_w[kRowChunk];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_trigger();
    pdl_wait();  // the step before may still be reading the routing arrays this kernel overwrites

    const bool alone = gridDim.x == 1 && T == 1;  // one block does it all: a warp per expert, nothing to join
    if (alone) {
        for (int e = warp; e < E; e += 8) {
            const float *wr = w_r + (size_t)e * d;
            float even = 0.f, odd = 0.f;
            for (int i0 = lane * 8; i0 < d; i0 += kAhead * 256) {
                Raw8<XT> xv[kAhead];
                Raw8<float> wv[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; u++) {  // addresses past the row are clamped, not branched around
                    xv[u].load(x + min(i0 + u * 256, d - 8));
                    wv[u].load(wr + min(i0 + u * 256, d - 8));
                }
#pragma unroll
                for (int u = 0; u < kAhead; u++) {
                    if (i0 + u * 256 >= d) break;
                    float v[8], w[8];
                    xv[u].get(v);
                    wv[u].get(w);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        even = fmaf(v[j], w[j], even);
                        odd = fmaf(v[j + 1], w[j + 1], odd);
                    }
                }
            }
            float v = even + odd;
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, m);
            if (lane == 0) {
                if (bias != nullptr) v = v + __ldg(bias + e);
                sl[0][e] = logits[e] = v;
            }
        }
        __syncthreads();
    } else {
        // ---- logit of expert blockIdx.x for token `warp` (the reduction tree of router.cu) ----
        const int e = blockIdx.x;
        const XT *xr = x + (size_t)min(warp, T - 1) * d;
        float even = 0.f, odd = 0.f;  // the two chains of the reduction rule
        for (int c0 = 0; c0 < d; c0 += kRowChunk) {
            const int len = min(kRowChunk, d - c0);
            if (c0 > 0) __syncthreads();  // everyone is done with the chunk before
            for (int i = tid * 4; i < len; i += 1024)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 static_cast<uint32_t>(__cvta_generic_to_shared(s_w + i))),
                             "l"(w_r + (size_t)e * d + c0 + i)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
            Raw8<XT> cur[kAhead], nxt[kAhead];
            // addresses past the chunk are clamped, not branched around
            auto request = [&](Raw8<XT> (&r)[kAhead], int i0) {
#pragma unroll
                for (int u = 0; u < kAhead; u++) r[u].load(xr + c0 + min(i0 + u * 256, len - 8));
            };
            if (warp < T) request(cur, lane * 8);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (warp < T) {
                for (int i0 = lane * 8; i0 < len; i0 += kAhead * 256) {
                    request(nxt, i0 + kAhead * 256);
#pragma unroll
                    for (int u = 0; u < kAhead; u++) {
                        const int i = i0 + u * 256;
                        if (i >= len) break;
                        const float4 a = *reinterpret_cast<const float4 *>(s_w + i), b = *reinterpret_cast<const float4 *>(s_w + i + 4);
                        const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                        float v[8];
                        cur[u].get(v);
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            even = fmaf(v[j], w[j], even);
                            odd = fmaf(v[j + 1], w[j + 1], odd);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kAhead; u++) cur[u] = nxt[u];
                }
            }
        }
        if (warp < T) {
            float v = even + odd;
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, m);
            if (lane == 0) logits[(size_t)warp * E + e] = bias != nullptr ? v + __ldg(bias + e) : v;
        }
    }
    if (!alone) {
        // ---- the block that finishes last does the rest ----
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = (atomicAdd(ticket, 1) == (int)gridDim.x - 1);
        __syncthreads();
        if (!s_last) return;
        __threadfence();
    }
    if (warp < T) {  // one warp per token
        if (!alone) {
            for (int e = lane; e < E; e += 32) sl[warp][e] = __ldcg(logits + (size_t)warp * E + e);
            __syncwarp();
        }
        int pick;
        float w;
        warp_softmax_topk<PL>(sl[warp], E, k, renorm, lane, pick, w);
        if (lane < k) {
            s_idx[warp * k + lane] = pick;
            topk_idx[(size_t)warp * k + lane] = pick;
            topk_w[(size_t)warp * k + lane] = w;
        }
    }
    const int n = T * k;
    __syncthreads();
    rank_picks(n, E, s_idx, s_rank, s_cnt);
    __syncthreads();
    if (warp == 0) {
        int off = 0, poff = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int c = e < E ? s_cnt[e] : 0, p = (c + kRowAlign - 1) / kRowAlign * kRowAlign;
            int ci = c, pi = p;  // inclusive sums over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int cv = __shfl_up_sync(0xffffffffu, ci, o), pv = __shfl_up_sync(0xffffffffu, pi, o);
                if (lane >= o) { ci += cv; pi += pv; }
            }
            if (e < E) {
                counts[e] = c;
                offsets[e] = off + ci - c;
                poffsets[e] = s_poff[e] = poff + pi - p;
                // at most 8 rows per expert: its segment is one tile or none
                if (c > 0) tile_expert[(poff + pi - p) / kRowAlign] = e;
            }
            off += __shfl_sync(0xffffffffu, ci, 31);
            poff += __shfl_sync(0xffffffffu, pi, 31);
        }
        if (lane == 0) {
            offsets[E] = off;
            poffsets[E] = poff;
            s_poff[E] = poff;
            *ticket = 0;  // ready for the next step
        }
    }
    __syncthreads();
    for (int i = s_poff[E] / kRowAlign + tid; i < max_tiles; i += blockDim.x) tile_expert[i] = -1;
    if (tid < n) {
        const int p = s_poff[s_idx[tid]] + s_rank[tid];
        s_pos[tid] = p;
        pos[tid] = p;
    }
    __syncthreads();
    // copy the token rows to their k places (bf16 rows out; fp32 rows are converted), four loads in flight per thread
    const int vec = d / 8, total = T * vec;  // 8 elements per step
    for (int i0 = tid; i0 < total; i0 += 4 * 256) {
        Raw8<XT> raw[4];
#pragma unroll
        for (int u = 0; u < 4; u++) raw[u].load(x + (size_t)min(i0 + u * 256, total - 1) * 8);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u * 256;
            if (i >= total) break;
            float v[8];
            raw[u].get(v);
            const int tt = i / vec, c = (i - tt * vec) * 8;
            const uint4 o = pack8(v);
            for (int j = 0; j < k; j++)
                *reinterpret_cast<uint4 *>(xp + (size_t)s_pos[tt * k + j] * d + c) = o;
        }
    }
}

template <int PL, typename XT>
cudaError_t launch_pl(omoe_handle *h, const XT *x, int T, cudaStream_t s) {
    const int E = h->cfg.n_experts, per_warp = (E + 7) / 8;
    // One block for one token where its warps' products are at most 1536 columns together, a round trip's loads: joining the blocks
    // (fence, ticket, logits back from L2) costs more than a narrow row's loads. Whole step with one block and with a block per expert, all
    // rows cold: 8 experts top-1 d 512 17.4 us against 19.1, top-2 d 1024 28.0 against 30.4, d 1536 28.2 against 29.5, but d 2040 45.3 against
    // 43.9; 16 experts d 512 24.4 against 25.3, but d 1536 33.1 against 30.3.  Two tokens, 8 experts, d 1024: 44 against 38.
    const bool alone = T == 1 && per_warp * h->cfg.d_model <= 1536;
    return launch_ex(route_small_kernel<PL, XT>, dim3(alone ? 1 : E), dim3(256), 0, s, h->pdl, x, h->w_router, h->router_bias, T,
                     h->cfg.d_model, E, h->cfg.top_k, h->cfg.renormalize, h->logits, h->topk_idx, h->topk_w, h->counts,
                     h->offsets, h->poffsets, h->tile_expert, (int)(h->rows_cap / kRowAlign), h->pos,
                     static_cast<__nv_bfloat16 *>(h->xp), h->ticket);
}

template <typename XT>
cudaError_t launch_typed(omoe_handle *h, const XT *x, int T, cudaStream_t s) {
    const int E = h->cfg.n_experts;
    if (E <= 32) return launch_pl<1, XT>(h, x, T, s);
    if (E <= 64) return launch_pl<2, XT>(h, x, T, s);
    return launch_pl<4, XT>(h, x, T, s);
}

}  // namespace

int route_small_max_tokens() { return kSmallMaxTokens; }

cudaError_t launch_route_small(omoe_handle *h, const void *x, int io_dtype, int T, cudaStream_t s, int *n) {
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) return cudaErrorMisalignedAddress;
    cudaError_t e = io_dtype == OMOE_F32 ? launch_typed<float>(h, static_cast<const float *>(x), T, s)
                                         : launch_typed<__nv_bfloat16>(h, static_cast<const __nv_bfloat16 *>(x), T, s);
    if (e == cudaSuccess) (*n)++;
    return e;
}

}  // namespace omoe
