// Weight gradients of the expert products on Blackwell tensor cores (compute_dtype = OMOE_BF16).
//
// FullyLayer.diff() forms diffW = delta^T * input with one cublasSgemm per layer
// (src/main/java/com/omega/engine/nn/layer/FullyLayer.java:292-301).  Here every expert has its own rows,
// so the product is grouped the other way round from the forward: per expert e
//     C_e [M, N] = sum over the expert's rows r of  A[r, m] * B[r, n]
// with the row index as the reduction.  The activations are stored [rows, features], so in this product the
// reduction index is the SLOW one of both operands: they are "MN-major" tiles for the tensor core.  TMA
// brings 64-feature x 64-row boxes (128-byte swizzle), the shared-memory descriptors say: 64 features contiguous,
// next row of the reduction 128 bytes on, next group of 8 rows 1024 bytes on, next 64 features one box (8 KB) on, and
// the instruction descriptor marks both operands MN-major.  Padding rows of an expert's segment must be zero in the A
// operand and finite in the B operand (backward.cu zeroes them).
//
// A pair of SMs (cluster of two CTAs, tcgen05.mma.cta_group::2) works on a 256 x 256 tile, each CTA bringing 128
// features of either operand: 32 KB per CTA and 64-row block where a CTA with a 128 x 256 tile of its own pulls
// 48 KB.  Pairs walk (matrix, expert, n-tile, m-tile); producer, MMA issuer and accumulator double buffering are those
// of experts_sm100_pair.cu.  The result is fp32 and as large as the weights: each epilogue warp stages 32 x 32
// blocks in the 128-byte swizzle and hands them to TMA stores, so the gradient leaves in full 128-byte lines (a
// thread that owns a row would write it 16 bytes at a time, one sector per lane).  An expert without rows has no K
// blocks: its tiles are written as zeros.
//
// Every mbarrier wait is bounded (sm100_ptx.cuh): when one runs out the kernel raises the device error
// word, lets outstanding copies land, frees its tensor memory and returns.
#include "backward.cuh"
#include "common.cuh"
#include "sm100_pair.cuh"

namespace omoe {

namespace {

using namespace sm100;
constexpr int kStagesW = 6;
constexpr int kAccStagesW = 2;
constexpr int kTmemColsW = 512;
constexpr int kBoxBytesW = 64 * BLOCK_K * 2;      // 64 features x 64 rows: 8 KB
constexpr int kABytesW = 2 * kBoxBytesW;          // this CTA's 128 features of A
constexpr int kStageBytesW = 2 * kABytesW;        // and 128 of B
constexpr int kOutWarpBytesW = 32 * 32 * 4;       // one epilogue warp's staging
constexpr int kSmemBytesW = kStagesW * kStageBytesW + 8 * kOutWarpBytesW + 256 /*barriers*/ + 1024 /*align slack*/;
static_assert(kSmemBytesW <= 227 * 1024, "shared memory of one CTA");
constexpr int kThreadsW = 320;  // warp 0 producer, warp 1 MMA (even CTA), warps 2-9 epilogue

struct WTile {
    int z, e, mt, nt;
};
// m-tiles fastest: neighbouring pairs share the B tile
__device__ __forceinline__ WTile wtile(int tile, int E, int m_tiles, int n_tiles) {
    WTile t;
    const int per_e = m_tiles * n_tiles;
    const int ze = tile / per_e, r = tile - ze * per_e;
    t.z = ze / E;
    t.e = ze - t.z * E;
    t.nt = r / m_tiles;
    t.mt = r - t.nt * m_tiles;
    return t;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsW, 1)
wgrad_kernel(const __grid_constant__ WgradMaps maps, int n_mat, int M, int N, const int32_t *__restrict__ poffsets,
             const int32_t *__restrict__ counts, int E, int32_t *dev_err) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzled tiles start on 1024 bytes; the same in both CTAs
    unsigned char *base_ptr = smem_raw + (base - raw);
    const uint32_t out_stage = base + kStagesW * kStageBytesW;
    const uint32_t bar0 = out_stage + 8 * kOutWarpBytesW;
    unsigned char *bar_ptr = base_ptr + kStagesW * kStageBytesW + 8 * kOutWarpBytesW;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kStagesW + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * kStagesW + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * kStagesW + kAccStagesW + s); };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_ptr + 8 * (2 * kStagesW + 2 * kAccStagesW));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

    pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesW; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < kAccStagesW; s++) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), 16);  // one arrival per epilogue warp of both CTAs
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemColsW)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();  // everything from here on reads what earlier kernels wrote
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int m_tiles = (M + 255) / 256, n_tiles = (N + 255) / 256;
    const int total = n_mat * E * m_tiles * n_tiles;
    const int pair0 = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (warp == 0) {
        // ---------------- producer ----------------
        {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = pair0; ok && tile < total; tile += pairs) {
                const WTile t = wtile(tile, E, m_tiles, n_tiles);
                const int seg0 = poffsets[t.e];
                const int num_kb = (counts[t.e] + BLOCK_K - 1) / BLOCK_K;
                const CUtensorMap *ma = t.z ? &maps.a1 : &maps.a0;
                const int xa = t.mt * 256 + (int)rank * 128, xb = t.nt * 256 + (int)rank * 128;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!warp_wait(empty_bar(stage), phase ^ 1u, abort_flag, dev_err)) { ok = false; break; }
                    if (elect_one()) {
                        const uint32_t sa = base + stage * kStageBytesW;
                        const uint32_t bar = map_to_rank(full_bar(stage), 0);
                        const int y = seg0 + kb * BLOCK_K;
                        if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * kStageBytesW);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            pair_load_2d(sa + i * kBoxBytesW, ma, bar, xa + 64 * i, y);
                            pair_load_2d(sa + kABytesW + i * kBoxBytesW, &maps.b, bar, xb + 64 * i, y);
                        }
                    }
                    __syncwarp();
                    if (++stage == kStagesW) { stage = 0; phase ^= 1u; }
                }
            }
            // The issuer's commits arrive in both CTAs, in their own time: every stage's last one has to be in before this CTA may
            // go (the cluster barrier at the end orders the threads' arrivals, not those of the tensor core).
            for (int i = 0; ok && i < kStagesW; i++) {
                ok = warp_wait(empty_bar(stage), phase ^ 1u, abort_flag, dev_err);
                if (++stage == kStagesW) { stage = 0; phase ^= 1u; }
            }
            if (!ok) {
                // let copies that were already issued land before the CTA retires
                const unsigned long long t0 = globaltimer_ns();
                while (globaltimer_ns() - t0 < 2000000ull) { }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (even CTA, for both) ----------------
        if (rank == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                       ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            int stage = 0, as = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            for (int tile = pair0; ok && tile < total; tile += pairs) {
                const WTile t = wtile(tile, E, m_tiles, n_tiles);
                const int num_kb = (counts[t.e] + BLOCK_K - 1) / BLOCK_K;
                if (!warp_wait(tempty_bar(as), aphase ^ 1u, abort_flag, dev_err)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * 256;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!warp_wait(full_bar(stage), phase, abort_flag, dev_err)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = base + stage * kStageBytesW;
                    const uint64_t adesc = make_mn_desc(sa), bdesc = make_mn_desc(sa + kABytesW);
                    // 16 rows of the reduction are 16 x 128 bytes further on: +128 in 16-byte units
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; k++)
                            pair_mma_bf16(d_tmem, adesc + 128u * k, bdesc + 128u * k, idesc, (kb | k) != 0 ? 1u : 0u);
                        pair_commit(empty_bar(stage));
                    }
                    __syncwarp();
                    if (++stage == kStagesW) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) pair_commit(tfull_bar(as));  // accumulator complete (at once for an expert without rows)
                __syncwarp();
                if (++as == kAccStagesW) { as = 0; aphase ^= 1u; }
            }
        }
    } else {
        // ---------------- epilogue: TMEM -> registers -> shared -> TMA store, each warp on its own ----------------
        // warp%4 selects the 32 TMEM lanes (rows of C) the hardware lets a warp read, (warp-2)/4 a 128-column half
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t stg = out_stage + (warp - 2) * kOutWarpBytesW;
        const uint32_t my_row = stg + lane * 128;
        int as = 0;
        uint32_t aphase = 0;
        for (int tile = pair0; tile < total; tile += pairs) {
            const WTile t = wtile(tile, E, m_tiles, n_tiles);
            const bool empty = counts[t.e] == 0;
            bool ok = mbar_wait(tfull_bar(as), aphase, abort_flag, dev_err);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + as * 256 + half * 128 + ((uint32_t)(quarter * 32) << 16);
            const int m0 = t.mt * 256 + (int)rank * 128 + quarter * 32;
            const CUtensorMap *mo = t.z ? &maps.o1 : &maps.o0;
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
                uint32_t a[32];
                if (!empty) {
                    tc_ld32(t_acc + c, a);
                    tc_wait_ld();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) a[j] = 0u;
                }
                if (c == 96) {  // all of this warp's accumulator reads are done
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_cluster(map_to_rank(tempty_bar(as), 0));
                }
                // the block before must have been read from the staging rows
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int v = 0; v < 8; v++)  // 128-byte swizzle: 16-byte chunk ^ (row % 8)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(my_row + ((v ^ (lane & 7)) << 4)),
                                 "r"(a[4 * v]), "r"(a[4 * v + 1]), "r"(a[4 * v + 2]), "r"(a[4 * v + 3])
                                 : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                const int n0 = t.nt * 256 + half * 128 + c;
                if (lane == 0 && m0 < M && n0 < N) {  // rows and columns past the matrix are clipped by the map
                    tma_store_3d(mo, stg, n0, m0, t.e);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            if (++as == kAccStagesW) { as = 0; aphase ^= 1u; }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    tc_fence_before();
    cluster_sync_all();  // no CTA leaves while its partner's MMAs, arrivals or accumulator reads may still need it
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColsW)
                     : "memory");
    }
}

}  // namespace

cudaError_t launch_wgrad(omoe_handle *h, cudaStream_t s, const WgradMaps &maps, int n_mat, int M, int N) {
    static PerDeviceOnce once;
    bool *done = once.slot();
    if (!done || !*done) {
        cudaError_t e = cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytesW);
        if (e != cudaSuccess) return e;
        if (done) *done = true;
    }
    return launch_ex(wgrad_kernel, dim3(h->sm_count & ~1), dim3(kThreadsW), kSmemBytesW, s, h->pdl && h->cfg.world == 1, maps, n_mat, M, N,
                     h->ex_poffsets, h->ex_counts, h->e_local, h->dev_err);
}

}  // namespace omoe
