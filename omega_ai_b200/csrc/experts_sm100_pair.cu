// Grouped expert products on pairs of SMs (compute_dtype = OMOE_BF16): tcgen05.mma.cta_group::2 with the WEIGHTS as
// the 256-row operand and the expert's token rows as the column operand.
//
//   up/gate:  h  = silu(xp * Wg^T) * (xp * Wu^T)       (training: g and u are stored too)
//   plain:    yp = h * Wd^T                            (K-major weights, as they lie)
//   back:     dg, du from dh = dyp * Wd                (the weights with the reduction along their slow index; dh stays here)
//   plain MN: dxp = dg * Wg + du * Wu                  (two such sources, one accumulator)
//
// What bounds it: the tensor pipe on large steps, and on the way there the shared-memory fill (L2 -> SM).  A CTA with a
// 128 x 256 tile of its own pulls 48 KB per 64-deep k-block; a pair shares one 256 x 256 tile, each CTA holding half of
// either operand, and pulls 32 KB for the same arithmetic.  A pair whose 256 rows are token rows cannot span two
// experts, so an odd number of 128-row tiles wastes half a pair; weight rows are always there in full, and the
// column operand may have any width that is a multiple of 32, so the tokens of an expert are cut into tiles of
// equal width (<= 256) and the padding work of a 128-row token tile goes away with it.
//
// Measured against the kernel of experts_sm100.cu (128 x 256 tiles, one CTA each): 4096 tokens, d 1024, d_ff 2816, 8 experts top-2
// up/gate 97 -> 73.5 us, down 45 -> 42.9; whole layer with 1531 tokens, d 1544, d_ff 4104, 12 experts top-3 358 -> 302 us; with 16384
// tokens, d 4096, d_ff 14336, under the power cap 10.50 -> 9.90 ms where one side's runs differ by 2 to 6 %.  That kernel stays for expert
// parallelism, whose rows it waits for and sends, and for a down product that it runs in one round (launch_experts_bf16).
//
// The accumulator comes out transposed (tensor-memory lane = output feature, column = token).  For up/gate the A tile
// interleaves 8 gate rows with 8 up rows (one 4-D tensor map over both matrices, which lie back to back), so
// the two halves of a SiLU product sit in lanes l and l^8 of one warp; one shuffle per pair of tokens brings them
// together, one more packs neighbouring features into a word, and the rows leave through swizzled staging and
// TMA stores of 32-token boxes.
//
// Roles per CTA: warp 0 producer (TMA), warp 1 of the even CTA issues the MMAs for both, the others epilogue.  A load
// signals the even CTA's "full" barrier; commits free the stage in both CTAs.  All mbarrier waits are bounded
// (sm100_ptx.cuh): when one runs out the kernel raises the device error word, lets outstanding copies land and leaves;
// the cluster barriers are reached by every thread whatever happened before.
#include "common.cuh"
#include "pair.cuh"
#include "sm100_pair.cuh"

namespace omoe {

namespace {

using namespace sm100;
constexpr int kAccStagesP = 2;
constexpr int kTmemColsP = 512;
constexpr int kABytesP = 128 * BLOCK_K * 2;       // 16 KB: this CTA's half of the 256 weight rows
constexpr int kStageBytesP = 2 * kABytesP;        // and up to 128 of the tile's (<= 256) token rows
// Ring depth and epilogue of a kind.  The epilogue is kParts groups of four warps, each with 256 / kParts of a tile's token
// columns, kPass of them staged at a time.  Six stages and 2 x 16 KB of results fit; the epilogues that move three
// results, or two rows in and two out, take a stage for their staging (five stages instead of six cost 1 % of a forward) and have
// twice the warps: with eight, shared-memory words, exponentials and arithmetic of a pass follow one another and a tile's
// epilogue outlasts a reduction of 1024 (training step of 4096 tokens, d 1024, d_ff 2816 764 us, with sixteen 727).  Sixteen gain
// nothing for the other two.
// Both epilogues are bound by instructions there. The exponential and the divisions of full accuracy are 13 of 98 us in the forward and 36 of
// 114 us in the backward kernel; with __expf and __fdividef in their place the step is some 40 us shorter, but the SiLU of a large negative
// g is off or zero (sm100_ptx.cuh).
template <PairKind KIND>
struct PairCfg {
    static constexpr bool kWide = KIND == PairKind::kUpGateKeep || KIND == PairKind::kSwigluBack;
    static constexpr int kStages = kWide ? 5 : 6;
    static constexpr int kParts = kWide ? 4 : 2;
    static constexpr int kPass = kWide ? 32 : (KIND == PairKind::kUpGate ? 128 : 64);
    // 128-byte rows (64 features of a token) staged per token: h; h, g, u; g, u of two feature halves; two feature halves
    static constexpr int kRows = KIND == PairKind::kUpGate ? 1 : (KIND == PairKind::kUpGateKeep ? 3 : (KIND == PairKind::kSwigluBack ? 4 : 2));
    static constexpr int kPartBytes = kPass * kRows * 128;
    static constexpr int kThreads = 64 + kParts * 128;
};
constexpr int kTableInts = 3 * kMaxExperts + 2;   // token-tile prefix, counts, first rows of the local experts; narrow step
constexpr int kBarBytesP = 256;
// A step whose experts hold at most 64 (128) rows each is bound by the weights' way from HBM: its stages need room for 32 (64)
// token rows per CTA, not 128, and nine (eight) of those take the ring's place (64 tokens, d 4096, d_ff 14336, 8 experts: 494 ->
// 479 us; 8 tokens, d 2048, 64 experts: 124.3 -> 122.1 us; 256 tokens of the first layer: 517 -> 502 us.  Requesting the two
// halves of a weight row's 256 bytes together instead: 3 % slower.)
constexpr int kStagesNarrow = 9, kStageBytesNarrow = kABytesP + 4096;
constexpr int kStagesMid = 8, kStageBytesMid = kABytesP + 8192;
template <PairKind KIND>
constexpr int pair_smem_bytes() {
    return PairCfg<KIND>::kStages * kStageBytesP + PairCfg<KIND>::kParts * PairCfg<KIND>::kPartBytes + kBarBytesP + kTableInts * 4 + 1024 /*align slack*/;
}
static_assert(kStagesNarrow * kStageBytesNarrow <= 6 * kStageBytesP && kStagesMid * kStageBytesMid <= 6 * kStageBytesP, "the narrow rings lie in the wide one's place");
static_assert(pair_smem_bytes<PairKind::kUpGate>() <= 227 * 1024 && pair_smem_bytes<PairKind::kUpGateKeep>() <= 227 * 1024 &&
                  pair_smem_bytes<PairKind::kSwigluBack>() <= 227 * 1024,
              "shared memory of one CTA");
constexpr int kTokensMax = 256;  // token columns of a tile

// Tokens of one tile of an expert with `cnt` rows when tiles hold at most `cap` (a multiple of 32): the expert's
// ceil(cnt / cap) tiles get the same width, rounded up to the 32 columns an MMA of a pair takes.
__device__ __forceinline__ int tile_width(int cnt, int cap) {
    const int n = (cnt + cap - 1) / cap;
    return ((cnt + n - 1) / n + 31) / 32 * 32;
}

struct PairTile {
    int e, row0, n, ft;  // expert, first row, token columns (multiple of 32), feature tile
};

template <PairKind KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<KIND>::kThreads, 1)
pair_gemm_kernel(const __grid_constant__ PairMaps maps, int n_out, int K, const int32_t *__restrict__ poffsets,
                 const int32_t *__restrict__ counts, int E, int cap, int row_round, int kband, int32_t *dev_err) {
    constexpr bool kGate = KIND == PairKind::kUpGate || KIND == PairKind::kUpGateKeep;
    constexpr bool kMN = KIND == PairKind::kSwigluBack || KIND == PairKind::kPlainMN2;
    constexpr int kRingStages = PairCfg<KIND>::kStages, kStagesMax = kRingStages == 6 ? kStagesNarrow : kRingStages, kParts = PairCfg<KIND>::kParts, kPass = PairCfg<KIND>::kPass;
    constexpr int kPartBytes = PairCfg<KIND>::kPartBytes, kPartCols = kTokensMax / kParts;
    constexpr int kFeatPair = kGate ? 128 : 256;  // output features of a pair's tile
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzled tiles start on 1024 bytes; the same in both CTAs
    unsigned char *base_ptr = smem_raw + (base - raw);
    const uint32_t out_stage = base + kRingStages * kStageBytesP;
    const uint32_t bar0 = out_stage + kParts * kPartBytes;
    unsigned char *bar_ptr = base_ptr + kRingStages * kStageBytesP + kParts * kPartBytes;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kStagesMax + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * kStagesMax + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * kStagesMax + kAccStagesP + s); };
    auto in_bar = [&](int part) { return bar0 + 8u * (2 * kStagesMax + 2 * kAccStagesP + part); };  // kSwigluBack: g and u are in
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_ptr + 8 * (2 * kStagesMax + 2 * kAccStagesP + kParts));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *s_tt = reinterpret_cast<int *>(bar_ptr + kBarBytesP);  // [E+1] token tiles before each expert
    int *s_cnt = s_tt + kMaxExperts + 1, *s_row = s_cnt + kMaxExperts, *s_narrow = s_row + kMaxExperts;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

    pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesMax; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < kAccStagesP; s++) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), 8 * kParts);  // one arrival per epilogue warp of both CTAs
        }
        for (int i = 0; i < kParts; i++) mbar_init(in_bar(i), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemColsP) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    // barriers and tensor memory are set up; everything from here on reads what earlier kernels wrote
    pdl_wait();
    if (warp == 2) {
        int run = 0, most = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int cnt = e < E ? counts[e] : 0;
            most = max(most, cnt);
            int n = (cnt + cap - 1) / cap;
            const int own = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, n, o);
                if (lane >= o) n += v;
            }
            if (e < E) {
                s_tt[e] = run + n - own;
                s_cnt[e] = cnt;
                s_row[e] = poffsets[e];
            }
            run += __shfl_sync(0xffffffffu, n, 31);
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) {
            s_tt[E] = run;
            *s_narrow = most <= 64 ? 2 : (most <= 128 ? 1 : 0);
        }
    }
    tc_fence_before();
    cluster_sync_all();  // both CTAs' barriers and tables are in place
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int narrow = kRingStages == 6 ? *s_narrow : 0;
    const int kStagesP = narrow == 2 ? kStagesNarrow : (narrow == 1 ? kStagesMid : kRingStages);
    const int stage_bytes = narrow == 2 ? kStageBytesNarrow : (narrow == 1 ? kStageBytesMid : kStageBytesP);
    const int token_tiles = s_tt[E];
    const int n_ft = (n_out + kFeatPair - 1) / kFeatPair;
    const int total = token_tiles * n_ft;
    const int kb_src = (K + BLOCK_K - 1) / BLOCK_K;
    const int num_kb = KIND == PairKind::kPlainMN2 ? 2 * kb_src : kb_src;
    const int pair0 = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    // Tiles are walked in bands of kband token tiles x all feature tiles, tokens fastest: the rows of a band stay
    // in L2 while the weights stream past them.
    auto tile_at = [&](int tile) {
        const int per_band = kband * n_ft;
        const int band = tile / per_band, r = tile - band * per_band;
        const int t0 = band * kband;
        const int bt = min(kband, token_tiles - t0);
        PairTile p;
        p.ft = r / bt;
        const int tt = t0 + r - p.ft * bt;
        int lo = 0, hi = E - 1;  // last expert whose tiles start at or before tt
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_tt[mid] <= tt) lo = mid;
            else hi = mid - 1;
        }
        p.e = lo;
        const int cnt = s_cnt[lo], i = tt - s_tt[lo], w = tile_width(cnt, cap);
        p.row0 = s_row[lo] + i * w;
        const int left = (cnt + row_round - 1) / row_round * row_round - i * w;
        p.n = (i + 1) * w < cnt ? w : left;  // the last tile ends with the expert's rows, rounded up
        return p;
    };

    if (warp == 0) {
        // ---------------- producer ----------------
        {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = pair0; ok && tile < total; tile += pairs) {
                const PairTile t = tile_at(tile);
                const int b_rows = t.n >> 1;  // this CTA's share of the token columns
                const int row_b = t.row0 + (int)rank * b_rows;
                const int small = b_rows > 64 ? 0 : (b_rows + 31) / 32;  // 32-row boxes instead of one of 128 rows
                const uint32_t bytes = kABytesP + (small ? small * 4096 : 16384);
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!warp_wait(empty_bar(stage), phase ^ 1u, abort_flag, dev_err)) { ok = false; break; }
                    if (elect_one()) {
                        const uint32_t sa = base + stage * stage_bytes, sb = sa + kABytesP;
                        const uint32_t bar = map_to_rank(full_bar(stage), 0);
                        if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * bytes);
                        const bool second = KIND == PairKind::kPlainMN2 && kb >= kb_src;
                        const int kx = (second ? kb - kb_src : kb) * BLOCK_K;
                        if constexpr (kGate) {
                            pair_load_4d(sa, &maps.a0, bar, kx, 0, 0, (t.e * n_out + t.ft * 128 + (int)rank * 64) >> 3);
                        } else if constexpr (!kMN) {
                            pair_load_2d(sa, &maps.a0, bar, kx, t.e * n_out + t.ft * 256 + (int)rank * 128);
                        } else {
                            const CUtensorMap *ma = second ? &maps.a1 : &maps.a0;
                            const int x = t.ft * 256 + (int)rank * 128;
                            pair_load_3d(sa, ma, bar, x, kx, t.e);
                            pair_load_3d(sa + 8192, ma, bar, x + 64, kx, t.e);
                        }
                        if (small == 0) {
                            pair_load_2d(sb, second ? &maps.b1 : &maps.b0, bar, kx, row_b);
                        } else {
                            const CUtensorMap *mb = second ? &maps.b1_32 : &maps.b0_32;
                            for (int i = 0; i < small; i++) pair_load_2d(sb + i * 4096, mb, bar, kx, row_b + i * 32);
                        }
                    }
                    __syncwarp();
                    if (++stage == kStagesP) { stage = 0; phase ^= 1u; }
                }
            }
            // The issuer's commits arrive in both CTAs, in their own time: every stage's last one has to be in before this CTA may
            // go (the cluster barrier at the end orders the threads' arrivals, not those of the tensor core).
            for (int i = 0; ok && i < kStagesP; i++) {
                ok = warp_wait(empty_bar(stage), phase ^ 1u, abort_flag, dev_err);
                if (++stage == kStagesP) { stage = 0; phase ^= 1u; }
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
            int stage = 0, as = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            for (int tile = pair0; ok && tile < total; tile += pairs) {
                const PairTile t = tile_at(tile);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (kMN ? 1u << 15 : 0u) |
                                       ((uint32_t)(t.n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
                if (!warp_wait(tempty_bar(as), aphase ^ 1u, abort_flag, dev_err)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * kTokensMax;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!warp_wait(full_bar(stage), phase, abort_flag, dev_err)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = base + stage * stage_bytes;
                    const uint64_t adesc = kMN ? make_mn_desc(sa) : make_sw128_desc(sa);
                    const uint64_t bdesc = make_sw128_desc(sa + kABytesP);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; k++)  // 16 of the reduction: 32 bytes on, or 16 rows of 128 bytes
                            pair_mma_bf16(d_tmem, adesc + (kMN ? 128u : 2u) * k, bdesc + 2u * k, idesc, (kb | k) != 0 ? 1u : 0u);
                        pair_commit(empty_bar(stage));
                    }
                    __syncwarp();
                    if (++stage == kStagesP) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) pair_commit(tfull_bar(as));
                __syncwarp();
                if (++as == kAccStagesP) { as = 0; aphase ^= 1u; }
            }
        }
    } else {
        // ---------------- epilogue: TMEM -> registers -> shared -> TMA store ----------------
        // warp%4 selects the 32 tensor-memory lanes (features), (warp-2)/4 the group, i.e. its share of
        // the token columns.  The four warps of a group share its staging and a named barrier.
        const int ew = warp - 2, quarter = warp & 3, part = ew >> 2;
        const uint32_t stg = out_stage + part * kPartBytes;
        const bool issuer = (ew & 3) == 0 && lane == 0;
        const int odd = lane & 1;
        auto part_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory"); };
        // true on all 128 threads of the group or on none: its warps leave the loop together
        auto part_all = [&](bool ok) {
            uint32_t r;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                "bar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(r) : "r"((uint32_t)ok), "r"(1 + part) : "memory");
            return r != 0;
        };
        auto word_at = [&](uint32_t sub, int row, int f) {  // features f, f+1 (f even, < 64) of a token row
            return sub + row * 128 + ((((uint32_t)f >> 3) ^ (row & 7)) << 4) + (f & 6) * 2;
        };
        auto put = [&](uint32_t sub, int row, int f, uint32_t word) {
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(word_at(sub, row, f)), "r"(word) : "memory");
        };
        // kSwigluBack: the issuer fetches g and u of the passes (kPass tokens of this group) one ahead of the arithmetic, so the
        // first pass of a tile is there before its accumulator is
        int in_tile = pair0, in_p = 0;
        uint32_t in_phase = 0;
        bool gone = false;
        auto request_next = [&]() {
            int cols = 0;
            PairTile t{};
            for (; in_tile < total; in_tile += pairs, in_p = 0) {
                t = tile_at(in_tile);
                cols = min(max(t.n - part * kPartCols, 0), kPartCols);
                if (in_p < cols) break;
            }
            if (in_tile >= total) return;
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the stores have read the staging rows
            const int x0 = t.ft * 256 + (int)rank * 128, y0 = t.row0 + part * kPartCols + in_p;
            const int subs = min(max((n_out - x0 + 63) / 64, 0), 2), top = min(kPass, cols - in_p);
            mbar_expect_tx(in_bar(part), (uint32_t)(2 * subs * (top / 32) * 4096));
            for (int q = 0; q < subs; q++)
                for (int c = 0; c < top; c += 32) {
                    tma_load_2d(stg + q * kPass * 128 + c * 128, &maps.s0, in_bar(part), x0 + 64 * q, y0 + c);
                    tma_load_2d(stg + (2 + q) * kPass * 128 + c * 128, &maps.s1, in_bar(part), x0 + 64 * q, y0 + c);
                }
            in_p += kPass;
        };
        if constexpr (KIND == PairKind::kSwigluBack) {
            if (issuer) request_next();
        }
        int as = 0;
        uint32_t aphase = 0;
        for (int tile = pair0; tile < total; tile += pairs) {
            const PairTile t = tile_at(tile);
            const bool ok = mbar_wait(tfull_bar(as), aphase, abort_flag, dev_err);
            __syncwarp();
            // the last stores of the tile before must have finished reading the staging rows
            if (KIND != PairKind::kSwigluBack && issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            if (!part_all(ok)) break;
            tc_fence_after();
            const int cols = min(max(t.n - part * kPartCols, 0), kPartCols);  // this group's token columns (a multiple of 32)
            const int y0 = t.row0 + part * kPartCols;
            const uint32_t t_acc = tmem_base + as * kTokensMax + part * kPartCols + ((uint32_t)(quarter * 32) << 16);
            auto release = [&]() {  // all of this warp's accumulator reads are done
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_cluster(map_to_rank(tempty_bar(as), 0));
            };
            if constexpr (kGate) {
                const int up = (lane >> 3) & 1;  // lanes 8-15 and 24-31 hold up rows, the others gate rows
                const int f = quarter * 16 + ((lane >> 4) << 3) + (lane & 6);
                const int x0 = t.ft * 128 + (int)rank * 64;
                constexpr int kOuts = KIND == PairKind::kUpGateKeep ? 3 : 1;  // h; with kUpGateKeep g and u too
                for (int p = 0; p < cols; p += kPass) {
                    if (p > 0) {
                        if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        part_sync();
                    }
                    const int top = min(kPass, cols - p);
                    for (int c = 0; c < top; c += 32) {
                        uint32_t r[32];
                        tc_ld32(t_acc + p + c, r);
                        tc_wait_ld();
                        if (p + c + 32 >= cols) release();
                        float g[16], u[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            // a gate lane finishes token 2i, its up lane token 2i + 1
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? r[2 * i] : r[2 * i + 1], 8);
                            g[i] = __uint_as_float(up ? got : r[2 * i]);
                            u[i] = __uint_as_float(up ? r[2 * i + 1] : got);
                            if constexpr (kOuts == 3) {
                                // h follows from the g and u that are kept: what the backward differentiates
                                g[i] = __bfloat162float(__float2bfloat16_rn(g[i]));
                                u[i] = __bfloat162float(__float2bfloat16_rn(u[i]));
                            }
                        }
                        // an even feature's lane finishes the first of two tokens, its neighbour the second
                        auto out = [&](uint32_t dst, const float (&v)[16]) {
#pragma unroll
                            for (int i = 0; i < 8; i++) {
                                const float got = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 1);
                                put(dst, c + 4 * i + 2 * odd + up, f, odd ? pack_bf16(got, v[2 * i + 1]) : pack_bf16(v[2 * i], got));
                            }
                        };
                        if constexpr (kOuts == 3) {
                            out(stg + kPass * 128, g);
                            out(stg + 2 * kPass * 128, u);
                        }
#pragma unroll
                        for (int i = 0; i < 16; i++) g[i] = (kOuts == 3 ? silu_full(g[i]) : silu_f(g[i])) * u[i];
                        out(stg, g);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    part_sync();
                    if (issuer && x0 < n_out) {
                        for (int c = 0; c < top; c += 32) {
                            tma_store_2d(&maps.o0, stg + c * 128, x0, y0 + p + c);
                            if constexpr (kOuts == 3) {
                                tma_store_2d(&maps.o1, stg + (kPass + c) * 128, x0, y0 + p + c);
                                tma_store_2d(&maps.o2, stg + (2 * kPass + c) * 128, x0, y0 + p + c);
                            }
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
                if (cols == 0) release();
            } else if constexpr (KIND == PairKind::kSwigluBack) {
                const int f = (quarter * 32 + lane) & 62;
                const uint32_t sub = stg + (quarter >> 1) * kPass * 128;  // g of kPass tokens x 64 features
                constexpr uint32_t kToU = 2 * kPass * 128;                  // u lies behind both feature halves of g
                const int x0 = t.ft * 256 + (int)rank * 128;
                for (int p = 0; p < cols; p += kPass) {
                    const bool in = mbar_wait(in_bar(part), in_phase, abort_flag, dev_err);
                    __syncwarp();
                    if (!part_all(in)) { gone = true; break; }
                    in_phase ^= 1u;
                    const int top = min(kPass, cols - p);
                    for (int c = 0; c < top; c += 32) {
                        uint32_t r[32];
                        tc_ld32(t_acc + p + c, r);
                        tc_wait_ld();
                        if (p + c + 32 >= cols) release();
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const float own = __uint_as_float(odd ? r[2 * i + 1] : r[2 * i]);
                            const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, odd ? r[2 * i] : r[2 * i + 1], 1));
                            // dh in the layer's element type, as a pass of its own would read it
                            const uint32_t dh = odd ? pack_bf16(got, own) : pack_bf16(own, got);
                            const uint32_t a = word_at(sub, c + 2 * i + odd, f);
                            uint32_t g, u;
                            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(g) : "r"(a) : "memory");
                            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(u) : "r"(a + kToU) : "memory");
                            float dg[2], du[2];
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                auto half_of = [&](uint32_t w) { return __uint_as_float(q ? w & 0xffff0000u : w << 16); };
                                const float x = half_of(g), d = half_of(dh);
                                const float den = 1.0f + expf(-x), sg = 1.0f / den;
                                du[q] = d * (x / den);
                                dg[q] = (d * half_of(u)) * (sg * (1.0f + x * (1.0f - sg)));
                            }
                            asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(pack_bf16(dg[0], dg[1])) : "memory");
                            asm volatile("st.shared.b32 [%0], %1;" ::"r"(a + kToU), "r"(pack_bf16(du[0], du[1])) : "memory");
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    part_sync();
                    if (issuer) {
                        for (int c = 0; c < top; c += 32)
                            for (int q = 0; q < 2; q++)
                                if (x0 + 64 * q < n_out) {
                                    tma_store_2d(&maps.o0, stg + (q * kPass + c) * 128, x0 + 64 * q, y0 + p + c);
                                    tma_store_2d(&maps.o1, stg + kToU + (q * kPass + c) * 128, x0 + 64 * q, y0 + p + c);
                                }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        request_next();
                    }
                }
                if (gone) break;
                if (cols == 0) release();
            } else {
                const int f = (quarter * 32 + lane) & 62;
                const uint32_t sub = stg + (quarter >> 1) * kPass * 128;  // kPass tokens x 64 features
                const int x0 = t.ft * 256 + (int)rank * 128;
                for (int p = 0; p < cols; p += kPass) {
                    if (p > 0) {
                        if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        part_sync();
                    }
                    const int top = min(kPass, cols - p);
                    for (int c = 0; c < top; c += 32) {
                        uint32_t r[32];
                        tc_ld32(t_acc + p + c, r);
                        tc_wait_ld();
                        if (p + c + 32 >= cols) release();
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const float own = __uint_as_float(odd ? r[2 * i + 1] : r[2 * i]);
                            const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, odd ? r[2 * i] : r[2 * i + 1], 1));
                            put(sub, c + 2 * i + odd, f, odd ? pack_bf16(got, own) : pack_bf16(own, got));
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    part_sync();
                    if (issuer) {
                        for (int c = 0; c < top; c += 32) {
                            if (x0 < n_out) tma_store_2d(&maps.o0, stg + c * 128, x0, y0 + p + c);
                            if (x0 + 64 < n_out) tma_store_2d(&maps.o0, stg + (kPass + c) * 128, x0 + 64, y0 + p + c);
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
                if (cols == 0) release();
            }
            if (++as == kAccStagesP) { as = 0; aphase ^= 1u; }
        }
        if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (*abort_flag && KIND == PairKind::kSwigluBack) {
            const unsigned long long t0 = globaltimer_ns();  // let g and u that were already requested land
            while (globaltimer_ns() - t0 < 2000000ull) { }
        }
    }

    tc_fence_before();
    cluster_sync_all();  // no CTA leaves while its partner's MMAs, arrivals or accumulator reads may still need it
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColsP) : "memory");
    }
}

template <PairKind KIND>
cudaError_t launch_pair_t(omoe_handle *h, cudaStream_t s, bool pdl, const PairMaps &maps, int n_out, int K, int row_round) {
    static PerDeviceOnce once;  // one per instantiation
    bool *done = once.slot();
    if (!done || !*done) {
        cudaError_t e = cudaFuncSetAttribute(pair_gemm_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             pair_smem_bytes<KIND>());
        if (e != cudaSuccess) return e;
        if (done) *done = true;
    }
    return launch_ex(pair_gemm_kernel<KIND>, dim3(h->sm_count & ~1), dim3(PairCfg<KIND>::kThreads), pair_smem_bytes<KIND>(), s, pdl, maps, n_out, K,
                     h->ex_poffsets, h->ex_counts, h->e_local, kTokensMax, row_round, 8, h->dev_err);
}

}  // namespace

cudaError_t launch_pair(omoe_handle *h, cudaStream_t s, bool pdl, PairKind kind, const PairMaps &maps, int n_out, int K,
                        int row_round) {
    switch (kind) {
        case PairKind::kUpGate: return launch_pair_t<PairKind::kUpGate>(h, s, pdl, maps, n_out, K, row_round);
        case PairKind::kUpGateKeep: return launch_pair_t<PairKind::kUpGateKeep>(h, s, pdl, maps, n_out, K, row_round);
        case PairKind::kPlain: return launch_pair_t<PairKind::kPlain>(h, s, pdl, maps, n_out, K, row_round);
        case PairKind::kSwigluBack: return launch_pair_t<PairKind::kSwigluBack>(h, s, pdl, maps, n_out, K, row_round);
        case PairKind::kPlainMN2: return launch_pair_t<PairKind::kPlainMN2>(h, s, pdl, maps, n_out, K, row_round);
    }
    return cudaErrorInvalidValue;
}

}  // namespace omoe
