// Split-KV decode for sm_100a: one to eight query rows per (batch, head) unit against a long
// K/V.  Replaces the reference's forward_kernel_splitkv (src/flash_forward_splitkv.h:14-344) and, where
// the parts of a unit fit one cluster, its combine kernel (:347-399) for those shapes.  The work is a pure
// stream of K and V through the SM: every byte is used once, so the kernel is built around the TMA ring and
// nothing else may stall it.
//
// One CTA = one (unit, part of its keys).  The operands are swapped so that the 128 lanes of tensor
// memory hold KEYS, not queries:
//     S^T[128 keys x 16] = K_tile[128 x d] * Qpad^T[d x 16]      (tcgen05.mma, M=128, N=16)
//     O^T[d x 16]       += V_tile^T[d x 128 keys] * P[128 keys x 16]
// The first kH columns of S^T / O^T belong to queries; the others are padding whose inputs (rows of the Q
// and P operand tiles) are never initialised and whose results are never read -- an operand row only
// influences its own output column.  Thread r of the four softmax warps owns key r of every tile, so masking,
// ALiBi, exp and dropout are spread over 128 threads; one CTA-wide max per chunk of tiles keeps them on a
// common scale.  The MMAs are tiny (N = 16): the tensor pipe is a convenient dot-product engine that
// reads K/V straight from the swizzled TMA tiles, and the kernel stays HBM-bound.
//
// Grouped-query attention and short query blocks: the query heads that share one K/V head, and the
// seqlen_q <= 8 query rows of each, ride in the columns of the same MMAs (column = head * seqlen_q + row), so
// a CTA streams its K/V once for up to sixteen queries.  Groups that need more columns are cut into
// sub-groups of whole heads, one CTA each.  What bounds a CTA beside HBM is the softmax of a chunk (columns x
// tiles per thread), hence kernels for 1, 4, 8 and 16 columns, no mask arithmetic on chunks that no mask
// touches, warp maxima by redux, and the running maxima kept one column per lane: [16 x 32 query heads on 8
// K/V heads, 4097 keys] 56.3 -> 44.6 us (6.0 TB/s), of which 6 us are start and drain; [8 x 32 on 8, 4 rows,
// 8000 keys] 90 -> 47 us (16 columns, four parts, instead of two CTAs per K/V head).  In the mask pass, the dropout draws and
// the epilogue a division or a Philox block per column and tile is what a launch of few tiles spends its time on: slopes, rows
// and draws are worked out once per column, head or tile ([64 heads on 4, 100 keys, 16 columns] 10.8 -> 9.7 us without the
// divisions; [2 x 4 heads, 8 rows, 2971 keys, dropout] 97 -> 28 with one Philox block per head and tile).
//
// The parts of a unit (plan_decode) are the CTAs of one cluster: each leaves its un-normalised O, max and sum
// in its own shared memory, and the CTAs share out the columns and merge them through distributed shared
// memory, so that no partial goes through HBM and no second kernel follows.
//
// Stream order of the TMA ring: K(0), K(1), V(0), K(2), V(1), ... (chunks of kChunk tiles), so
// the scores of chunk c+1 are computed while the softmax of chunk c runs.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "fa_internal.h"
#include "sm100_ptx.cuh"

// Test build only (-DFA_TEST_SHORT_WAIT): the producer can be told to leave out the loads of one tile of the stream, so
// that a consumer's bounded wait runs out and the give-up path can be checked without faulting or hanging anything.
#ifdef FA_TEST_SHORT_WAIT
__device__ int fa_test_decode_skip = -1;
extern "C" int fa_test_skip_decode_tile(int t) {
    return static_cast<int>(cudaMemcpyToSymbol(fa_test_decode_skip, &t, sizeof(int)));
}
#define FA_TEST_SKIPS(t) (fa_test_decode_skip == (t))
#else
#define FA_TEST_SKIPS(t) false
#endif

namespace fa {

namespace {

constexpr int kDThreads = 192;
constexpr int kDTmemCols = 256;            // S^T: 2 buffers x up to 4 tiles x 16 columns; O^T: 16 columns at 128

// kH = columns in use of the 16 (queries that share the CTA's K/V): 1, 4, 8 or 16.  The work of the softmax
// warps goes with kH (plan_decode weighs it against reading K/V once).  D = 64 or 128 (head_dim rounded up).
template <int kH, int D>
struct DCfg {
    // KV tiles per softmax chunk: with 16 columns two, which keeps P and the score registers at the size
    // that two CTAs per SM allow
    static constexpr int kChunk = kH == 16 ? 2 : 4;
    static constexpr int kTileBytes = kTile * D * 2;  // one K or V tile: [128 keys x D], one or two 64-column boxes
    static constexpr int kStages = D == 64 ? 6 : 3;   // 96 KB in flight either way
    static constexpr int kNumBars = 2 * kStages + 2 + 2 + 3;
    // K-major operand of 16 rows (Q, and P of one tile): 1 KB atoms of 8 rows x 64 elements.  Rows 8-15 are
    // the next atom; with at most 8 columns in use they fall on the second half's atom and are never looked at.
    static constexpr int kHalfBytes = kH == 16 ? 2048 : 1024;  // from the first 64 elements to the second
    static constexpr int kOperandBytes = 2 * kHalfBytes;
    static constexpr int kSmemRing = 0;
    static constexpr int kSmemP = kStages * kTileBytes;
    static constexpr int kSmemQ = kSmemP + kChunk * kOperandBytes + (kH == 16 ? 0 : 1024);  // (+ what rows 8-15 touch)
    static constexpr int kSmemBar = kSmemQ + kOperandBytes + (kH == 16 ? 0 : 1024);
    static constexpr int kSmemRed = (kSmemBar + 8 * kNumBars + 15) / 16 * 16;  // float[2][4][kH] maxima, float[4][kH] sums
    static constexpr int kSmemMisc = kSmemRed + 3 * 4 * kH * 4;
    static constexpr int kSmemEnd = kSmemMisc + 16;
    // V^T is always an M = 128 operand; with D = 64 its upper 64 rows read the 16 KB behind the tile (the next
    // slot, or what follows the ring) and only reach accumulator lanes that nobody reads
    static constexpr int kSmemReach = kSmemP + (D == 64 ? kTile * 128 : 0);
    static constexpr int kSmemBytes = (kSmemEnd > kSmemReach ? kSmemEnd : kSmemReach) + 1024;  // + alignment slack
    static_assert(kSmemBytes <= 115712, "two CTAs per SM");
};

constexpr float kDLog2e = 1.4426950408889634f;
constexpr float kDLn2 = 0.6931471805599453f;

__host__ __device__ constexpr uint32_t make_idesc_swapped(bool is_bf16, bool a_mn_major) {
    return (1u << 4) | ((is_bf16 ? 1u : 0u) << 7) | ((is_bf16 ? 1u : 0u) << 10) |
           ((a_mn_major ? 1u : 0u) << 15) | (0u << 16) | (static_cast<uint32_t>(16 >> 3) << 17) |
           (static_cast<uint32_t>(kTile >> 4) << 24);
}

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t tmem_ld1(uint32_t taddr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
    return r;
}
__device__ __forceinline__ void tmem_st1(uint32_t taddr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// kH columns of one TMEM lane
template <int kH>
__device__ __forceinline__ void tmem_ld_heads(uint32_t taddr, uint32_t (&r)[kH]) {
    if constexpr (kH == 1) r[0] = tmem_ld1(taddr);
    else if constexpr (kH == 4) tmem_ld4(taddr, r);
    else if constexpr (kH == 8) tmem_ld8(taddr, r);
    else tmem_ld16(taddr, r);
}
template <int kH>
__device__ __forceinline__ void tmem_st_heads(uint32_t taddr, const uint32_t (&r)[kH]) {
    if constexpr (kH == 1) tmem_st1(taddr, r[0]);
    else if constexpr (kH == 4) tmem_st4(taddr, r);
    else if constexpr (kH == 8) tmem_st8(taddr, r);
    else tmem_st16(taddr, r);
}
// Maximum over the lanes of a warp.
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ bool mbar_wait_warp_ok(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag) ? 1 : 0) != 0;
}
__device__ __forceinline__ void named_barrier_128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// One element of a finished output row, and (thread 0) its log-sum-exp.
template <bool kBf16>
__device__ __forceinline__ void store_result(const DecodeArgs& a, long long row, int col, float o_val, float lse_val) {
    if (col < a.o_dim) {
        if (a.o_is_fp32) static_cast<float*>(a.o)[row * a.o_dim + col] = o_val;
        else if (kBf16) static_cast<__nv_bfloat16*>(a.o)[row * a.o_dim + col] = __float2bfloat16_rn(o_val);
        else static_cast<__half*>(a.o)[row * a.o_dim + col] = __float2half_rn(o_val);
    }
    if (col == 0 && a.lse != nullptr) a.lse[row] = lse_val;
}

template <bool kBf16, int kH, int D, bool kDropout>
__global__ void __launch_bounds__(kDThreads, 2)
decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const DecodeArgs a) {
    using C = DCfg<kH, D>;
    constexpr int kChunkTiles = C::kChunk, kDStages = C::kStages, kDTileBytes = C::kTileBytes;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t sRing = smem_base + C::kSmemRing;
    const uint32_t sP = smem_base + C::kSmemP;
    const uint32_t sQ = smem_base + C::kSmemQ;
    const uint32_t bar0 = smem_base + C::kSmemBar;
    const uint32_t bar_full = bar0;                          // [kDStages]
    const uint32_t bar_empty = bar_full + 8 * kDStages;      // [kDStages]
    const uint32_t bar_s_full = bar_empty + 8 * kDStages;    // [2]
    const uint32_t bar_s_free = bar_s_full + 16;             // [2]
    const uint32_t bar_p_full = bar_s_free + 16;
    const uint32_t bar_p_free = bar_p_full + 8;
    const uint32_t bar_o_done = bar_p_free + 8;
    float* red = reinterpret_cast<float*>(smem_gen + C::kSmemRed);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + C::kSmemMisc);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + C::kSmemMisc + 4);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // the kernel behind this one in the stream may take its place on the SMs as they free up
    // (it waits for this grid's completion before it touches memory)
    grid_dep_launch_dependents();
    if (warp == 4 && lane == 0) {
        *abort_flag = 0;
        tma_prefetch_desc(&tmap_k);
        tma_prefetch_desc(&tmap_v);
        for (int s = 0; s < kDStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_s_full + 8 * i, 1);
            mbar_init(bar_s_free + 8 * i, 4);
        }
        mbar_init(bar_p_full, 4);
        mbar_init(bar_p_free, 1);
        mbar_init(bar_o_done, 1);
        mbar_fence_init();
    }
    // kH = 1: one CTA per (query unit, part of its keys).  kH = 4, 8, 16: one CTA per (K/V unit, sub-group of its query
    // heads whose rows fit kH columns, part); `unit` is then the first query unit of the sub-group.
    const int cta_unit = static_cast<int>(fast_div(a.div_parts, blockIdx.x));
    const int part = static_cast<int>(blockIdx.x) - cta_unit * a.parts;
    int unit, kv_unit, gh = 1;
    const int sq = (kH == 1) ? 1 : a.seqlen_q;  // query rows per head (columns per head)
    if constexpr (kH == 1) {
        unit = kv_unit = cta_unit;
    } else {
        const int heads_per_cta = kH / sq;
        kv_unit = static_cast<int>(fast_div(a.div_subgroups, static_cast<uint32_t>(cta_unit)));
        const int sub = cta_unit - kv_unit * a.subgroups;
        unit = kv_unit * a.kv_group + sub * heads_per_cta;
        gh = min(heads_per_cta, a.kv_group - sub * heads_per_cta);  // query heads of this CTA
    }
    const int nc = gh * sq;  // columns in use: column n = head n / sq, query row n % sq
    const long long row0 = static_cast<long long>(unit) * sq;  // column n is row row0 + n of Q, O and LSE

    // KV tiles of this part.  With dropout the parts are the caller's splits, whose tile ranges are part of
    // the dropout streams' geometry; otherwise the visible tiles are dealt out evenly.
    int lo, hi;
    if (a.by_split) {
        lo = max(a.tiles_per_split * part, a.vis_lo);
        hi = min(min(a.tiles_per_split * (part + 1), a.tc), a.vis_hi);
    } else {
        const int n = a.vis_hi - a.vis_lo;
        lo = a.vis_lo + static_cast<int>(fast_div(a.div_parts, static_cast<uint32_t>(n * part)));
        hi = a.vis_lo + static_cast<int>(fast_div(a.div_parts, static_cast<uint32_t>(n * (part + 1))));
    }
    const int n_tiles = hi > lo ? hi - lo : 0;
    const int n_chunks = (n_tiles + kChunkTiles - 1) / kChunkTiles;
    auto chunk_tiles = [&](int c) { return min(kChunkTiles, n_tiles - c * kChunkTiles); };
    int pushed = 0;  // tiles whose loads have been issued (producer lane only)

    if (warp == 5 && n_tiles > 0) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kDTmemCols);
        tmem_relinquish();
    }
    grid_dep_wait();  // every thread, before its first global access
    if (warp == 4 && lane == 0) {
        // the first K tiles are put in flight before the CTA-wide sync: their latency overlaps Q's
        const int first = min(min(kDStages, kChunkTiles), n_tiles);
        for (; pushed < first; ++pushed) {
            mbar_expect_tx(bar_full + 8 * pushed, kDTileBytes);
#pragma unroll
            for (int b = 0; b < D / 64; ++b)
                tma_load_3d(sRing + pushed * kDTileBytes + b * (kTile * 128), &tmap_k, bar_full + 8 * pushed, b * 64,
                            (lo + pushed) * kTile, kv_unit);
        }
    }
    if (n_tiles > 0) {
        // query n (head n / sq, row n % sq: consecutive rows of Q) goes to row n of the Q operand
        // (16-byte unit u -> half u/8, unit (u%8) ^ (n%8) of row n: the 128-byte swizzle)
        constexpr int kUnits = D / 8;
        for (int i = threadIdx.x; i < kUnits * kH; i += kDThreads) {
            const int u = i % kUnits, n = i / kUnits;
            uint4 val = make_uint4(0u, 0u, 0u, 0u);
            if (n < nc && u * 8 < a.head_dim)
                val = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.q) +
                                                      (row0 + n) * a.head_dim + u * 8);
            *reinterpret_cast<uint4*>(smem_gen + C::kSmemQ + (u >> 3) * C::kHalfBytes + n * 128 + (((u & 7) ^ (n & 7)) << 4)) = val;
        }
        fence_proxy_async_smem();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = (n_tiles > 0) ? *tmem_slot : 0u;
    const uint32_t tmem_o = tmem_base + 128;

    int fail = 0;

    if (n_tiles > 0 && warp == 4) {
        // ======================= TMA producer ===================================
        if (lane == 0) {
            int slot = 0;  // running count of tiles in stream order
            auto push = [&](const CUtensorMap* map, int tile) -> bool {
                if (slot < pushed) { ++slot; return true; }  // issued during set-up
                const int st = slot % kDStages;
                const uint32_t ph = (slot / kDStages) & 1;
                if (!mbar_wait(bar_empty + 8 * st, ph ^ 1, abort_flag)) return false;
                if (FA_TEST_SKIPS(slot)) { ++slot; return true; }
                mbar_expect_tx(bar_full + 8 * st, kDTileBytes);
#pragma unroll
                for (int b = 0; b < D / 64; ++b)
                    tma_load_3d(sRing + st * kDTileBytes + b * (kTile * 128), map, bar_full + 8 * st, b * 64, tile * kTile, kv_unit);
                ++slot;
                return true;
            };
            auto push_chunk = [&](const CUtensorMap* map, int c) -> bool {
                for (int t = 0; t < chunk_tiles(c); ++t)
                    if (!push(map, lo + c * kChunkTiles + t)) return false;
                return true;
            };
            bool ok = push_chunk(&tmap_k, 0);
            for (int c = 0; ok && c < n_chunks; ++c) {
                if (c + 1 < n_chunks) ok = push_chunk(&tmap_k, c + 1);
                if (ok) ok = push_chunk(&tmap_v, c);
            }
            if (!ok) fail = 1;
        }
    } else if (n_tiles > 0 && warp == 5) {
        // ======================= MMA issuer =====================================
        if (lane == 0) {
            constexpr uint32_t idesc_qk = make_idesc_swapped(kBf16, false);
            constexpr uint32_t idesc_pv = make_idesc_swapped(kBf16, true);
            int slot = 0;
            auto qk_chunk = [&](int c) -> bool {
                const int buf = c & 1;
                if (c >= 2 && !mbar_wait(bar_s_free + 8 * buf, ((c >> 1) - 1) & 1, abort_flag)) return false;
                tc_fence_after_sync();
                for (int t = 0; t < chunk_tiles(c); ++t) {
                    const int st = slot % kDStages;
                    if (!mbar_wait(bar_full + 8 * st, (slot / kDStages) & 1, abort_flag)) return false;
                    tc_fence_after_sync();
                    const uint32_t kt = sRing + st * kDTileBytes;
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) {
                        const uint32_t off = (ks / 4) * (kTile * 128) + (ks % 4) * 32;
                        const uint32_t qoff = (ks / 4) * C::kHalfBytes + (ks % 4) * 32;
                        umma_ss(tmem_base + buf * 64 + t * 16, make_smem_desc(kt + off, 0, 1024),
                                make_smem_desc(sQ + qoff, 0, 1024), idesc_qk, ks > 0 ? 1u : 0u);
                    }
                    umma_commit(bar_empty + 8 * st);
                    ++slot;
                }
                umma_commit(bar_s_full + 8 * buf);
                return true;
            };
            auto pv_chunk = [&](int c) -> bool {
                if (!mbar_wait(bar_p_full, c & 1, abort_flag)) return false;
                tc_fence_after_sync();
                for (int t = 0; t < chunk_tiles(c); ++t) {
                    const int st = slot % kDStages;
                    if (!mbar_wait(bar_full + 8 * st, (slot / kDStages) & 1, abort_flag)) return false;
                    tc_fence_after_sync();
                    const uint32_t vt = sRing + st * kDTileBytes;
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        // A = V^T: 16 keys (2048 bytes) per step, the two 64-column halves 16 KB apart
                        const uint32_t poff = t * C::kOperandBytes + (ks / 4) * C::kHalfBytes + (ks % 4) * 32;
                        umma_ss(tmem_o, make_smem_desc(vt + ks * 2048, kTile * 128, 1024),
                                make_smem_desc(sP + poff, 0, 1024), idesc_pv, (c > 0 || t > 0 || ks > 0) ? 1u : 0u);
                    }
                    umma_commit(bar_empty + 8 * st);
                    ++slot;
                }
                umma_commit(bar_p_free);
                return true;
            };
            bool ok = qk_chunk(0);
            for (int c = 0; ok && c < n_chunks; ++c) {
                if (c + 1 < n_chunks) ok = qk_chunk(c + 1);
                if (ok) ok = pv_chunk(c);
            }
            if (ok) umma_commit(bar_o_done);
            else fail = 2;
        }
    } else if (warp < 4) {
        // ======================= softmax over keys / epilogue ===================
        const int r = threadIdx.x;  // key inside a tile; output column in the epilogue
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        // scores stay unscaled and the scale is folded into the exponent's FMA, except with ALiBi
        const bool alibi = a.alibi_slopes != nullptr;
        const float scale2 = a.scale_log2, exp_scale = alibi ? 1.0f : a.scale_log2;
        float slope = 0.0f;  // ALiBi slope of column `lane`, handed round like the maxima
        if (alibi && lane < nc) slope = a.alibi_slopes[(unit + lane / sq) % a.heads] * kDLog2e;
        float m_ref = -INFINITY;  // CTA-wide running max of column `lane` (lanes < kH of every warp), log2 units
        float l_part[kH];         // this thread's share of each column's row sum
#pragma unroll
        for (int n = 0; n < kH; ++n) l_part[n] = 0.0f;
        // this key's element of column n in the P operand: row n, 128-byte swizzled
        uint8_t* p_half = smem_gen + C::kSmemP + (r >> 6) * C::kHalfBytes + (r & 7) * 2;
        const uint32_t p_unit = static_cast<uint32_t>((r & 63) >> 3);

        for (int c = 0; c < n_chunks; ++c) {
            const int buf = c & 1;
            const int nt = chunk_tiles(c);
            const int tile0 = lo + c * kChunkTiles;
            bool ok = mbar_wait_warp_ok(bar_s_full + 8 * buf, (c >> 1) & 1, abort_flag);
            if (!ok) fail = 3;
            tc_fence_after_sync();
            uint32_t raw[kChunkTiles][kH];
#pragma unroll
            for (int t = 0; t < kChunkTiles; ++t) {
                if (t < nt) {
                    tmem_ld_heads<kH>(tmem_base + lane_base + buf * 64 + t * 16, raw[t]);
                } else {
#pragma unroll
                    for (int n = 0; n < kH; ++n) raw[t][n] = 0xff800000u;  // -inf
                }
            }
            tmem_wait_ld();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_s_free + 8 * buf);
            float v[kChunkTiles][kH];
#pragma unroll
            for (int t = 0; t < kChunkTiles; ++t) {
#pragma unroll
                for (int n = 0; n < kH; ++n) v[t][n] = __uint_as_float(raw[t][n]);
            }
            // masks and ALiBi, on the chunks that have any (the tiles [full_lo, full_hi) are visible whole)
            if (alibi || tile0 < a.full_lo || tile0 + nt > a.full_hi) {
                int rel[kChunkTiles];      // key positions relative to query row 0, saturated far outside any window
                bool in_range[kChunkTiles];
#pragma unroll
                for (int t = 0; t < kChunkTiles; ++t) {
                    const long long key = static_cast<long long>(tile0 + t) * kTile + r;
                    in_range[t] = t < nt && key < a.seqlen_k;
                    rel[t] = static_cast<int>(max(-0x40000000LL, min(a.k_pos0 + key - a.q_pos0, 0x40000000LL)));
                }
                int q_row = 0;  // query row of column n, n % sq
#pragma unroll
                for (int n = 0; n < kH; ++n) {
                    const float slope_n = alibi ? __shfl_sync(0xffffffffu, slope, n) : 0.0f;
#pragma unroll
                    for (int t = 0; t < kChunkTiles; ++t) {
                        const int ahead = rel[t] - q_row;  // > 0: the key lies after the query
                        bool keep = in_range[t];
                        if (a.is_causal && ahead > 0) keep = false;
                        if (a.window_left >= 0 && -ahead > a.window_left) keep = false;
                        if (a.window_right >= 0 && ahead > a.window_right) keep = false;
                        if (alibi) v[t][n] = fmaf(-slope_n, fabsf(static_cast<float>(ahead)), v[t][n] * scale2);
                        if (!keep) v[t][n] = -INFINITY;
                    }
                    if (++q_row == sq) q_row = 0;
                }
            }
            float* red_c = red + buf * 4 * kH;
            {
                float m_w[kH];
#pragma unroll
                for (int n = 0; n < kH; ++n) {
                    float m = v[0][n];
#pragma unroll
                    for (int t = 1; t < kChunkTiles; ++t) m = fmaxf(m, v[t][n]);
                    m_w[n] = warp_max(m);
                }
                if (lane == 0) {
#pragma unroll
                    for (int n = 0; n < kH; ++n) red_c[warp * kH + n] = m_w[n];
                }
            }
            named_barrier_128();

            // the previous chunk's P V must be done before P is overwritten or O rescaled
            if (c > 0) {
                if (!mbar_wait_warp_ok(bar_p_free, (c - 1) & 1, abort_flag)) fail = 4;
                tc_fence_after_sync();
            }
            // lane n keeps column n's running max (lazily raised, as in the tiled kernel) and hands it round
            float m_new = m_ref, factor = 1.0f;
            if (lane < kH) {
                const float m_chunk = fmaxf(fmaxf(red_c[lane], red_c[kH + lane]), fmaxf(red_c[2 * kH + lane], red_c[3 * kH + lane])) * exp_scale;
                if (m_chunk > m_ref + 8.0f || m_ref == -INFINITY) m_new = fmaxf(m_ref, m_chunk);
                if (m_new != m_ref) factor = (m_ref == -INFINITY) ? 0.0f : ex2f(m_ref - m_new);
            }
            if (__any_sync(0xffffffffu, m_new != m_ref)) {  // CTA-uniform: every warp sees the same maxima
                float f[kH];
#pragma unroll
                for (int n = 0; n < kH; ++n) {
                    f[n] = __shfl_sync(0xffffffffu, factor, n);
                    l_part[n] *= f[n];
                }
                if (c > 0) {
                    uint32_t ov[kH];
                    tmem_ld_heads<kH>(tmem_o + lane_base, ov);
                    tmem_wait_ld();
#pragma unroll
                    for (int n = 0; n < kH; ++n) ov[n] = __float_as_uint(__uint_as_float(ov[n]) * f[n]);
                    tmem_st_heads<kH>(tmem_o + lane_base, ov);
                    tmem_wait_st();
                }
            }
            m_ref = m_new;
            const float neg_lane = (m_new == -INFINITY) ? 0.0f : -m_new;

            // Keep bits of this key, tile t's column n at bit 16 t + n.  The rows of a head share their draws (the reference's
            // draw order gives one 8-row group the same: draw 64*tile_index + 8*(col/16) + 2*((col%16)/8) + col%2), so one
            // Philox block per head and tile serves them all.
            unsigned long long kept = 0ull;
            if constexpr (kDropout) {
#pragma unroll 1
                for (int t = 0; t < nt; ++t) {
                    const unsigned long long first = continuation(a.drop, n_tiles) +
                                                     64ull * static_cast<unsigned long long>(c * kChunkTiles + t) + 8ull * (r >> 4);
#pragma unroll 1
                    for (int h = 0; h < gh; ++h) {
                        const unsigned long long subseq = (a.drop.unit0 + unit + h) * static_cast<unsigned long long>(a.parts) +
                                                          static_cast<unsigned long long>(part);
                        const uint32_t bits = philox_keep4(a.drop, subseq, first);
                        if ((bits >> (2 * ((r >> 3) & 1) + (r & 1))) & 1u) kept |= ((1ull << sq) - 1ull) << (16 * t + h * sq);
                    }
                }
            }

#pragma unroll
            for (int n = 0; n < kH; ++n) {
                const float neg_m = __shfl_sync(0xffffffffu, neg_lane, n);
                uint8_t* p_row = p_half + n * 128 + ((p_unit ^ (n & 7)) << 4);
#pragma unroll
                for (int t = 0; t < kChunkTiles; t += 2) {
                    float p[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        p[i] = ex2f(fmaf(v[t + i][n], exp_scale, neg_m));
                        l_part[n] += p[i];
                        if constexpr (kDropout) {
                            if (!((kept >> (16 * (t + i) + n)) & 1ull)) p[i] = 0.0f;
                        }
                    }
                    uint32_t h;  // the two tiles' elements, rounded together
                    if constexpr (kBf16) {
                        const __nv_bfloat162 x = __floats2bfloat162_rn(p[0], p[1]);
                        h = *reinterpret_cast<const uint32_t*>(&x);
                    } else {
                        const __half2 x = __floats2half2_rn(p[0], p[1]);
                        h = *reinterpret_cast<const uint32_t*>(&x);
                    }
                    if (t < nt) *reinterpret_cast<uint16_t*>(p_row + t * C::kOperandBytes) = static_cast<uint16_t>(h);
                    if (t + 1 < nt) *reinterpret_cast<uint16_t*>(p_row + (t + 1) * C::kOperandBytes) = static_cast<uint16_t>(h >> 16);
                }
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_full);
        }

        // ---- epilogue ----------------------------------------------------------------
#pragma unroll
        for (int n = 0; n < kH; ++n) {
            float l_warp = l_part[n];
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) l_warp += __shfl_xor_sync(0xffffffffu, l_warp, o);
            if (lane == 0) red[8 * kH + warp * kH + n] = l_warp;
        }
        uint32_t o_raw[kH];
#pragma unroll
        for (int n = 0; n < kH; ++n) o_raw[n] = 0u;
        if (n_tiles > 0 && fail == 0) {
            if (mbar_wait_warp_ok(bar_o_done, 0, abort_flag)) {
                tc_fence_after_sync();
                tmem_ld_heads<kH>(tmem_o + lane_base, o_raw);
                tmem_wait_ld();
            } else {
                fail = 5;
            }
        }
        named_barrier_128();
        // A wait of this CTA gave up (the flag was set by whoever waited, before the barrier above): none of its columns
        // may pass for the part of a softmax, so they and their sums are NaN, which the merges carry on; and the copies
        // still in flight land first, since they write where the columns are staged.
        const bool gave_up = *abort_flag != 0;
        if (gave_up) {
            const long long t0 = clock64();
            while (clock64() - t0 < 200000) { }
        }
        float m_col[kH];
#pragma unroll
        for (int n = 0; n < kH; ++n) m_col[n] = __shfl_sync(0xffffffffu, m_ref, n);
        if (a.merge) {
            // this part's un-normalised row of every column, its max and its sum, for the peers to read
            // (the ring is free: the last P V has completed)
            float* part_o = reinterpret_cast<float*>(smem_gen + C::kSmemRing);
#pragma unroll
            for (int n = 0; n < kH; ++n) {
                part_o[n * kTile + r] = gave_up ? __int_as_float(0x7fc00000) : __uint_as_float(o_raw[n]);
                if (r == 0) {
                    const float l_sum = (red[8 * kH + n] + red[9 * kH + n]) + (red[10 * kH + n] + red[11 * kH + n]);
                    part_o[kH * kTile + 2 * n] = m_col[n];
                    part_o[kH * kTile + 2 * n + 1] = gave_up ? __int_as_float(0x7fc00000) : l_sum;
                }
            }
        } else {
            long long prow = (unit * static_cast<long long>(a.parts) + part) * sq;  // row of column n in the partials
            int q_row = 0;
#pragma unroll
            for (int n = 0; n < kH; ++n) {
                if (n >= nc) continue;
                const float l_sum = (red[8 * kH + n] + red[9 * kH + n]) + (red[10 * kH + n] + red[11 * kH + n]);
                const float inv = l_sum > 0.0f ? a.drop.inv_keep / l_sum : 0.0f;
                const float lse_val = l_sum > 0.0f ? m_col[n] * kDLn2 + __logf(l_sum) : -INFINITY;
                const float o_val = __uint_as_float(o_raw[n]) * inv;
                if (a.parts > 1) {  // partial of this part, for the combine kernel
                    if (r < a.head_dim) a.o_partial[prow * a.head_dim + r] = o_val;
                    if (r == 0) a.lse_partial[prow] = gave_up ? __int_as_float(0x7fc00000) : lse_val;
                    ++prow;
                    if (++q_row == sq) {  // the next head's partials
                        q_row = 0;
                        prow += static_cast<long long>(a.parts - 1) * sq;
                    }
                } else {
                    store_result<kBf16>(a, row0 + n, r, o_val, lse_val);
                }
            }
        }
    }

    if (fail != 0) {
        *abort_flag = 1;
        if (a.status != nullptr) atomicExch(a.status, 200 + fail);
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) { }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 5 && n_tiles > 0) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kDTmemCols);
    }
    if (a.merge) {
        // The parts of a unit are one cluster: each CTA reads its share of the columns from all of them
        // through distributed shared memory and writes the finished rows.  O = sum_j 2^(m_j - m) O_j / l,
        // l = sum_j 2^(m_j - m) l_j (src/flash_forward_splitkv.h:359-397).
        __syncwarp();
        cluster_sync();
        if (warp < 4) {
            const int r = threadIdx.x;
            const uint32_t base = sRing;
            for (int n = part; n < nc; n += a.parts) {
                float m_j[kDecodeCluster], l_j[kDecodeCluster], o_j[kDecodeCluster];
#pragma unroll
                for (int j = 0; j < kDecodeCluster; ++j) {
                    m_j[j] = -INFINITY;
                    l_j[j] = o_j[j] = 0.0f;
                    if (j < a.parts) {
                        const uint32_t peer = cluster_map(base, j);
                        m_j[j] = ld_cluster_f32(peer + (kH * kTile + 2 * n) * 4);
                        l_j[j] = ld_cluster_f32(peer + (kH * kTile + 2 * n + 1) * 4);
                        o_j[j] = ld_cluster_f32(peer + (n * kTile + r) * 4);
                    }
                }
                float m = m_j[0];
#pragma unroll
                for (int j = 1; j < kDecodeCluster; ++j) m = fmaxf(m, m_j[j]);
                float l = 0.0f, o = 0.0f;
                if (m != -INFINITY) {
#pragma unroll
                    for (int j = 0; j < kDecodeCluster; ++j) {
                        // (a part without visible keys has m_j = -inf and weight 0; its o_j is 0)
                        const float w = ex2f(m_j[j] - m);
                        l = fmaf(w, l_j[j], l);
                        o = fmaf(w, o_j[j], o);
                    }
                } else {
                    // no visible key (all zero), or nothing but NaN
#pragma unroll
                    for (int j = 0; j < kDecodeCluster; ++j) {
                        l += l_j[j];
                        o += o_j[j];
                    }
                }
                const float inv = l > 0.0f ? a.drop.inv_keep / l : 0.0f;
                store_result<kBf16>(a, row0 + n, r, o * inv, l > 0.0f ? m * kDLn2 + __logf(l) : -INFINITY);
            }
            __syncwarp();
        }
        cluster_sync();  // the peers' shared memory stays until everyone has read it
    }
}

}  // namespace

void plan_decode(DecodeArgs* a, int units, int splits, int most, int sms, const ClusterRoom& room) {
    // key tiles visible to any query row: the tile-granular clip of the masks (src/flash_forward.h:39-48)
    // for the query rows at positions q_pos0 .. q_pos0 + seqlen_q - 1
    long long lo = 0, hi = a->tc;
    auto tiles_to = [&](long long last) { return last < 0 ? 0LL : std::min<long long>(last / kTile + 1, a->tc); };
    const long long last_q = a->q_pos0 + a->seqlen_q - 1 - a->k_pos0;
    if (a->window_left >= 0)
        lo = std::max(0LL, std::min<long long>((a->q_pos0 - a->window_left - a->k_pos0) / kTile, a->tc));
    if (a->window_right >= 0) hi = std::min(hi, tiles_to(last_q + a->window_right));
    if (a->is_causal) hi = std::min(hi, tiles_to(last_q));
    a->vis_lo = static_cast<int>(lo);
    a->vis_hi = static_cast<int>(std::max(lo, hi));
    const int n = a->vis_hi - a->vis_lo;

    // tiles that need no mask: inside seqlen_k and visible to every query row
    long long flo = 0, fhi = a->seqlen_k / kTile;
    const long long first_q = a->q_pos0 - a->k_pos0;
    if (a->window_left >= 0) flo = std::max(0LL, (last_q - a->window_left + kTile - 1) / kTile);
    if (a->window_right >= 0) fhi = std::min(fhi, std::max(0LL, (first_q + a->window_right + 1) / kTile));
    if (a->is_causal) fhi = std::min(fhi, std::max(0LL, (first_q + 1) / kTile));
    a->full_lo = static_cast<int>(std::min<long long>(flo, a->tc));
    a->full_hi = static_cast<int>(fhi);

    // How many columns a CTA has (query heads that share a K/V head are packed into one CTA, whole heads with their query rows;
    // what does not fit goes to further sub-groups, CTAs of their own that read the same K/V) and how many CTAs share a unit's
    // keys: the fastest by a model of the kernel's time, in us, fitted to 461 shapes of 8 to 512 K/V heads x 1 to 256 tiles, each
    // swept over its columns and parts: what it takes is 0.3 % slower than the best on average, at most 14 %.
    //   A CTA takes `fixed` to start, mask and drain and `rate` for a K + V tile, a sixth more with a second CTA on its SM; what
    //   does not fit (two CTAs an SM, clusters as the device has room for them) follows in waves.  Columns cost by the CTA, since a
    //   softmax thread takes its key through all of them: sixteen pay only where CTAs are many or HBM bounds the launch ([1 x 64
    //   heads on 4, 100 keys] 10.7 us in sixteen columns, 5.1 in four; [16 x 32 on 8, 4 rows, 8192 keys] 130 in four, 88 in sixteen).
    //   A merge in the cluster costs 1 to 2 us, partials through memory and the combine kernel 7.5 and 0.34 a part.
    //   HBM gives 7.65 TB/s, the dropout bits of a head and tile take 0.12.
    struct Cost {
        double fixed[4], rate[4];
    };
    static constexpr Cost kCost[2] = {{{3.0, 4.2, 6.1, 7.3}, {0.79, 0.84, 0.68, 1.06}},    // by columns 1, 4, 8, 16: D = 128
                                      {{3.05, 4.2, 6.2, 7.7}, {0.69, 0.68, 0.65, 0.81}}};  // D = 64
    static constexpr int kColumns[4] = {1, 4, 8, 16};
    static constexpr double kMerge[5] = {0.0, 2.05, 1.15, 1.45, 1.0};  // 1, 2, 4, 8, 16 parts
    const Cost& cost = kCost[a->head_dim <= 64];
    const bool dropout = a->drop.threshold != 0ull;
    const int queries = a->kv_group * a->seqlen_q, kv_units = units / a->kv_group;
    const double hbm_us = static_cast<double>(kv_units) * n * kTile * a->head_dim * 4.0 / 7.65e6;
    double best_us = 1e30;
    for (int i = queries == 1 ? 0 : 1; i < 4; ++i) {
        const int heads_per_cta = kColumns[i] / a->seqlen_q;
        if (heads_per_cta < 1) continue;
        const int subgroups = (a->kv_group + heads_per_cta - 1) / heads_per_cta;
        const double rate = cost.rate[i] + (dropout ? 0.12 * std::min(heads_per_cta, a->kv_group) : 0.0);
        // (with dropout the parts are the caller's splits, part of the streams' geometry)
        for (int p = 0, parts = dropout ? splits : 1; dropout || (parts <= most && (p == 0 || parts <= n)); ++p, parts *= 2) {
            const bool cluster = parts == 2 || parts == 4 || parts == 8 || parts == 16, merged = cluster && room.fits(parts, 2) > 0;
            if (cluster && !merged && !dropout) continue;
            const long long ctas = static_cast<long long>(kv_units) * subgroups * parts;
            const long long slots = merged ? static_cast<long long>(room.fits(parts, 2)) * parts : 2LL * sms;
            const double chain = cost.fixed[i] + rate * ((n + parts - 1) / parts);
            auto wave = [&](long long c) { return c > 0 ? chain * (1.0 + 0.166 * std::min(1.0, std::max(0.0, static_cast<double>(c) / sms - 1.0))) : 0.0; };
            double us = static_cast<double>(ctas / slots) * wave(slots) + wave(ctas % slots);
            if (merged) us += kMerge[parts == 2 ? 1 : parts == 4 ? 2 : parts == 8 ? 3 : 4] - (i > 0 ? 0.8 : 0.0);
            else if (parts > 1) us += 7.5 + 0.34 * parts;
            const double floor_us = 0.65 + hbm_us * (ctas <= slots ? 1.02 : 1.0);
            us = std::max(us, floor_us) + 0.2 * std::min(us, floor_us);
            if (us < best_us) {
                best_us = us;
                a->columns = kColumns[i];
                a->subgroups = subgroups;
                a->parts = parts;
                a->merge = merged;
            }
            if (dropout) break;
        }
        if (kColumns[i] >= queries) break;  // (no use for more)
    }
    a->by_split = dropout && splits > 1;
}

cudaError_t launch_decode(const DecodeArgs& a_in, const CUtensorMap& tk, const CUtensorMap& tv, int units, bool bf16,
                          cudaStream_t stream) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    DecodeArgs a = a_in;
    if (a.seqlen_q < 1 || a.seqlen_q > 8) return cudaErrorInvalidValue;
    const long long ctas = static_cast<long long>(units / a.kv_group) * a.subgroups * a.parts;
    if (ctas <= 0 || ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    a.div_parts = make_fastdiv(static_cast<uint32_t>(a.parts));
    a.div_subgroups = make_fastdiv(static_cast<uint32_t>(a.subgroups));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(kDThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(a.parts);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.merge ? 2 : 1;
    auto run = [&](auto kern, int smem, std::atomic<bool>* configured) -> cudaError_t {
        if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
            cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (err == cudaSuccess) err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (err != cudaSuccess) return err;
            if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
        }
        cfg.dynamicSmemBytes = smem;
        return cudaLaunchKernelEx(&cfg, kern, tk, tv, a);
    };
    auto by_type = [&](auto h, auto wide) -> cudaError_t {
        constexpr int kH = decltype(h)::value, D = decltype(wide)::value, smem = DCfg<kH, D>::kSmemBytes;
        static std::atomic<bool> configured[4][64];
        if (a.drop.threshold != 0ull)
            return bf16 ? run(decode_kernel<true, kH, D, true>, smem, configured[0]) : run(decode_kernel<false, kH, D, true>, smem, configured[1]);
        return bf16 ? run(decode_kernel<true, kH, D, false>, smem, configured[2]) : run(decode_kernel<false, kH, D, false>, smem, configured[3]);
    };
    auto by_dim = [&](auto h) -> cudaError_t {
        return a.head_dim <= 64 ? by_type(h, std::integral_constant<int, 64>()) : by_type(h, std::integral_constant<int, 128>());
    };
    switch (a.columns) {
        case 1: return by_dim(std::integral_constant<int, 1>());
        case 4: return by_dim(std::integral_constant<int, 4>());
        case 8: return by_dim(std::integral_constant<int, 8>());
        default: return by_dim(std::integral_constant<int, 16>());
    }
}

}  // namespace fa
