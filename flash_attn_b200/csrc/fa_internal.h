// Internal declarations shared by the C-ABI translation unit and the kernels.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "philox.cuh"

namespace fa {

constexpr int kTile = 128;  // Br = Bc = 128, as the reference fixes them (src/main.cu:116-117)

// Division by a launch-constant divisor without the hardware's slow integer divide: the
// quotient is mulhi(x, m) with m = floor(2^32 / d) + 1, which is floor(x / d) or one more.
struct FastDiv {
    uint32_t d, m;
};
inline FastDiv make_fastdiv(uint32_t d) {
    FastDiv f;
    f.d = d < 1 ? 1 : d;
    f.m = f.d == 1 ? 0u : static_cast<uint32_t>((1ull << 32) / f.d) + 1u;
    return f;
}

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t fast_div(const FastDiv& f, uint32_t x) {
    if (f.d == 1) return x;
    uint32_t q = __umulhi(x, f.m);
    if (q * f.d > x) --q;
    return q;
}
#endif

// Device-side argument block of the tiled forward kernel (the successor of
// mykernelParamType, include/utils.h:21-44).  Q/K/V travel as TMA tensor maps.
struct FwdArgs {
    void* o;                // [units, Nq, d] in o dtype (non-split)
    float* lse;             // [units, Nq] or null
    float* o_partial;       // [units, splits, Nq, d] fp32 (split)
    float* lse_partial;     // [units, splits, Nq]
    const float* alibi_slopes;
    int* status;
    int heads;
    int units;              // batch * heads of this launch
    int unit_group;         // units whose CTAs are interleaved in launch order (1 = unit-major)
    int kv_group;           // query units per K/V unit (grouped-query attention); K/V unit = unit / kv_group
    int seqlen_q, seqlen_k, head_dim;
    int tr, tc;             // query / key tiles
    int pair;               // query tiles of a CTA: two, or one
    int num_splits, tiles_per_split;
    float scale_log2;       // softmax_scale * log2(e)
    int is_causal, window_left, window_right;
    long long q_pos0, k_pos0;
    int o_is_fp32;
    int o_tma;              // O leaves through the TMA store map (16-bit output, unsplit launch)
    float* accum_o;         // running fp32 result [units, Nq, d] merged in the epilogue, or null
    float* accum_lse;       // running log-sum-exp [units, Nq]
    int accum_first;        // nothing is carried yet: the running pair is only written
    int accum_final;        // last block: o / lse receive the merged result (the running O is then left as it is)
    // The launches whose rows leave through shared memory (fwd_tiled_kernel with kStaged):
    int staged;
    int parts;              // CTAs (one cluster) that share the keys of a query block
    int pack_rows;          // query rows per head when the heads of a K/V head are stacked into one unit, else 0
    int o_dim;              // columns (and row pitch) of O: head_dim, or less when Q, K, V are padded copies
    // launch order of the CTAs (filled by launch_fwd_tiled): divisors of the block index
    FastDiv div_group_ctas, div_gsize, div_last_gsize, div_splits, div_kv_group;
    FastDiv div_parts, div_pack, div_o_dim;
    DropoutParams drop;
};

constexpr int kUnitGroup = 16;  // units whose CTAs are interleaved in launch order where query blocks differ in length, at most

// Clusters that the device holds at once.  A cluster lies within a GPC, and GPCs differ in their SMs from device to device: a
// B200 with 148 SMs holds 74 clusters of 2 CTAs at one CTA an SM, 45 of 3, 33 of 4, 26 of 5, 22 of 6, 15 of 7 or 8, 7 of 16.
struct ClusterRoom {
    static constexpr int kMax = 16;
    int one_per_sm[kMax + 1];  // by size (1 to 8 and 16), with one CTA an SM
    int fits(int parts, int ctas_per_sm) const;
};
ClusterRoom cluster_room(int sms);  // of the current device; none above one CTA where the runtime does not say

// Decides how a launch is cut: pair and, without dropout, staged, parts and, for short grouped queries, a problem
// restated with the heads of a K/V head stacked (units, heads, kv_group, seqlen_q, tr, pack_rows).
void plan_tiled(FwdArgs* a, int sms, const ClusterRoom& room, bool dropout);

// Launchers implemented in the .cu files; all return a cudaError_t.  `to` is the store map of O, or of the running
// result where the launch leaves that (32-row boxes); it is read only when a.o_tma or a.accum_o is set.  `tc` is the load
// map of the running result, read only when a.accum_o is set and something is carried.
cudaError_t launch_fwd_tiled(const FwdArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                             const CUtensorMap& to, const CUtensorMap& tc, int units, bool bf16, bool dropout, cudaStream_t stream);

// ... for one head dimension and number of query tiles a CTA (each a unit of compilation of fa_fwd_tiled.cu).
typedef cudaError_t launch_tiled_fn(const FwdArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                    const CUtensorMap& to, const CUtensorMap& tc, int units, bool bf16, bool alibi, bool dropout, cudaStream_t stream);
launch_tiled_fn launch_tiled_64_1, launch_tiled_64_2, launch_tiled_128_1, launch_tiled_128_2;

// Device-side argument block of the decode kernel (seqlen_q <= 8).
struct DecodeArgs {
    const void* q;          // [units, seqlen_q, d]
    void* o;                // [units, seqlen_q, d] (a whole unit, or the parts of one merged in its cluster)
    float* lse;             // [units, seqlen_q] or null
    float* o_partial;       // [units, parts, seqlen_q, d] fp32 (parts left to the combine kernel)
    float* lse_partial;     // [units, parts, seqlen_q]
    const float* alibi_slopes;
    int* status;
    int heads;
    int kv_group;           // query units per K/V unit; K/V unit = unit / kv_group
    int columns;            // query columns of a CTA: 1, 4, 8 or 16
    int subgroups;          // CTAs (each a part of the group's heads) per K/V unit
    int seqlen_q;           // query rows per unit, 1..8
    int seqlen_k, head_dim;
    int o_dim;              // columns (and row pitch) of O: head_dim, or less when Q, K, V are padded copies
    int tc;                 // key tiles
    int vis_lo, vis_hi;     // key tiles that the masks leave visible to some query row: [vis_lo, vis_hi)
    int full_lo, full_hi;   // key tiles that no mask touches
    int parts;              // CTAs that share the keys of a unit
    int merge;              // the parts are one cluster and merge their results themselves
    int by_split;           // the parts are the caller's splits (dropout), tiles_per_split tiles each
    int tiles_per_split;
    float scale_log2;
    int is_causal, window_left, window_right;
    long long q_pos0, k_pos0;
    int o_is_fp32;
    FastDiv div_parts, div_subgroups;
    DropoutParams drop;
};
constexpr int kDecodeCluster = 16;  // parts of a unit that one cluster merges (above 8: non-portable cluster size)
constexpr int kDecodeParts = 64;    // parts at most
// How many CTAs, at most `most`, share the keys of a unit and how many columns each has (fills parts, merge, by_split, columns, subgroups and the
// tile ranges; the problem's fields are set).  `splits` is the resolved split count of the caller.  A plan with parts > 1
// and merge == 0 writes partials: they need a workspace, and the combine kernel behind.
void plan_decode(DecodeArgs* a, int units, int splits, int most, int sms, const ClusterRoom& room);
cudaError_t launch_decode(const DecodeArgs& a, const CUtensorMap& tk, const CUtensorMap& tv, int units, bool bf16,
                          cudaStream_t stream);

struct CombineArgs {
    const float* o_partial; const float* lse_partial;
    void* o; float* lse;
    long long rows_per_unit;   // Nq
    int num_splits, head_dim;
    int o_dim;                 // columns (and row pitch) of O, at most head_dim
    int o_dtype;               // FA_DTYPE_*
};
cudaError_t launch_combine(const CombineArgs& a, long long units, cudaStream_t stream);
cudaError_t launch_merge(float* o_acc, float* lse_acc, const void* o_part, const float* lse_part, int part_dtype,
                         long long rows, int d, cudaStream_t stream);
cudaError_t launch_cast(const float* src, void* dst, int o_dtype, long long n, cudaStream_t stream);
cudaError_t launch_repitch(const void* src, void* dst, int elem_bytes, long long rows, int d_src, int d_dst,
                           cudaStream_t stream);
// Q, K and V (16-bit rows of d_src elements) to rows of d_dst, in one launch.
cudaError_t launch_pad_qkv(const void* q, const void* k, const void* v, void* qp, void* kp, void* vp, long long rows_q,
                           long long rows_k, int d_src, int d_dst, cudaStream_t stream);
cudaError_t launch_dropout_mask(const FwdArgs& a, uint8_t* keep, long long units, cudaStream_t stream);

}  // namespace fa
