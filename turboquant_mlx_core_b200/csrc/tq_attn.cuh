// The compressed cache's storage and the kernels on it (tq_kv_kernels.cu, tq_attention.cu), and the fp16 decode window.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace tq {

// ---- storage of the compressed cache -----------------------------------------------------------------
// A layer's storage is one allocation of blocks [16-token tile][KV head].  A block holds the 16 tokens' records of one
// head in the order the attention kernel consumes them, so a tile is ONE contiguous bulk copy whatever the head count
// (the reference's token-major arrays took six copies per tile, or one per token and array beyond four heads).  A byte
// is an entry of the kernel's table of code PAIRS:
//   keys    16 tokens x D/2 bytes.  Byte b of a token: codes of dims 2b (bits 0-2) and 2b + 1 (bits 3-5), and the signs of
//           their residuals in bits 6 and 7.
//   values  8 token pairs x 8 groups of D/8 dims.  A byte holds one dim's codes of an even token (bits 0-2) and the odd
//           token after it (bits 3-5): the operand of the value product wants two tokens side by side.  D = 128 packs a
//           group's 16 dims into three words: bytes for the first 12, and the six bits of dim 12 + i's byte two by two in
//           bits 6 and 7 of byte i of the three words - 48 bytes per token.  Words 0 and 1 of all (pair, group) come
//           first, then word 2.  Other D: a byte per dim, bits 6 and 7 zero.
//   norms   16 x (key norm, value norm), then 16 residual norms (fp32)
// D = 128: 124 bytes per token and head (the reference's words of ten codes: 132).  Snapshots, deltas and exports convert
// to and from the reference's arrays (tq_kv_kernels.cu).
constexpr int kKvTile = 16;
template <int D>
struct KvBlock {
    static constexpr int kKeyBytes = kKvTile * D / 2;
    static constexpr int kValueBytes = D == 128 ? kKvTile * 48 : kKvTile * D / 2;
    static constexpr int kValueOff = kKeyBytes, kNormOff = kKeyBytes + kValueBytes;
    static constexpr int kBytes = kNormOff + 3 * kKvTile * 4;
    static_assert(kBytes % 16 == 0, "a block is a bulk copy");
};
__host__ __device__ constexpr size_t kv_block_bytes(int dim) {
    return static_cast<size_t>(kKvTile) * dim / 2 + (dim == 128 ? kKvTile * 48 : kKvTile * dim / 2) + 3 * kKvTile * 4;
}
// Bytes of a layer's storage for `cap` tokens (a multiple of 16).
inline size_t kv_layer_bytes(int cap, int heads, int dim) { return static_cast<size_t>(cap / kKvTile) * heads * kv_block_bytes(dim); }

// The value words of (token pair p of the tile, dim group g): words 0 and 1, and word 2, of a D = 128 block; the first
// of the D/32 words of other blocks.
__host__ __device__ __forceinline__ uint32_t* kv_value01(unsigned char* block, int p, int g) {
    return reinterpret_cast<uint32_t*>(block + KvBlock<128>::kValueOff) + (p * 8 + g) * 2;
}
__host__ __device__ __forceinline__ uint32_t* kv_value2(unsigned char* block, int p, int g) {
    return reinterpret_cast<uint32_t*>(block + KvBlock<128>::kValueOff + 512) + p * 8 + g;
}
__host__ __device__ __forceinline__ uint32_t* kv_value_row(unsigned char* block, int dim, int p, int g) {
    return reinterpret_cast<uint32_t*>(block + kKvTile * dim / 2) + (p * 8 + g) * (dim / 32);
}
// The bytes of a packed group's last four dims.
__host__ __device__ __forceinline__ uint32_t kv_value_spare(uint32_t w0, uint32_t w1, uint32_t w2) {
    return ((w0 >> 6) & 0x03030303u) | ((w1 >> 4) & 0x0C0C0C0Cu) | ((w2 >> 2) & 0x30303030u);
}
// ... and the other way, their bits for word k.
__host__ __device__ __forceinline__ uint32_t kv_spare_bits(uint32_t spare, int k) { return ((spare >> (2 * k)) & 0x03030303u) << 6; }
// Norms of a block: index into its floats from kNormOff on.
__host__ __device__ constexpr int kv_key_norm(int slot) { return 2 * slot; }
__host__ __device__ constexpr int kv_value_norm(int slot) { return 2 * slot + 1; }
__host__ __device__ constexpr int kv_residual_norm(int slot) { return 2 * kKvTile + slot; }
// The bits of value word k that belong to the odd token of its pair (the others: the even token's).
__host__ __device__ __forceinline__ uint32_t kv_odd_bits(int dim, int k) {
    return dim != 128 ? 0xF8F8F8F8u : (k == 0 ? 0x38383838u : (k == 1 ? 0xB8B8B8B8u : 0xF8F8F8F8u));
}

// One append: `tokens` tokens of a layer, from token `first` on, written to the storage at `base`.
struct KvSegment {
    unsigned char* base;
    int first;
};
constexpr int kKvMaxSegments = 32;
void launch_kv_encode(const void* keys, const void* values, bool is_f16, int tokens_per_seg, int heads, int dim, uint32_t k_seed,
                      uint32_t v_seed, uint32_t qjl_seed, const KvSegment* segs, int n_segs, cudaStream_t stream);
// fp16 [tokens, heads, dim] of tokens [start, start + tokens).
void launch_kv_decode_f16(const unsigned char* base, int start, int tokens, int heads, int dim, bool values, uint32_t wht_seed,
                          __half* out, cudaStream_t stream);
// The reference's token-major arrays (src/kv_cache.cpp:119-128; ceil(D/10) words of ten codes, norms, sign words, sign
// norms) of tokens [start, start + tokens), out of the storage or into it.
struct KvArrays {
    uint32_t *k_words, *v_words;
    float *k_norms, *v_norms;
    uint32_t* qjl_words;
    float* qjl_norms;
};
void launch_kv_unpack(const unsigned char* base, int start, int tokens, int heads, int dim, const KvArrays& out, cudaStream_t stream);
void launch_kv_pack(unsigned char* base, int start, int tokens, int heads, int dim, const KvArrays& in, cudaStream_t stream);

// ---- decode attention over the compressed cache (tq_attention.cu) --------------------------------------
// One sequence of a call: the layer's storage and the token range [start, end) the query attends to.  tile0 counts the
// tiles of the sequences before it.
struct AttnSeq {
    const unsigned char* base;
    int start, end, tile0, pad;
};
// A decode step moves every range by a token, so the descriptors of up to kAttnInlineSeqs sequences travel as kernel
// parameters (24 bytes each): a table in device memory cost an upload per call, and the copy between two kernels a gap
// in the stream.  Larger batches use the table.
constexpr int kAttnInlineSeqs = 32;
struct AttnSeqs {
    const AttnSeq* table;              // nullptr: the descriptors are in `inl`
    AttnSeq inl[kAttnInlineSeqs];
};
__device__ __forceinline__ AttnSeq attn_seq(const AttnSeqs& s, int i) { return s.table != nullptr ? s.table[i] : s.inl[i]; }

// The pair table holds kAttnCentroidScale * centroid: with this factor all four centroid
// magnitudes round to fp16 with a relative error below 1.4e-5 (unscaled: up to 3e-4, which the
// softmax amplifies); the factor is divided out of the key and value norms.
constexpr float kAttnCentroidScale = 1.1979075f;
// The decode window's lazy softmax reference (tq_attn_dense.cu): it only moves when a score exceeds it by more than this.
constexpr float kAttnSoftmaxSlack = 2.0f;

// Sets the descriptors' tile0 and returns the tiles of all sequences; `longest`, `shortest`: of the longest, of the shortest.
long attn_number_tiles(AttnSeq* seqs, int n_seqs, long* longest, long* shortest);
// How the work is cut: a team's tiles are a range.  parts != 0: each job (sequence, KV head, 8 query heads) is so many ranges; whole_jobs: a range is
// whole jobs; otherwise all ranges have an equal share of the tiles.  units: the tiles of all jobs.
struct AttnPlan {
    int ranges, parts, whole_jobs;
};
AttnPlan attn_plan(int head_dim, long jobs, long units, long longest, long shortest, int sm_count);
constexpr int kAttnJobHeads = 8;
size_t attn_scratch_bytes(int dim, int sm_count);
size_t attn_counters(int n_seqs, int q_heads, int kv_heads);   // zeroed words; every launch leaves them zero
void launch_kv_attention(const AttnSeqs& seqs, int n_seqs, long tiles, long longest, long shortest, const void* q, bool q_is_f16, int q_heads, int kv_heads, int head_dim,
                         uint32_t k_seed, uint32_t v_seed, uint32_t qjl_seed, bool use_qjl, void* scratch, unsigned int* counters,
                         __half* out, float* lse, unsigned int* status, int sm_count, cudaStream_t stream);

// fp16 decode window (tq_attn_dense.cu): ring writes / reads and scaled-dot-product attention over a
// contiguous run of ring slots.  `row` = heads * head_dim.
void launch_ring_write(const void* keys, const void* values, bool is_f16, long n_tokens, long src_token0, int row, int window,
                       long slot0, __half* ring_k, __half* ring_v, cudaStream_t stream);
void launch_ring_read(const __half* ring, long n_tokens, int row, int window, long start, __half* out, cudaStream_t stream);
int dense_attention_splits(int n_tokens, int kv_heads, int q_heads, int sm_count);
size_t dense_attention_scratch_bytes(int q_heads, int head_dim, int n_splits);
void launch_dense_attention(const __half* keys, const __half* values, int n_tokens, int kv_heads, int head_dim, const void* q,
                            bool q_is_f16, int q_heads, int n_splits, size_t l2_bytes, void* scratch, __half* out, cudaStream_t stream);

}  // namespace tq
