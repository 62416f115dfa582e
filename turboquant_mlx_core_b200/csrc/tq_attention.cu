// Decode attention over the compressed cache: one query position per sequence, all query heads of a KV head at once.
//
// Scores need no un-rotation: q . k = norm_k / sqrt(D) * sum_j c[code_j] (H(s o q))_j / sqrt(D), so the query is rotated
// once, values are accumulated in the rotated domain, and the sum is un-rotated once at the end.
//
// Tile body (a warp, 16 tokens of one KV head, up to 8 query heads), products on mma.sync.m16n8k16 (fp16 in, fp32 out):
//   S^T [16 tokens x 8 heads]  = K [16 x D] . Qrot^T           centroids
//   S2^T                        = Sgn [16 x D] . Qsgn^T         the residual's signs (use_qjl)
//   O^T [D dims x 8 heads]     += V^T [D x 16] . P^T
// A storage byte holds the codes of two neighbouring dims (tq_attn.cuh).  One byte permutation makes it a table address
// (256 entries of 256 bytes at the fixed window address 0x10000, entry e at 0x10000 + 256 e, a private copy per lane, so
// lookups meet no bank conflict), and the table's word is the fp16 pair the fragment needs: two instructions per pair,
// where words of ten 3-bit codes took a shift, a mask and a load.  The order in which a thread takes its dims is the same
// on both operands and undone at the end.  Value fragments are transposed in registers (movmatrix).
//
// Work split.  A job is (sequence, KV head, group of 8 query heads); its tiles are consecutive in a flat numbering of all
// tiles of the call, which is cut into equal ranges, one per CTA - one CTA per SM, whatever the mix of lengths.  A CTA
// walks its range job by job: its 16 warps take the job's tiles in turn, each through a ring of its own (one
// cp.async.bulk per tile, no synchronisation between warps), and merge their (max, sum, accumulator) in shared memory.
// A job that lies in one range is finished there; the parts of one that several ranges share go to scratch, and the CTA
// that arrives last (a counter per job) adds them in range order - the result does not depend on timing - un-rotates
// and writes.  One launch, no combine kernel.
//
// Bound: issue slots and the shared-memory pipe (about 330 warp instructions and 90 shared wavefronts per tile) ahead of
// DRAM.
#include <cmath>

#include "tq_attn.cuh"
#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

__constant__ float kC3[8] = {-2.152176f, -1.344318f, -0.756130f, -0.245379f, 0.245379f, 0.756130f, 1.344318f, 2.152176f};

constexpr uint32_t kTabAddr = 0x10000u, kTabBytes = 0x10000u;   // window address and size of the pair table
constexpr uint32_t kLowBase = 0x800u;                           // shared memory below is the runtime's and the statics'
constexpr int kGroup = 8;                                       // query heads of a job
constexpr unsigned long long kWaitLimitNs = 200ull * 1000 * 1000;

template <int D>
struct AttnCfg {
    static constexpr int kWarps = D == 256 ? 8 : 16;            // 256 dims: 64 accumulator registers
    static constexpr int kThreads = 32 * kWarps;
    static constexpr int kStages = D == 256 ? 3 : 4;
    static constexpr int kRing = kStages * KvBlock<D>::kBytes;  // bytes of a warp's ring
    static constexpr int kLowRings = (kTabAddr - kLowBase) / kRing < static_cast<uint32_t>(kWarps) ? (kTabAddr - kLowBase) / kRing : kWarps;
    static constexpr int kAccStride = D + 4;                    // floats per head of a published accumulator
    static constexpr uint32_t kHighBase = kTabAddr + kTabBytes;
    static constexpr int kQStride = D + 8;                      // halves per rotated query
    static constexpr uint32_t kOffQ = kHighBase + (kWarps - kLowRings) * kRing;
    static constexpr uint32_t kOffOut = kOffQ + kGroup * kQStride * 2;
    static constexpr uint32_t kOffMl = kOffOut + kGroup * kAccStride * 4;      // [2][warps][8]
    static constexpr uint32_t kEnd = kOffMl + 2 * kWarps * kGroup * 4;
    static constexpr int kPartFloats = kGroup * D + 2 * kGroup;                // a job part in scratch: accumulators, then (max, sum)
    static_assert(kRing >= kGroup * kAccStride * 4, "a warp publishes its accumulator through its ring");
    static_assert(kOffQ % 16 == 0 && kOffOut % 16 == 0, "alignment");
    static_assert(kEnd <= 227u * 1024u + 1024u, "shared memory of an SM");
};

struct AttnArgs {
    AttnSeqs seqs;
    const void* q;
    __half* out;
    float* lse;
    float* part;               // [CTA][2][kPartFloats]
    unsigned int* counters;    // [job]
    unsigned int* status;
    int q_is_f16, n_seqs, q_heads, kv_heads, gchunks, units;
    uint32_t k_seed, v_seed, qjl_seed;
    float inv_sqrt, inv_scale, score_scale, qscale;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned long long timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// False when the phase did not complete in time.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
        if (spin == 64) t0 = timer_ns();
        if (spin > 64 && (spin & 63) == 0 && timer_ns() - t0 > kWaitLimitNs) return false;
    }
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}
// The table word of byte BYTE of `word`: address = lane constant with its second byte replaced (byte 1 the entry,
// byte 0 the lane's copy, bytes 2 and 3 the table's base).
template <int BYTE>
__device__ __forceinline__ uint32_t pair_addr(uint32_t word, uint32_t lane_const) {
    return __byte_perm(word, lane_const, 0x7604u | (static_cast<uint32_t>(BYTE) << 4));
}
__device__ __forceinline__ uint32_t table_load(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// Words of one token of a nibble array: word w of thread q's quarter.
template <int W>
__device__ __forceinline__ void load_words(uint32_t (&w)[W], uint32_t addr) {
    if constexpr (W % 4 == 0) {
#pragma unroll
        for (int i = 0; i < W; i += 4)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]) : "r"(addr + 4 * i));
    } else if constexpr (W == 2) {
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr));
    } else {
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[0]) : "r"(addr));
    }
}
__device__ __forceinline__ float load_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

template <int D, bool QJL>
__global__ void __launch_bounds__(AttnCfg<D>::kThreads, 1) attn_kernel(const __grid_constant__ AttnArgs a) {
    using C = AttnCfg<D>;
    using B = KvBlock<D>;
    constexpr int kSteps = D / 16;   // k steps of a score product = m tiles of the value product
    constexpr int W = D / 32;        // nibble words of a token that a thread takes
    extern __shared__ __align__(16) unsigned char attn_smem[];
    __shared__ __align__(8) unsigned long long s_bars[C::kWarps * C::kStages];
    __shared__ unsigned int s_last;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(attn_smem));
    if (base > kLowBase) {   // layout assumption broken: refuse to run
        if (tid == 0) raise_status(a.status, 1u);
        return;
    }
    auto at = [&](uint32_t window) { return attn_smem + (window - base); };
    const uint32_t ring = warp < C::kLowRings ? kLowBase + warp * C::kRing : C::kHighBase + (warp - C::kLowRings) * C::kRing;
    const uint32_t bars = static_cast<uint32_t>(__cvta_generic_to_shared(&s_bars[warp * C::kStages]));
    __half* const s_q = reinterpret_cast<__half*>(at(C::kOffQ));
    float* const s_out = reinterpret_cast<float*>(at(C::kOffOut));
    float* const s_m = reinterpret_cast<float*>(at(C::kOffMl));
    float* const s_l = s_m + C::kWarps * kGroup;

    if (lane == 0) {
        for (int s = 0; s < C::kStages; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8u * s), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The table does not depend on the kernels before this one.  Entry: [32 lanes] centroid pair, [32 lanes] sign pair.
    for (int i = tid; i < 256 * 16; i += C::kThreads) {
        const int e = i >> 4, part = i & 15;   // 4 copies per store
        const uint32_t v = part < 8 ? pack_half2(kAttnCentroidScale * kC3[e & 7], kAttnCentroidScale * kC3[(e >> 4) & 7])
                                    : ((e & 8) ? 0x3C00u : 0xBC00u) | ((e & 128) ? 0x3C000000u : 0xBC000000u);
        *reinterpret_cast<uint4*>(at(kTabAddr + e * 256 + part * 16)) = make_uint4(v, v, v, v);
    }
    pdl_wait_release();

    const uint32_t lane_const = kTabAddr | static_cast<uint32_t>(lane * 4);
    const int cta = static_cast<int>(blockIdx.x), n_ctas = static_cast<int>(gridDim.x);
    const int u_end = static_cast<int>(static_cast<long>(a.units) * (cta + 1) / n_ctas);
    const int jobs_per_seq = a.kv_heads * a.gchunks, G = a.q_heads / a.kv_heads;
    uint32_t phase = 0;      // bit s: parity of the next completion of stage s
    int stage = 0;
    bool ok = true;

    for (int u = static_cast<int>(static_cast<long>(a.units) * cta / n_ctas); u < u_end;) {
        // ---- which job, which of its tiles ----
        int lo = 0, hi = a.n_seqs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (attn_seq(a.seqs, mid).tile0 * jobs_per_seq <= u) lo = mid;
            else hi = mid - 1;
        }
        const AttnSeq S = attn_seq(a.seqs, lo);
        const int first_tile = S.start / kKvTile, tiles = (S.end + kKvTile - 1) / kKvTile - first_tile;
        const int in_seq = u - S.tile0 * jobs_per_seq;
        const int hg = in_seq / tiles, tile0 = in_seq - hg * tiles;
        const int n_tiles = min(u_end - u, tiles - tile0);
        const int kvh = hg / a.gchunks, g0 = (hg - kvh * a.gchunks) * kGroup, ng = min(kGroup, G - g0);
        const int q_row0 = lo * a.q_heads + kvh * G + g0;
        const int job = lo * jobs_per_seq + hg, job_u0 = u - tile0;
        u += n_tiles;

        const unsigned char* const src = S.base + (static_cast<size_t>(first_tile + tile0) * a.kv_heads + kvh) * B::kBytes;
        const size_t tile_stride = static_cast<size_t>(a.kv_heads) * B::kBytes;
        const int mine = n_tiles > warp ? (n_tiles - warp + C::kWarps - 1) / C::kWarps : 0;   // tiles warp, warp + kWarps, ...
        if (lane == 0) {
            for (int i = 0; i < min(mine, C::kStages); ++i) {
                const int s = (stage + i) % C::kStages;
                bulk_copy(ring + s * B::kBytes, src + static_cast<size_t>(warp + i * C::kWarps) * tile_stride, B::kBytes, bars + 8u * s);
            }
        }
        // ---- rotated queries: fp16-round, sign, butterfly, 1 / sqrt(D), fp16-round (a warp per head) ----
        if (warp < kGroup) {
            constexpr int E = D / 32;
            float v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int d = lane * E + j;
                float t = 0.f;
                if (warp < ng) {
                    const size_t qi = static_cast<size_t>(q_row0 + warp) * D + d;
                    t = a.q_is_f16 ? __half2float(static_cast<const __half*>(a.q)[qi])
                                   : __half2float(__float2half_rn(static_cast<const float*>(a.q)[qi]));
                }
                v[j] = t * sign_value(a.k_seed, static_cast<uint32_t>(d));
            }
            warp_fwht<E>(v, lane);
#pragma unroll
            for (int j = 0; j < E; ++j) s_q[warp * C::kQStride + lane * E + j] = __float2half_rn(v[j] * a.inv_sqrt);
        }
        __syncthreads();
        // B fragments of head g.  Pair p of thread q: dims (D/4) q + 2 p and the next.  Sign pair 4 w + r: dims 8 w + r
        // and 8 w + r + 4 of the quarter, the sign of the residual's own rotation folded in.
        uint32_t bq[2 * kSteps], bs[QJL ? 2 * kSteps : 1];
        {
            const __half* const sq = s_q + g * C::kQStride + (D / 4) * q;
#pragma unroll
            for (int p = 0; p < 2 * kSteps; ++p) bq[p] = *reinterpret_cast<const uint32_t*>(sq + 2 * p);
            if constexpr (QJL) {
#pragma unroll
                for (int p = 0; p < 2 * kSteps; ++p) {
                    const int d0 = 8 * (p / 4) + p % 4, d1 = d0 + 4;
                    const uint32_t s0 = qjl_sign_is_positive(a.qjl_seed, static_cast<uint32_t>((D / 4) * q + d0)) ? 0u : 0x8000u;
                    const uint32_t s1 = qjl_sign_is_positive(a.qjl_seed, static_cast<uint32_t>((D / 4) * q + d1)) ? 0u : 0x80000000u;
                    bs[p] = (static_cast<uint32_t>(__half_as_ushort(sq[d0])) | (static_cast<uint32_t>(__half_as_ushort(sq[d1])) << 16)) ^ (s0 | s1);
                }
            }
        }

        float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // heads 2q, 2q + 1; in units of log2
        float acc[kSteps][4];
#pragma unroll
        for (int mt = 0; mt < kSteps; ++mt)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[mt][k] = 0.f;

        int token = (first_tile + tile0 + warp) * kKvTile + g;   // this thread's tokens of the tile: token, token + 8
        for (int i = 0; i < mine; ++i, token += C::kWarps * kKvTile) {
            if (!bar_wait(bars + 8u * stage, (phase >> stage) & 1u)) {
                ok = false;
                break;
            }
            const uint32_t blk = ring + stage * B::kBytes;
            // ---- scores ----
            float c1[4] = {0.f, 0.f, 0.f, 0.f}, c1b[4] = {0.f, 0.f, 0.f, 0.f};
            {
                uint32_t ka[W], kb[W];
                load_words<W>(ka, blk + g * (D / 2) + q * (D / 8));
                load_words<W>(kb, blk + (g + 8) * (D / 2) + q * (D / 8));
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    mma_f16(c1, table_load(pair_addr<0>(ka[w], lane_const)), table_load(pair_addr<0>(kb[w], lane_const)),
                            table_load(pair_addr<1>(ka[w], lane_const)), table_load(pair_addr<1>(kb[w], lane_const)), bq[4 * w], bq[4 * w + 1]);
                    mma_f16(c1b, table_load(pair_addr<2>(ka[w], lane_const)), table_load(pair_addr<2>(kb[w], lane_const)),
                            table_load(pair_addr<3>(ka[w], lane_const)), table_load(pair_addr<3>(kb[w], lane_const)), bq[4 * w + 2], bq[4 * w + 3]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) c1[k] += c1b[k];
                if constexpr (QJL) {
                    float c2[4] = {0.f, 0.f, 0.f, 0.f}, c2b[4] = {0.f, 0.f, 0.f, 0.f};
                    // sign bits of nibbles r and r + 4 -> fp16 pair (+-1, +-1): the shifted bits over the pattern of (-1, -1)
                    auto sgn = [](uint32_t w, int r) { return ((w << (12 - 4 * r)) & 0x80008000u) ^ 0xBC00BC00u; };
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        mma_f16(c2, sgn(ka[w], 0), sgn(kb[w], 0), sgn(ka[w], 1), sgn(kb[w], 1), bs[4 * w], bs[4 * w + 1]);
                        mma_f16(c2b, sgn(ka[w], 2), sgn(kb[w], 2), sgn(ka[w], 3), sgn(kb[w], 3), bs[4 * w + 2], bs[4 * w + 3]);
                    }
                    const float qa = load_f32(blk + B::kNormOff + 2 * kKvTile * 4 + g * 4) * a.qscale;
                    const float qb = load_f32(blk + B::kNormOff + 2 * kKvTile * 4 + (g + 8) * 4) * a.qscale;
                    c1[0] = fmaf(qa, c2[0] + c2b[0], c1[0]);
                    c1[1] = fmaf(qa, c2[1] + c2b[1], c1[1]);
                    c1[2] = fmaf(qb, c2[2] + c2b[2], c1[2]);
                    c1[3] = fmaf(qb, c2[3] + c2b[3], c1[3]);
                }
            }
            const bool va = token >= S.start && token < S.end, vb = token + 8 >= S.start && token + 8 < S.end;
            const float kna = load_f32(blk + B::kNormOff + g * 4) * a.score_scale, knb = load_f32(blk + B::kNormOff + (g + 8) * 4) * a.score_scale;
            float vna = load_f32(blk + B::kNormOff + kKvTile * 4 + g * 4), vnb = load_f32(blk + B::kNormOff + kKvTile * 4 + (g + 8) * 4);
            vna = va ? vna * (1.0f / kAttnCentroidScale) : 0.f;
            vnb = vb ? vnb * (1.0f / kAttnCentroidScale) : 0.f;
            const float s00 = va ? c1[0] * kna : -INFINITY, s01 = va ? c1[1] * kna : -INFINITY;
            const float s10 = vb ? c1[2] * knb : -INFINITY, s11 = vb ? c1[3] * knb : -INFINITY;
            // value words, then the stage can be refilled
            uint32_t xa[W], xb[W];
            if constexpr (D == 128) {
                uint32_t t[2];
                load_words<2>(t, blk + B::kValueOff + g * 32 + q * 8);
                xa[0] = t[0];
                xa[1] = t[1];
                load_words<2>(t, blk + B::kValueOff + (g + 8) * 32 + q * 8);
                xb[0] = t[0];
                xb[1] = t[1];
                uint32_t o[1];
                load_words<1>(o, blk + B::kValueOff + 512 + g * 16 + q * 4);
                xa[2] = o[0];
                load_words<1>(o, blk + B::kValueOff + 512 + (g + 8) * 16 + q * 4);
                xb[2] = o[0];
                xa[3] = kv_value_spare(xa[0], xa[1], xa[2]);
                xb[3] = kv_value_spare(xb[0], xb[1], xb[2]);
            } else {
                load_words<W>(xa, blk + B::kValueOff + g * (D / 2) + q * (D / 8));
                load_words<W>(xb, blk + B::kValueOff + (g + 8) * (D / 2) + q * (D / 8));
            }
            __syncwarp();
            if (lane == 0 && i + C::kStages < mine)
                bulk_copy(blk, src + static_cast<size_t>(warp + (i + C::kStages) * C::kWarps) * tile_stride, B::kBytes, bars + 8u * stage);
            phase ^= 1u << stage;
            stage = stage + 1 == C::kStages ? 0 : stage + 1;

            // ---- online softmax with a lazy reference: it moves (and the sums are rescaled) only when some score exceeds
            // it by more than the slack, so the usual tile needs one vote instead of a reduction over the tokens.  Every
            // tile holds a token of [start, end), so the reference is finite from a warp's first tile on.
            constexpr float kSlack = kAttnSoftmaxSlack * 1.4426950408889634f;
            const float tm0 = fmaxf(s00, s10), tm1 = fmaxf(s01, s11);
            if (__any_sync(0xffffffffu, tm0 > m_run[0] + kSlack || tm1 > m_run[1] + kSlack)) {
                float mx0 = tm0, mx1 = tm1;
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
                    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
                }
                const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
                const float cr0 = exp2_approx(m_run[0] - mn0), cr1 = exp2_approx(m_run[1] - mn1);
                l_run[0] *= cr0;
                l_run[1] *= cr1;
                m_run[0] = mn0;
                m_run[1] = mn1;
#pragma unroll
                for (int mt = 0; mt < kSteps; ++mt) {
                    acc[mt][0] *= cr0;
                    acc[mt][1] *= cr1;
                    acc[mt][2] *= cr0;
                    acc[mt][3] *= cr1;
                }
            }
            const float p00 = exp2_approx(s00 - m_run[0]), p01 = exp2_approx(s01 - m_run[1]);
            const float p10 = exp2_approx(s10 - m_run[0]), p11 = exp2_approx(s11 - m_run[1]);
            l_run[0] += p00 + p10;
            l_run[1] += p01 + p11;
            // P^T fragment: (tokens 2q, 2q+1 | 2q+8, 2q+9 ; head g) from (token g | g+8 ; heads 2q, 2q+1)
            const uint32_t pb0 = movmatrix_trans(pack_half2(p00 * vna, p01 * vna));
            const uint32_t pb1 = movmatrix_trans(pack_half2(p10 * vnb, p11 * vnb));
            // ---- values: V [token x dim] fragments -> V^T [dim x token] ----
#pragma unroll
            for (int w = 0; w < W; ++w) {
                mma_f16(acc[2 * w], movmatrix_trans(table_load(pair_addr<0>(xa[w], lane_const))), movmatrix_trans(table_load(pair_addr<1>(xa[w], lane_const))),
                        movmatrix_trans(table_load(pair_addr<0>(xb[w], lane_const))), movmatrix_trans(table_load(pair_addr<1>(xb[w], lane_const))), pb0, pb1);
                mma_f16(acc[2 * w + 1], movmatrix_trans(table_load(pair_addr<2>(xa[w], lane_const))), movmatrix_trans(table_load(pair_addr<3>(xa[w], lane_const))),
                        movmatrix_trans(table_load(pair_addr<2>(xb[w], lane_const))), movmatrix_trans(table_load(pair_addr<3>(xb[w], lane_const))), pb0, pb1);
            }
        }

        // ---- merge the warps: every warp publishes through its ring, which is idle now ----
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
            l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
        }
        if (g == 0) {
            s_m[warp * kGroup + 2 * q] = m_run[0];
            s_m[warp * kGroup + 2 * q + 1] = m_run[1];
            s_l[warp * kGroup + 2 * q] = l_run[0];
            s_l[warp * kGroup + 2 * q + 1] = l_run[1];
        }
        {
            float* const mine_acc = reinterpret_cast<float*>(at(ring));
            // row slot of an m tile: slot = g + 8 half -> thread (slot & 7) / 2 of a quad, pair 2 mt + half, low or high code
            const int d0 = (D / 4) * (g >> 1) + (g & 1);
#pragma unroll
            for (int mt = 0; mt < kSteps; ++mt)
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const int d = d0 + 2 * (2 * mt + hf);
                    mine_acc[(2 * q) * C::kAccStride + d] = acc[mt][2 * hf];
                    mine_acc[(2 * q + 1) * C::kAccStride + d] = acc[mt][2 * hf + 1];
                }
        }
        __syncthreads();
        const bool whole = n_tiles == tiles;
        // which ranges share the job: the range of flat tile x is ((x + 1) n_ctas - 1) / units
        const int c_first = whole ? cta : static_cast<int>((static_cast<long>(job_u0 + 1) * n_ctas - 1) / a.units);
        const int c_last = whole ? cta : static_cast<int>((static_cast<long>(job_u0 + tiles) * n_ctas - 1) / a.units);
        float* const my_part = a.part + static_cast<size_t>(2 * cta + (tile0 == 0 ? 1 : 0)) * C::kPartFloats;
        for (int idx = tid; idx < kGroup * D; idx += C::kThreads) {
            const int h = idx / D, d = idx - h * D;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < C::kWarps; ++w) M = fmaxf(M, s_m[w * kGroup + h]);
            float L = 0.f, A = 0.f;
#pragma unroll
            for (int w = 0; w < C::kWarps; ++w) {
                const float m = s_m[w * kGroup + h];
                const float f = m == -INFINITY ? 0.f : exp2_approx(m - M);
                const float* const wa = reinterpret_cast<const float*>(at(w < C::kLowRings ? kLowBase + w * C::kRing : C::kHighBase + (w - C::kLowRings) * C::kRing));
                L = fmaf(s_l[w * kGroup + h], f, L);
                A = fmaf(wa[h * C::kAccStride + d], f, A);
            }
            if (whole) {
                s_out[h * C::kAccStride + d] = A;
            } else {
                my_part[idx] = A;
                if (d == 0) {
                    my_part[kGroup * D + 2 * h] = M;
                    my_part[kGroup * D + 2 * h + 1] = L;
                }
            }
            if (whole && d == 0) {
                s_out[h * C::kAccStride + D] = M;
                s_out[h * C::kAccStride + D + 1] = L;
            }
        }
        bool finish = whole;
        if (!whole) {
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                const unsigned int prev = atomicAdd(&a.counters[job], 1u);
                s_last = prev == static_cast<unsigned int>(c_last - c_first) ? 1u : 0u;
                if (s_last) a.counters[job] = 0u;   // ready for the next launch
            }
            __syncthreads();
            finish = s_last != 0u;
            if (finish) {
                __threadfence();
                auto part_of = [&](int c) {
                    // the first range's part of the job starts at its tile 0
                    return a.part + static_cast<size_t>(2 * c + (c == c_first ? 1 : 0)) * C::kPartFloats;
                };
                for (int idx = tid; idx < kGroup * D; idx += C::kThreads) {
                    const int h = idx / D, d = idx - h * D;
                    float M = -INFINITY, L = 0.f, A = 0.f;
                    for (int c0 = c_first; c0 <= c_last; c0 += 4) {   // four parts at a time, added in order
                        float pm[4], pl[4], pa[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float* const p = part_of(min(c0 + k, c_last));
                            pm[k] = c0 + k <= c_last ? __ldcg(p + kGroup * D + 2 * h) : -INFINITY;
                            pl[k] = __ldcg(p + kGroup * D + 2 * h + 1);
                            pa[k] = __ldcg(p + idx);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (pm[k] == -INFINITY) continue;
                            const float mn = fmaxf(M, pm[k]);
                            const float f0 = exp2_approx(M - mn), f1 = exp2_approx(pm[k] - mn);
                            L = fmaf(L, f0, pl[k] * f1);
                            A = fmaf(A, f0, pa[k] * f1);
                            M = mn;
                        }
                    }
                    s_out[h * C::kAccStride + d] = A;
                    if (d == 0) {
                        s_out[h * C::kAccStride + D] = M;
                        s_out[h * C::kAccStride + D + 1] = L;
                    }
                }
            }
        }
        // generic accesses to the rings end here; the next job's bulk copies write them
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        // ---- un-rotate and write: out = (inv_sqrt * sign_v) o H(inv_scale * acc) / L, a warp per head ----
        if (finish && warp < ng) {
            constexpr int E = D / 32;
            const float M = s_out[warp * C::kAccStride + D], L = s_out[warp * C::kAccStride + D + 1];
            float v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = s_out[warp * C::kAccStride + lane * E + j] * a.inv_scale;
            warp_fwht<E>(v, lane);
            const float invL = L > 0.f ? 1.0f / L : 0.f;
            const size_t row = static_cast<size_t>(q_row0 + warp);
            // log of the softmax denominator: lets a caller merge results over disjoint token ranges
            if (a.lse != nullptr && lane == 0) a.lse[row] = L > 0.f ? M * 0.6931471805599453f + __logf(L) : -INFINITY;
#pragma unroll
            for (int j = 0; j < E; ++j)
                a.out[row * D + lane * E + j] = __float2half_rn(v[j] * a.inv_sqrt * sign_value(a.v_seed, static_cast<uint32_t>(lane * E + j)) * invL);
        }
        if (__syncthreads_or(!ok)) break;   // (also: s_out and s_q are free again)
    }
    if (!ok && lane == 0) {
        // let whatever was requested land before the shared memory is released
        raise_status(a.status, 11u);
        const unsigned long long t0 = timer_ns();
        while (timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
}

template <int D, bool QJL>
void launch_d(const AttnArgs& args, int grid, cudaStream_t stream) {
    using C = AttnCfg<D>;
    // the window starts at the dynamic memory's base, at most kLowBase; asking up to the end of the map covers any base
    constexpr int kSmem = static_cast<int>(C::kEnd - 0x400u);
    static bool configured[64] = {false};   // the opt-in size is a per-device attribute
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute(attn_kernel<D, QJL>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    launch_pdl(attn_kernel<D, QJL>, dim3(static_cast<unsigned>(grid)), dim3(C::kThreads), kSmem, stream, args);
}

}  // namespace

long attn_number_tiles(AttnSeq* seqs, int n_seqs) {
    long total = 0;
    for (int i = 0; i < n_seqs; ++i) {
        seqs[i].tile0 = static_cast<int>(total);
        total += (seqs[i].end + kKvTile - 1) / kKvTile - seqs[i].start / kKvTile;
    }
    return total;
}

size_t attn_scratch_bytes(int dim, int sm_count) { return static_cast<size_t>(sm_count) * 2 * (kGroup * dim + 2 * kGroup) * sizeof(float); }

size_t attn_counters(int n_seqs, int q_heads, int kv_heads) {
    return static_cast<size_t>(n_seqs) * kv_heads * ((q_heads / kv_heads + kGroup - 1) / kGroup);
}

void launch_kv_attention(const AttnSeqs& seqs, int n_seqs, long tiles, const void* q, bool q_is_f16, int q_heads, int kv_heads, int head_dim,
                         uint32_t k_seed, uint32_t v_seed, uint32_t qjl_seed, bool use_qjl, void* scratch, unsigned int* counters,
                         __half* out, float* lse, unsigned int* status, int sm_count, cudaStream_t stream) {
    if (n_seqs == 0) return;
    TQ_REQUIRE(q_heads % kv_heads == 0, "query heads must be a multiple of KV heads");
    AttnArgs a;
    a.seqs = seqs;
    a.q = q;
    a.out = out;
    a.lse = lse;
    a.part = static_cast<float*>(scratch);
    a.counters = counters;
    a.status = status;
    a.q_is_f16 = q_is_f16 ? 1 : 0;
    a.n_seqs = n_seqs;
    a.q_heads = q_heads;
    a.kv_heads = kv_heads;
    a.gchunks = (q_heads / kv_heads + kGroup - 1) / kGroup;
    const long units = tiles * kv_heads * a.gchunks;
    TQ_REQUIRE(units > 0 && units < (1L << 31), "attention: too many tokens for one call");
    a.units = static_cast<int>(units);
    a.k_seed = k_seed;
    a.v_seed = v_seed;
    a.qjl_seed = qjl_seed;
    const double d = head_dim;
    a.inv_sqrt = 1.0f / std::sqrt(static_cast<float>(head_dim));
    a.inv_scale = a.inv_sqrt;
    // softmax scale 1 / sqrt(D) (src/attention_dispatch.cpp:35) and the rotation's 1 / sqrt(D), in units of log2
    a.score_scale = static_cast<float>(1.4426950408889634 / d / kAttnCentroidScale);
    a.qscale = static_cast<float>(std::sqrt(2.0 / (3.14159265358979323846 * d)) * kAttnCentroidScale);
    // A CTA per SM while every CTA gets a tile per warp; fewer for short jobs, whose time is the merge of the parts.
    const int warps = head_dim == 256 ? 8 : 16;
    const int grid = static_cast<int>(std::min<long>(sm_count, std::max<long>(1, (units + warps - 1) / warps)));
#define TQ_ATT(DV)                                                   \
    case DV:                                                         \
        if (use_qjl) launch_d<DV, true>(a, grid, stream);            \
        else launch_d<DV, false>(a, grid, stream);                   \
        break;
    switch (head_dim) {
        TQ_ATT(32) TQ_ATT(64) TQ_ATT(128) TQ_ATT(256)
        default: throw Error("attention: head_dim must be 32, 64, 128 or 256");
    }
#undef TQ_ATT
}

}  // namespace tq
