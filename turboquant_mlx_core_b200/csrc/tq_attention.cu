// Decode attention over the compressed cache: one query position per sequence, all query heads of a KV head at once.
//
// Scores need no un-rotation: q . k = norm_k / sqrt(D) * sum_j c[code_j] (H(s o q))_j / sqrt(D), so the query is rotated
// once, values are accumulated in the rotated domain, and the sum is un-rotated once at the end.
//
// Tile body (a warp, 16 tokens of one KV head, up to 8 query heads), products on mma.sync.m16n8k16 (fp16 in, fp32 out):
//   S^T [16 tokens x 8 heads]  = K [16 x D] . Qrot^T           centroids
//   S2^T                        = Sgn [16 x D] . Qsgn^T         the residual's signs (use_qjl)
//   O^T [D dims x 8 heads]     += V^T [D x 16] . P^T
// A storage byte holds a pair of codes (tq_attn.cuh): two dims of a key, or one dim of two tokens' values, as the two
// products want them.  One dot-product instruction makes it the address of a table entry (256 entries of 128 bytes, a
// private copy per lane, so lookups meet no bank conflict), and the entry is the fp16 pair the fragment needs: two
// instructions per pair, where words of ten 3-bit codes took a shift, a mask and a load, and values a transposition
// (movmatrix) on top, which the shared-memory pipe carries.  The order in which a thread takes its dims is the same on both
// operands and undone at the end.
//
// Work split.  A job is (sequence, KV head, group of 8 query heads); its tiles are consecutive in a flat numbering of all
// tiles of the call, which is cut into equal ranges, two per SM, whatever the mix of lengths.  A CTA is two teams of
// warps that share the table and nothing else, so that one team computes while the other is between jobs (with one team
// of 16 warps 27 of 92 us went into the jobs' ends).  A team walks its range job by job: its warps take the job's tiles in
// turn, each through a ring of its own (one cp.async.bulk per tile, no synchronisation between warps), and merge their
// (max, sum, accumulator) in shared memory.  A job that lies in one range is finished there; the parts of one that several
// ranges share go to scratch, and the team that arrives last (a counter per job) adds them in range order - the result
// does not depend on timing - un-rotates and writes.  One launch, no combine kernel.  Where a job has many parts their
// weights are computed first, side by side, so that the accumulators stream: as a chain of rescaled sums, six parts a round
// trip, 3 jobs of 2500 tiles spent 23 of 50 us there.  Where cutting the jobs costs more than it levels out, a range is a
// number of whole jobs, or each job is cut into as many parts (launch_kv_attention).  A job's start and end cost a team about
// as much as `pad` tiles, so the flat numbering gives every job that many empty tiles in front: a range with two jobs gets
// fewer tiles than one with a single one.
//
// The next job's first tiles are requested before the merge of the current one, which has shared memory of its own.
#include <algorithm>
#include <climits>
#include <cmath>

#include "tq_attn.cuh"
#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

__constant__ float kC3[8] = {-2.152176f, -1.344318f, -0.756130f, -0.245379f, 0.245379f, 0.756130f, 1.344318f, 2.152176f};

constexpr uint32_t kTabBytes = 256 * 128;                       // the pair table, at the start of shared memory
constexpr float kNone = -1e30f;
constexpr int kGroup = kAttnJobHeads;
constexpr int kTeamWarps = 8;
constexpr int kMaxRanges = 320;                                 // two per SM
constexpr int kFewParts = 6;                                    // parts of a job that its last team adds in one round trip
constexpr unsigned long long kWaitLimitNs = 200ull * 1000 * 1000;

template <int D>
struct AttnCfg {
    static constexpr int kWarps = D == 256 ? 8 : 16;            // 256 dims: 64 accumulator registers, and one team
    static constexpr int kThreads = 32 * kWarps;
    static constexpr int kPer = D == 256 ? 1 : 2;               // tiles of a stage: one wait and one refill per two tiles, where they fit
    static constexpr int kStages = 2;
    static constexpr int kStageBytes = kPer * KvBlock<D>::kBytes;
    static constexpr int kRing = kStages * kStageBytes;         // bytes of a warp's ring
    static constexpr int kAccRegs = D / 4;                      // accumulators of a thread
    static constexpr int kAccStride = D + 4;                    // floats per head of a published accumulator
    static constexpr int kTeams = D == 256 ? 1 : 2, kTeam = kWarps / kTeams;   // teams, warps of a team
    static constexpr int kHalf = kTeam / 2;                     // the upper half of a team hands over to the lower one
    static constexpr int kPubBytes = 32 * (kAccRegs + 4) * 4;   // registers of a warp, or [8 heads][kAccStride]
    static constexpr int kQStride = D + 8;                      // halves per rotated query
    // Heads of other sizes than 128 are multiplied as fp32 numbers would be: centroids, rotated queries and weights as two fp16
    // numbers each, 22 bits (the centroids' second halves in a table of their own behind the first), and three products.  128
    // dims have always been multiplied in fp16, with centroids scaled so that fp16 holds them to 1.4e-5.
    static constexpr bool kSplit = D != 128;
    static constexpr uint32_t kTables = kSplit ? 2 * kTabBytes : kTabBytes;
    static constexpr uint32_t kOffQ = kTables + kWarps * kRing;                         // rotated queries
    static constexpr uint32_t kOffQs = kOffQ + kGroup * kQStride * 2;                   // ... with the residual's signs
    static constexpr uint32_t kOffQl = kOffQs + kGroup * kQStride * 2;                  // what fp16 left of both, in fragment order
    static constexpr uint32_t kOffQsl = kOffQl + (kSplit ? kGroup * kQStride * 2 : 0);
    static constexpr uint32_t kOffPub = kOffQsl + (kSplit ? kGroup * kQStride * 2 : 0);
    static constexpr uint32_t kOffOut = kOffPub + kHalf * kPubBytes;
    static constexpr uint32_t kOffMl = kOffOut + kGroup * kAccStride * 4;               // [2][kHalf][8], then flags, the job and the queries' scales
    static constexpr uint32_t kTeamBytes = kOffMl + 2 * kHalf * kGroup * 4 + 80 + kGroup * 4 - kOffQ;   // of one team, from kOffQ on
    static constexpr uint32_t kEnd = kOffQ + kTeams * kTeamBytes;
    static constexpr int kPartFloats = kGroup * D + 2 * kGroup;                // a job part in scratch: accumulators, then (max, sum)
    static_assert(kPubBytes >= kGroup * kAccStride * 4, "a warp's accumulator in head order fits its place");
    static constexpr int kMaxParts = kHalf * kPubBytes / (kGroup * 4);         // whose weights the publishing places hold
    static_assert(kMaxParts >= kMaxRanges || D < 64, "parts of a job: up to all ranges");
    static_assert(kGroup * kAccStride >= 2 * kTeam * kGroup, "the output's place holds two values per warp and head");
    static_assert(kOffQ % 16 == 0 && kOffPub % 16 == 0 && kOffOut % 16 == 0, "alignment");
    static_assert(kEnd + 1024u <= 227u * 1024u, "shared memory of an SM");
};

struct AttnArgs {
    AttnSeqs seqs;
    const void* q;
    __half* out;
    float* lse;
    float* part;               // [range][2][kPartFloats]
    unsigned int* counters;    // [job]
    unsigned int* status;
    int q_is_f16, n_seqs, q_heads, kv_heads, gchunks, units, ranges, pad, whole_jobs, parts;
    uint32_t k_seed, v_seed, qjl_seed;
    float inv_sqrt, inv_scale, score_scale, qscale;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void add4(float (&c)[4], const float (&t)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += t[i];
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
// The larger one, NaN where either is.
__device__ __forceinline__ float max_or_nan(float x, float y) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(x), "f"(y));
    return m;
}
__device__ __forceinline__ unsigned long long timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}
// False when the phase did not complete in time.
__device__ __noinline__ bool bar_wait_long(uint32_t bar, uint32_t parity) {
    const unsigned long long t0 = timer_ns();
    for (uint32_t spin = 1; !bar_try(bar, parity); ++spin)
        if ((spin & 63) == 0 && timer_ns() - t0 > kWaitLimitNs) return false;
    return true;
}
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    return bar_try(bar, parity) || bar_try(bar, parity) || bar_wait_long(bar, parity);
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}
// Address of the table word of byte BYTE of `word`: byte * 128 + the address of this lane's copy of entry 0, one
// dot-product instruction.  (A byte permutation would do with entries of 256 bytes, but the logic pipe it runs on also
// carries the sign and mask operations and issues every other cycle.)
template <int BYTE>
__device__ __forceinline__ uint32_t pair_addr(uint32_t word, uint32_t lane_base) {
    return __dp4a(word, 128u << (8 * BYTE), lane_base);
}
__device__ __forceinline__ uint32_t table_load(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// The second half of the same entry.
__device__ __forceinline__ uint32_t table_load_low(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1 + 32768];" : "=r"(v) : "r"(addr));
    return v;
}
static_assert(kTabBytes == 32768u, "table_load_low's immediate");
// W consecutive words.
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

template <int D, bool QJL, bool PARTS>
__global__ void __launch_bounds__(AttnCfg<D>::kThreads, 1) attn_kernel(const __grid_constant__ AttnArgs a) {
    using C = AttnCfg<D>;
    using B = KvBlock<D>;
    constexpr int kSteps = D / 16;   // k steps of a score product, m tiles of the value product
    constexpr int W = D / 32;        // nibble words of a token that a thread takes
    constexpr bool kSplit = C::kSplit;
    extern __shared__ __align__(16) unsigned char attn_smem[];
    __shared__ __align__(8) unsigned long long s_bars[C::kWarps * C::kStages];

    const int lane = threadIdx.x & 31, cta_warp = threadIdx.x >> 5;
    const int team = cta_warp / C::kTeam, warp = cta_warp - team * C::kTeam, tid = threadIdx.x - team * (C::kTeam * 32);   // in the team
    const int g = lane >> 2, q = lane & 3;
    auto team_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(C::kTeam * 32) : "memory"); };
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(attn_smem));
    const uint32_t ring = base + C::kTables + cta_warp * C::kRing;
    const uint32_t bars = static_cast<uint32_t>(__cvta_generic_to_shared(&s_bars[cta_warp * C::kStages]));
    unsigned char* const mine = attn_smem + C::kOffQ + team * C::kTeamBytes;   // this team's shared memory
    __half* const s_q = reinterpret_cast<__half*>(mine);
    __half* const s_qs = reinterpret_cast<__half*>(mine + (C::kOffQs - C::kOffQ));
    [[maybe_unused]] __half* const s_ql = reinterpret_cast<__half*>(mine + (C::kOffQl - C::kOffQ));
    [[maybe_unused]] __half* const s_qsl = reinterpret_cast<__half*>(mine + (C::kOffQsl - C::kOffQ));
    unsigned char* const s_pub = mine + (C::kOffPub - C::kOffQ);
    float* const s_out = reinterpret_cast<float*>(mine + (C::kOffOut - C::kOffQ));
    float* const s_m = reinterpret_cast<float*>(mine + (C::kOffMl - C::kOffQ));
    float* const s_l = s_m + C::kHalf * kGroup;
    volatile unsigned int* const s_flag = reinterpret_cast<volatile unsigned int*>(s_l + C::kHalf * kGroup);   // [0] last, [1] stop
    // The job's fields that only its end needs, kept out of the tile loop's registers: two of them, the next job is located
    // before the last one's end.
    volatile int* const s_job = reinterpret_cast<volatile int*>(s_l + C::kHalf * kGroup) + 4;
    float* const s_scale = reinterpret_cast<float*>(const_cast<int*>(s_job)) + 16;   // per query head: a product's weight in the score
    int job_slot = 0;

    if (lane == 0) {
        for (int s = 0; s < C::kStages; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8u * s), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The table does not depend on the kernels before this one.  (Bits 6 and 7 of a byte are not part of its codes.)
    for (int i = threadIdx.x; i < 256 * 8; i += C::kThreads) {
        const int e = i >> 3;
        const float c0 = kAttnCentroidScale * kC3[e & 7], c1 = kAttnCentroidScale * kC3[(e >> 3) & 7];
        const uint32_t v = pack_half2(c0, c1);
        *reinterpret_cast<uint4*>(attn_smem + i * 16) = make_uint4(v, v, v, v);   // 4 copies per store
        if constexpr (kSplit) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
            const uint32_t lo = pack_half2(c0 - f.x, c1 - f.y);
            *reinterpret_cast<uint4*>(attn_smem + kTabBytes + i * 16) = make_uint4(lo, lo, lo, lo);
        }
    }
    if (tid == 0) s_flag[1] = 0u;
    __syncthreads();

    const uint32_t lane_base = base + static_cast<uint32_t>(lane * 4);
    // the first teams of all CTAs come first: few ranges spread over the SMs
    const int range = static_cast<int>(blockIdx.x + gridDim.x * static_cast<unsigned>(team));
    if (range >= a.ranges) {
        pdl_wait_release();
        return;
    }
    const int jobs_per_seq = a.kv_heads * a.gchunks, G = a.q_heads / a.kv_heads;
    // where range r starts: an equal share of the flat tiles, or of the jobs, or (PARTS) of a job's tiles
    auto range_start = [&](int r) {
        if (!PARTS && !a.whole_jobs) return static_cast<int>(static_cast<long>(a.units) * r / a.ranges);
        const int job = PARTS ? r / a.parts : static_cast<int>(static_cast<long>(a.n_seqs) * jobs_per_seq * r / a.ranges);
        if (job >= a.n_seqs * jobs_per_seq) return a.units;
        const int seq = job / jobs_per_seq;
        const AttnSeq S = attn_seq(a.seqs, seq);
        const int start = (S.tile0 + seq * a.pad) * jobs_per_seq + (job - seq * jobs_per_seq) * ((S.end + kKvTile - 1) / kKvTile - S.start / kKvTile + a.pad);
        if constexpr (PARTS) return start + static_cast<int>(static_cast<long>((S.end + kKvTile - 1) / kKvTile - S.start / kKvTile) * (r - job * a.parts) / a.parts);
        else return start;
    };
    if (a.seqs.table != nullptr) pdl_wait_release();   // the table may have been uploaded just before
    int u = range_start(range);
    const int u_end = range_start(range + 1);
    const size_t tile_stride = static_cast<size_t>(a.kv_heads) * B::kBytes;
    uint32_t phase = 0;      // parity of the completion waited for next; flips every kStages = 2 stages
    int stage = 0;
    bool ok = true;

    // The job of flat tile u, and this range's tiles of it.
    struct Segment {
        const unsigned char* src;   // block of the segment's first tile
        int start, end, first_token;
        int tiles, tile0, n_tiles;  // of the job; the segment's first; its count
        int q_row0, ng, job, mine;
        int next_u;
    };
    auto locate = [&](int u) {
        int lo = 0, hi = a.n_seqs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((attn_seq(a.seqs, mid).tile0 + mid * a.pad) * jobs_per_seq <= u) lo = mid;
            else hi = mid - 1;
        }
        const AttnSeq S = attn_seq(a.seqs, lo);
        Segment g;
        const int first_tile = S.start / kKvTile;
        g.tiles = (S.end + kKvTile - 1) / kKvTile - first_tile;
        const int in_seq = u - (S.tile0 + lo * a.pad) * jobs_per_seq, hg = in_seq / (g.tiles + a.pad);
        const int at = in_seq - hg * (g.tiles + a.pad);          // position in the job, its empty tiles included
        const int skip = max(a.pad - at, 0);
        g.tile0 = at + skip - a.pad;
        g.n_tiles = max(min(u_end - u - skip, g.tiles - g.tile0), 0);   // 0: the range ends in the job's empty tiles
        g.next_u = u + skip + g.n_tiles;
        const int kvh = hg / a.gchunks, g0 = (hg - kvh * a.gchunks) * kGroup;
        g.ng = min(kGroup, G - g0);
        g.q_row0 = lo * a.q_heads + kvh * G + g0;
        g.job = lo * jobs_per_seq + hg;
        g.start = S.start;
        g.end = S.end;
        g.first_token = (first_tile + g.tile0) * kKvTile;
        g.src = S.base + static_cast<size_t>(first_tile + g.tile0) * tile_stride + static_cast<size_t>(kvh) * B::kBytes;
        if (tid == 0) {
            volatile int* const j = s_job + 7 * job_slot;
            j[0] = g.tiles; j[1] = g.tile0; j[2] = g.n_tiles; j[3] = g.q_row0; j[4] = g.ng; j[5] = g.job; j[6] = g.next_u;
        }
        g.mine = g.n_tiles > warp ? (g.n_tiles - warp + C::kTeam - 1) / C::kTeam : 0;   // tiles warp, warp + kTeam, ...
        return g;
    };
    // One stage: this warp's next kPer tiles, or its last one.  (a lane)
    auto request = [&](uint32_t dst, const unsigned char* src, int left, uint32_t bar) {
        const bool two = C::kPer == 2 && left > 1;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(two ? 2 * B::kBytes : B::kBytes) : "memory");
        bulk_copy(dst, src, B::kBytes, bar);
        if (two) bulk_copy(dst + B::kBytes, src + C::kTeam * tile_stride, B::kBytes, bar);
    };
    // Before a place in the ring is filled again: every lane's reads of it have ended.  (A tile's value words are needed only
    // beside the next tile's scores, and nothing else keeps their loads in front of the copy, which is of another proxy.
    // The fence costs 2 of 92 us at 16 x 32768 tokens.)
    auto end_reads = [] {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
    };
    auto request_first = [&](const Segment& g) {
        for (int i = 0; i < C::kStages && C::kPer * i < g.mine; ++i) {
            const int s = stage ^ i;
            request(ring + s * C::kStageBytes, g.src + static_cast<size_t>(warp + C::kPer * i * C::kTeam) * tile_stride, g.mine - C::kPer * i, bars + 8u * s);
        }
    };

    Segment seg = locate(u);
    if (a.seqs.table == nullptr) pdl_wait_release();
    if (lane == 0) request_first(seg);
    for (;;) {
        // ---- rotated queries: fp16-round, sign, butterfly, 1 / sqrt(D) (a warp per head), times the power of two that takes
        // the largest to 2^13 .. 2^14, which the score's scale takes back: small and large queries keep all bits of fp16 ----
        for (int h = warp; h < kGroup; h += C::kTeam) {
            constexpr int E = D / 32;
            float v[E], most = 0.f;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int d = lane * E + j;
                float t = 0.f;
                if (h < seg.ng) {
                    const size_t qi = static_cast<size_t>(seg.q_row0 + h) * D + d;
                    t = a.q_is_f16 ? __half2float(static_cast<const __half*>(a.q)[qi])
                                   : __half2float(__float2half_rn(static_cast<const float*>(a.q)[qi]));
                }
                v[j] = t * sign_value(a.k_seed, static_cast<uint32_t>(d));
            }
            warp_fwht<E>(v, lane);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                v[j] *= a.inv_sqrt;
                most = fmaxf(most, fabsf(v[j]));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
            const uint32_t e = __float_as_uint(most) >> 23;
            const bool scaled = e >= 64 && e < 255;   // not zero, not infinite
            const float up = scaled ? __uint_as_float((267 - e) << 23) : 1.f, down = scaled ? __uint_as_float((e - 13) << 23) : 1.f;
            if (lane == 0) s_scale[h] = down * a.score_scale;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int d = lane * E + j;
                const float r = v[j] * up;
                s_q[h * C::kQStride + d] = __float2half_rn(r);
                if constexpr (kSplit) s_ql[h * C::kQStride + d] = __float2half_rn(r - __half2float(__float2half_rn(r)));
                if constexpr (QJL) {
                    const float rs = r * (qjl_sign_is_positive(a.qjl_seed, static_cast<uint32_t>(d)) ? a.qscale : -a.qscale);
                    s_qs[h * C::kQStride + d] = __float2half_rn(rs);
                    // dims 8 w + r and 8 w + r + 4 of a quarter side by side (sign pair 4 w + r)
                    if constexpr (kSplit) s_qsl[h * C::kQStride + (d & ~7) + 2 * (d & 3) + ((d >> 2) & 1)] = __float2half_rn(rs - __half2float(__float2half_rn(rs)));
                }
            }
        }
        team_sync();
        // B fragments of head g.  Pair p of thread q: dims (D/4) q + 2 p and the next.  Sign pair 4 w + r: dims 8 w + r
        // and 8 w + r + 4 of the quarter.
        uint32_t bq[2 * kSteps], bs[QJL ? 2 * kSteps : 1];
        float c2_init[2] = {0.f, 0.f};
        const float scale0 = s_scale[2 * q], scale1 = s_scale[2 * q + 1];   // of the heads of an accumulator fragment
        {
            const __half* const sq = s_q + g * C::kQStride + (D / 4) * q;
#pragma unroll
            for (int p = 0; p < 2 * kSteps; ++p) bq[p] = *reinterpret_cast<const uint32_t*>(sq + 2 * p);
            if constexpr (QJL) {
                // Pairs 0 and 2 meet {0, 2} instead of {-1, 1} (one logic op less per pair, see below): the sum of their
                // dims over the whole head is taken off the product up front.
                const __half* const ss = s_qs + g * C::kQStride + (D / 4) * q;
                float even = 0.f;
#pragma unroll
                for (int p = 0; p < 2 * kSteps; ++p) {
                    const int d0 = 8 * (p / 4) + p % 4;
                    bs[p] = static_cast<uint32_t>(__half_as_ushort(ss[d0])) | (static_cast<uint32_t>(__half_as_ushort(ss[d0 + 4])) << 16);
                    if ((p & 1) == 0) even += __half2float(ss[d0]) + __half2float(ss[d0 + 4]);
                    if constexpr (kSplit)
                        if ((p & 1) == 0) even += __half2float(s_qsl[g * C::kQStride + (D / 4) * q + 2 * p]) + __half2float(s_qsl[g * C::kQStride + (D / 4) * q + 2 * p + 1]);
                }
                even += __shfl_xor_sync(0xffffffffu, even, 1);
                even += __shfl_xor_sync(0xffffffffu, even, 2);
                // an accumulator fragment holds heads 2q and 2q + 1
                c2_init[0] = -__shfl_sync(0xffffffffu, even, 8 * q);
                c2_init[1] = -__shfl_sync(0xffffffffu, even, 8 * q + 4);
            }
        }

        // Reference of heads 2q, 2q + 1 in units of log2, kNone before the first tile (finite: scores are taken relative to it);
        // sum of 2^(score - reference); sum of the values with those weights.
        float m_run[2] = {kNone, kNone}, l_run[2] = {0.f, 0.f};
        float acc[kSteps][4];
#pragma unroll
        for (int mt = 0; mt < kSteps; ++mt)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[mt][k] = 0.f;

        // The values of a tile are multiplied one iteration late, beside the next tile's scores: the two are independent, and
        // together they cover each other's shared-memory and tensor latencies.
        [[maybe_unused]] uint32_t pl0 = 0u, pl1 = 0u;   // what fp16 left of P^T
        uint32_t xa[W], xb[W], pb0 = 0u, pb1 = 0u;   // value words (token pairs q and q + 4, dim group g) and P^T of the last tile
#pragma unroll
        for (int w = 0; w < W; ++w) xa[w] = xb[w] = 0u;
        // rows g and g + 8 of m tile 2 w + h are dims 4 w + 2 h and the next of group g
        auto multiply_values = [&] {
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const uint32_t A = D == 128 && w == 3 ? kv_value_spare(xa[0], xa[1 % W], xa[2 % W]) : xa[w];
                const uint32_t Bw = D == 128 && w == 3 ? kv_value_spare(xb[0], xb[1 % W], xb[2 % W]) : xb[w];
                const uint32_t a0 = pair_addr<0>(A, lane_base), a1 = pair_addr<1>(A, lane_base), a2 = pair_addr<0>(Bw, lane_base), a3 = pair_addr<1>(Bw, lane_base);
                const uint32_t a4 = pair_addr<2>(A, lane_base), a5 = pair_addr<3>(A, lane_base), a6 = pair_addr<2>(Bw, lane_base), a7 = pair_addr<3>(Bw, lane_base);
                const uint32_t v0 = table_load(a0), v1 = table_load(a1), v2 = table_load(a2), v3 = table_load(a3);
                const uint32_t v4 = table_load(a4), v5 = table_load(a5), v6 = table_load(a6), v7 = table_load(a7);
                mma_f16(acc[2 * w], v0, v1, v2, v3, pb0, pb1);
                mma_f16(acc[2 * w + 1], v4, v5, v6, v7, pb0, pb1);
                if constexpr (kSplit) {
                    mma_f16(acc[2 * w], v0, v1, v2, v3, pl0, pl1);
                    mma_f16(acc[2 * w + 1], v4, v5, v6, v7, pl0, pl1);
                    mma_f16(acc[2 * w], table_load_low(a0), table_load_low(a1), table_load_low(a2), table_load_low(a3), pb0, pb1);
                    mma_f16(acc[2 * w + 1], table_load_low(a4), table_load_low(a5), table_load_low(a6), table_load_low(a7), pb0, pb1);
                }
            }
        };
        // This lane's fragments of the queries' remainders: words 4 w .. of quarter q, head g.
        [[maybe_unused]] const uint32_t frag_ql = static_cast<uint32_t>(__cvta_generic_to_shared(s_ql)) + (g * C::kQStride + (D / 4) * q) * 2;
        [[maybe_unused]] const uint32_t frag_qsl = static_cast<uint32_t>(__cvta_generic_to_shared(s_qsl)) + (g * C::kQStride + (D / 4) * q) * 2;
        // One tile: its block in shared memory, its first token.
        auto take_tile = [&](uint32_t blk, int token) {
            // ---- scores ----
            float c1[4] = {0.f, 0.f, 0.f, 0.f}, c1b[4] = {0.f, 0.f, 0.f, 0.f};
            float c2[4] = {c2_init[0], c2_init[1], c2_init[0], c2_init[1]}, c2b[4] = {0.f, 0.f, 0.f, 0.f};
            {
                uint32_t ka[W], kb[W];
                load_words<W>(ka, blk + g * (D / 2) + q * (D / 8));
                load_words<W>(kb, blk + (g + 8) * (D / 2) + q * (D / 8));
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const uint32_t a0 = pair_addr<0>(ka[w], lane_base), a1 = pair_addr<0>(kb[w], lane_base), a2 = pair_addr<1>(ka[w], lane_base), a3 = pair_addr<1>(kb[w], lane_base);
                    const uint32_t a4 = pair_addr<2>(ka[w], lane_base), a5 = pair_addr<2>(kb[w], lane_base), a6 = pair_addr<3>(ka[w], lane_base), a7 = pair_addr<3>(kb[w], lane_base);
                    const uint32_t k0 = table_load(a0), k1 = table_load(a1), k2 = table_load(a2), k3 = table_load(a3);
                    const uint32_t k4 = table_load(a4), k5 = table_load(a5), k6 = table_load(a6), k7 = table_load(a7);
                    if constexpr (kSplit) {
                        // the small products first, sums of 16 dims added up in fp32: the tensor cores' accumulation rounds toward
                        // zero, which as one chain left 1e-6 of a score
                        float t[4] = {0.f, 0.f, 0.f, 0.f}, tb[4] = {0.f, 0.f, 0.f, 0.f};
                        uint32_t lo[4];
                        load_words<4>(lo, frag_ql + 16u * w);
                        mma_f16(t, table_load_low(a0), table_load_low(a1), table_load_low(a2), table_load_low(a3), bq[4 * w], bq[4 * w + 1]);
                        mma_f16(tb, table_load_low(a4), table_load_low(a5), table_load_low(a6), table_load_low(a7), bq[4 * w + 2], bq[4 * w + 3]);
                        mma_f16(t, k0, k1, k2, k3, lo[0], lo[1]);
                        mma_f16(tb, k4, k5, k6, k7, lo[2], lo[3]);
                        mma_f16(t, k0, k1, k2, k3, bq[4 * w], bq[4 * w + 1]);
                        mma_f16(tb, k4, k5, k6, k7, bq[4 * w + 2], bq[4 * w + 3]);
                        add4(c1, t);
                        add4(c1b, tb);
                    } else {
                        mma_f16(c1, k0, k1, k2, k3, bq[4 * w], bq[4 * w + 1]);
                        mma_f16(c1b, k4, k5, k6, k7, bq[4 * w + 2], bq[4 * w + 3]);
                    }
                }
                if constexpr (QJL) {
                    // Bits 14 and 30 (dims 2, 6 of a word) as they stand are fp16 {0, 2}; bits 15 and 31 (dims 3, 7) over the
                    // pattern of (-1, -1) are {-1, 1}; the word shifted by a byte gives dims 0, 4 and 1, 5 the same way.
                    auto two = [](uint32_t w) { return w & 0x40004000u; };
                    auto one = [](uint32_t w) { return (w & 0x80008000u) ^ 0xBC00BC00u; };
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        const uint32_t la = ka[w] << 8, lb = kb[w] << 8;
                        const uint32_t s0 = two(la), s1 = two(lb), s2 = one(la), s3 = one(lb);
                        const uint32_t s4 = two(ka[w]), s5 = two(kb[w]), s6 = one(ka[w]), s7 = one(kb[w]);
                        if constexpr (kSplit) {
                            float t[4] = {0.f, 0.f, 0.f, 0.f}, tb[4] = {0.f, 0.f, 0.f, 0.f};
                            uint32_t lo[4];
                            load_words<4>(lo, frag_qsl + 16u * w);
                            mma_f16(t, s0, s1, s2, s3, lo[0], lo[1]);
                            mma_f16(tb, s4, s5, s6, s7, lo[2], lo[3]);
                            mma_f16(t, s0, s1, s2, s3, bs[4 * w], bs[4 * w + 1]);
                            mma_f16(tb, s4, s5, s6, s7, bs[4 * w + 2], bs[4 * w + 3]);
                            add4(c2, t);
                            add4(c2b, tb);
                        } else {
                            mma_f16(c2, s0, s1, s2, s3, bs[4 * w], bs[4 * w + 1]);
                            mma_f16(c2b, s4, s5, s6, s7, bs[4 * w + 2], bs[4 * w + 3]);
                        }
                    }
                }
            }
            multiply_values();   // of the tile before
            // ---- this tile's norms and value words; then the stage can be refilled ----
            float kna, knb, vna, vnb, qna = 0.f, qnb = 0.f;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(kna), "=f"(vna) : "r"(blk + B::kNormOff + g * 8));
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(knb), "=f"(vnb) : "r"(blk + B::kNormOff + (g + 8) * 8));
            if constexpr (QJL) {
                qna = load_f32(blk + B::kNormOff + 2 * kKvTile * 4 + g * 4);
                qnb = load_f32(blk + B::kNormOff + 2 * kKvTile * 4 + (g + 8) * 4);
            }
            if constexpr (D == 128) {
                uint32_t t[2], o[1];
                load_words<2>(t, blk + B::kValueOff + (q * 8 + g) * 8);
                xa[0] = t[0];
                xa[1] = t[1];
                load_words<2>(t, blk + B::kValueOff + ((q + 4) * 8 + g) * 8);
                xb[0] = t[0];
                xb[1] = t[1];
                load_words<1>(o, blk + B::kValueOff + 512 + (q * 8 + g) * 4);
                xa[2] = o[0];
                load_words<1>(o, blk + B::kValueOff + 512 + ((q + 4) * 8 + g) * 4);
                xb[2] = o[0];
            } else {
                load_words<W>(xa, blk + B::kValueOff + (q * 8 + g) * (D / 8));
                load_words<W>(xb, blk + B::kValueOff + ((q + 4) * 8 + g) * (D / 8));
            }
            // ---- online softmax.  What multiplies the values is w = 2^(score - reference) * value norm in fp16, so the
            // reference follows the largest w, not the largest score: any norm fits, and a weight keeps all its bits down to
            // 2^-27 of the largest.  It is lazy: it moves (and the sums are rescaled) only when some w no longer fits, so the
            // usual tile needs one vote instead of a reduction over the tokens.  Every tile holds a token of [start, end), so
            // the reference is finite from a warp's first tile on.  A norm of next to nothing counts as kLeastNorm (an
            // output below fp16's range), which bounds the sum of 2^(score - reference) too.
            constexpr float kMostWeight = 61440.f, kTopBits = 13.f;   // a new reference takes the largest w to 2^kTopBits
            constexpr float kLeastNorm = 1e-18f, kMostNormBits = 100.f;
            float x0 = c1[0] + c1b[0], x1 = c1[1] + c1b[1], x2 = c1[2] + c1b[2], x3 = c1[3] + c1b[3];
            if constexpr (QJL) {
                x0 = fmaf(qna, c2[0] + c2b[0], x0);
                x1 = fmaf(qna, c2[1] + c2b[1], x1);
                x2 = fmaf(qnb, c2[2] + c2b[2], x2);
                x3 = fmaf(qnb, c2[3] + c2b[3], x3);
            }
            const float ka0 = kna * scale0, ka1 = kna * scale1, kb0 = knb * scale0, kb1 = knb * scale1;
            // scores relative to the reference: (token g: heads 2q, 2q + 1), (token g + 8: the same)
            float s00 = fmaf(x0, ka0, -m_run[0]), s01 = fmaf(x1, ka1, -m_run[1]), s10 = fmaf(x2, kb0, -m_run[0]), s11 = fmaf(x3, kb1, -m_run[1]);
            if (token < seg.start || token + kKvTile > seg.end) {   // tokens outside the range, only in a job's end tiles
                const int ta = token + g, tb = ta + 8;
                if (ta < seg.start || ta >= seg.end) { s00 = s01 = -INFINITY; vna = 0.f; }
                if (tb < seg.start || tb >= seg.end) { s10 = s11 = -INFINITY; vnb = 0.f; }
            }
            vna = max_or_nan(vna, kLeastNorm);
            vnb = max_or_nan(vnb, kLeastNorm);
            float p00 = exp2_approx(s00), p01 = exp2_approx(s01), p10 = exp2_approx(s10), p11 = exp2_approx(s11);
            float w00 = p00 * vna, w01 = p01 * vna, w10 = p10 * vnb, w11 = p11 * vnb;
            if (__any_sync(0xffffffffu, fmaxf(fmaxf(w00, w01), fmaxf(w10, w11)) > kMostWeight)) {
                // absolute again: relative to the first tile's reference (kNone) a score has no bits left
                const float t00 = s00 == -INFINITY ? s00 : x0 * ka0, t01 = s01 == -INFINITY ? s01 : x1 * ka1;
                const float t10 = s10 == -INFINITY ? s10 : x2 * kb0, t11 = s11 == -INFINITY ? s11 : x3 * kb1;
                const float la = fminf(__log2f(vna), kMostNormBits) - kTopBits, lb = fminf(__log2f(vnb), kMostNormBits) - kTopBits;
                float mx0 = fmaxf(t00 + la, t10 + lb), mx1 = fmaxf(t01 + la, t11 + lb);
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
                p00 = exp2_approx(t00 - mn0);
                p01 = exp2_approx(t01 - mn1);
                p10 = exp2_approx(t10 - mn0);
                p11 = exp2_approx(t11 - mn1);
                w00 = p00 * vna;
                w01 = p01 * vna;
                w10 = p10 * vnb;
                w11 = p11 * vnb;
#pragma unroll
                for (int mt = 0; mt < kSteps; ++mt) {
                    acc[mt][0] *= cr0;
                    acc[mt][1] *= cr1;
                    acc[mt][2] *= cr0;
                    acc[mt][3] *= cr1;
                }
            }
            l_run[0] += p00 + p10;
            l_run[1] += p01 + p11;
            // P^T fragment: (tokens 2q, 2q+1 | 2q+8, 2q+9 ; head g) from (token g | g+8 ; heads 2q, 2q+1)
            const uint32_t pa = pack_half2(w00, w01), pb = pack_half2(w10, w11);
            pb0 = movmatrix_trans(pa);
            pb1 = movmatrix_trans(pb);
            if constexpr (kSplit) {
                const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&pa)), fb = __half22float2(*reinterpret_cast<const __half2*>(&pb));
                pl0 = movmatrix_trans(pack_half2(w00 - fa.x, w01 - fa.y));
                pl1 = movmatrix_trans(pack_half2(w10 - fb.x, w11 - fb.y));
            }
        };
        const unsigned char* next_src = seg.src + static_cast<size_t>(warp + C::kPer * C::kStages * C::kTeam) * tile_stride;
        int token = seg.first_token + warp * kKvTile;
        for (int left = seg.mine; left > 0; left -= C::kPer, token += C::kPer * C::kTeam * kKvTile) {
            if (!bar_wait(bars + 8u * stage, phase)) {
                ok = false;
                break;
            }
            const uint32_t blk = ring + stage * C::kStageBytes;
            take_tile(blk, token);
            if (C::kPer == 2 && left > 1) take_tile(blk + B::kBytes, token + C::kTeam * kKvTile);
            if (left > C::kPer * C::kStages) {
                end_reads();
                if (lane == 0) request(blk, next_src, left - C::kPer * C::kStages, bars + 8u * stage);
            }
            next_src += C::kPer * C::kTeam * tile_stride;
            phase ^= static_cast<uint32_t>(stage);
            stage ^= 1;
        }
        multiply_values();   // of the last tile
        struct { int tiles, tile0, n_tiles, q_row0, ng, job; } done;
        {
            const volatile int* const j = s_job + 7 * job_slot;
            done.tiles = j[0]; done.tile0 = j[1]; done.n_tiles = j[2]; done.q_row0 = j[3]; done.ng = j[4]; done.job = j[5];
        }
        u = s_job[7 * job_slot + 6];
        bool more = u < u_end;
        job_slot ^= 1;
        if (more) {
            seg = locate(u);
            more = seg.n_tiles > 0;
            end_reads();
            if (lane == 0 && ok) request_first(seg);
        }

        // ---- merge the warps: the upper half hands its registers to the lower half, which publishes in head order ----
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
            l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
        }
        float* const pub = reinterpret_cast<float*>(s_pub + (warp & (C::kHalf - 1)) * C::kPubBytes);
        if (warp >= C::kHalf) {
#pragma unroll
            for (int mt = 0; mt < kSteps; ++mt) *reinterpret_cast<float4*>(pub + (mt * 32 + lane) * 4) = make_float4(acc[mt][0], acc[mt][1], acc[mt][2], acc[mt][3]);
            *reinterpret_cast<float4*>(pub + (kSteps * 32 + lane) * 4) = make_float4(m_run[0], m_run[1], l_run[0], l_run[1]);
        }
        team_sync();
        if (warp < C::kHalf) {
            const float4 ml = *reinterpret_cast<const float4*>(pub + (kSteps * 32 + lane) * 4);
            const float M0 = fmaxf(m_run[0], ml.x), M1 = fmaxf(m_run[1], ml.y);
            // (a warp without tiles has the reference kNone and sums of zero)
            const float f0 = exp2_approx(m_run[0] - M0), f1 = exp2_approx(m_run[1] - M1);
            const float h0 = exp2_approx(ml.x - M0), h1 = exp2_approx(ml.y - M1);
            l_run[0] = fmaf(l_run[0], f0, ml.z * h0);
            l_run[1] = fmaf(l_run[1], f1, ml.w * h1);
#pragma unroll
            for (int mt = 0; mt < kSteps; ++mt) {
                const float4 o = *reinterpret_cast<const float4*>(pub + (mt * 32 + lane) * 4);
                acc[mt][0] = fmaf(acc[mt][0], f0, o.x * h0);
                acc[mt][1] = fmaf(acc[mt][1], f1, o.y * h1);
                acc[mt][2] = fmaf(acc[mt][2], f0, o.z * h0);
                acc[mt][3] = fmaf(acc[mt][3], f1, o.w * h1);
            }
            __syncwarp();   // the place is this warp's own from here on
            if (g == 0) {
                s_m[warp * kGroup + 2 * q] = M0;
                s_m[warp * kGroup + 2 * q + 1] = M1;
                s_l[warp * kGroup + 2 * q] = l_run[0];
                s_l[warp * kGroup + 2 * q + 1] = l_run[1];
            }
#pragma unroll
            for (int mt = 0; mt < kSteps; ++mt) {
                const int d = (D / 8) * g + 2 * mt;   // rows g and g + 8: dims d and d + 1; columns: heads 2q and 2q + 1
                *reinterpret_cast<float2*>(pub + (2 * q) * C::kAccStride + d) = make_float2(acc[mt][0], acc[mt][2]);
                *reinterpret_cast<float2*>(pub + (2 * q + 1) * C::kAccStride + d) = make_float2(acc[mt][1], acc[mt][3]);
            }
        }
        team_sync();
        const bool whole = done.n_tiles == done.tiles;
        // which ranges share the job: the range of flat tile x is ((x + 1) ranges - 1) / units
        const int job_u0 = u - done.n_tiles - done.tile0;   // the job's first tile
        const int c_first = whole ? range : PARTS ? done.job * a.parts : static_cast<int>((static_cast<long>(job_u0 + 1) * a.ranges - 1) / a.units);
        const int c_last = whole ? range : PARTS ? c_first + a.parts - 1 : static_cast<int>((static_cast<long>(job_u0 + done.tiles) * a.ranges - 1) / a.units);
        float* const my_part = a.part + static_cast<size_t>(2 * range + (done.tile0 == 0 ? 1 : 0)) * C::kPartFloats;
        auto scale_add = [](float4& x, float f0, const float4& y, float f1) {
            x.x = fmaf(x.x, f0, y.x * f1);
            x.y = fmaf(x.y, f0, y.y * f1);
            x.z = fmaf(x.z, f0, y.z * f1);
            x.w = fmaf(x.w, f0, y.w * f1);
        };
        for (int idx = tid * 4; idx < kGroup * D; idx += C::kTeam * 128) {
            const int h = idx / D, d = idx - h * D;
            float m[C::kHalf], M = kNone;
#pragma unroll
            for (int w = 0; w < C::kHalf; ++w) {
                m[w] = s_m[w * kGroup + h];
                M = fmaxf(M, m[w]);
            }
            float L = 0.f;
            float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < C::kHalf; ++w) {
                const float f = exp2_approx(m[w] - M);
                L = fmaf(s_l[w * kGroup + h], f, L);
                scale_add(A, 1.f, *reinterpret_cast<const float4*>(s_pub + w * C::kPubBytes + (h * C::kAccStride + d) * 4), f);
            }
            *reinterpret_cast<float4*>((whole ? s_out + h * C::kAccStride : my_part + h * D) + d) = A;
            if (d == 0) *reinterpret_cast<float2*>(whole ? s_out + h * C::kAccStride + D : my_part + kGroup * D + 2 * h) = make_float2(M, L);
        }
        bool finish = whole;
        if (!whole) {
            __threadfence();
            team_sync();
            if (tid == 0) {
                const unsigned int prev = atomicAdd(&a.counters[done.job], 1u);
                const bool last = prev == static_cast<unsigned int>(c_last - c_first);
                s_flag[0] = last ? 1u : 0u;
                if (last) a.counters[done.job] = 0u;   // ready for the next launch
            }
            team_sync();
            finish = s_flag[0] != 0u;
            if (finish) {
                __threadfence();
                auto part_of = [&](int c) {
                    // the first range's part of the job starts at its tile 0
                    return a.part + static_cast<size_t>(2 * c + (c == c_first ? 1 : 0)) * C::kPartFloats;
                };
                const int n_parts = c_last - c_first + 1;
                if (n_parts > kFewParts) {
                    // Weights first: thread tid holds (max, sum) of head tid % 8 in parts tid / 8, tid / 8 + 32, ...
                    constexpr int kHeld = (kMaxRanges * kGroup + C::kTeam * 32 - 1) / (C::kTeam * 32), kStep = C::kTeam * 32 / kGroup;
                    const int h0 = tid & (kGroup - 1), p0 = tid / kGroup;
                    float2 held[kHeld];
                    float M = kNone;
#pragma unroll
                    for (int k = 0; k < kHeld; ++k) {
                        const int c = p0 + k * kStep;
                        held[k] = c < n_parts ? __ldcg(reinterpret_cast<const float2*>(part_of(c_first + c) + kGroup * D + 2 * h0)) : make_float2(kNone, 0.f);
                    }
#pragma unroll
                    for (int k = 0; k < kHeld; ++k) M = fmaxf(M, held[k].x);
                    M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 8));
                    M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 16));
                    float* const s_red = s_out;   // [warps][8] maxima, then the same of the sums; read before s_out is written
                    if (lane < kGroup) s_red[warp * kGroup + lane] = M;
                    team_sync();
#pragma unroll
                    for (int w = 0; w < C::kTeam; ++w) M = fmaxf(M, s_red[w * kGroup + h0]);
                    float* const s_w = reinterpret_cast<float*>(s_pub);   // [parts][8]: the publishing places are free
                    float L = 0.f;
#pragma unroll
                    for (int k = 0; k < kHeld; ++k) {
                        const float f = exp2_approx(held[k].x - M);
                        L = fmaf(held[k].y, f, L);
                        if (p0 + k * kStep < n_parts) s_w[(p0 + k * kStep) * kGroup + h0] = f;
                    }
                    L += __shfl_xor_sync(0xffffffffu, L, 8);
                    L += __shfl_xor_sync(0xffffffffu, L, 16);
                    if (lane < kGroup) s_red[(C::kTeam + warp) * kGroup + lane] = L;
                    team_sync();
                    float sum = 0.f;
#pragma unroll
                    for (int w = 0; w < C::kTeam; ++w) sum += s_red[(C::kTeam + w) * kGroup + h0];
                    team_sync();   // the reduction's place is read: s_out may be written
                    if (p0 == 0) *reinterpret_cast<float2*>(s_out + h0 * C::kAccStride + D) = make_float2(M, sum);
                    for (int idx = tid * 4; idx < kGroup * D; idx += C::kTeam * 128) {
                        const int h = idx / D, d = idx - h * D;
                        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
                        for (int c0 = 0; c0 < n_parts; c0 += 8) {
                            float4 pa[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) pa[k] = __ldcg(reinterpret_cast<const float4*>(part_of(c_first + min(c0 + k, n_parts - 1)) + idx));
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (c0 + k < n_parts) scale_add(A, 1.f, pa[k], s_w[(c0 + k) * kGroup + h]);
                        }
                        *reinterpret_cast<float4*>(s_out + h * C::kAccStride + d) = A;
                    }
                } else
                for (int idx = tid * 4; idx < kGroup * D; idx += C::kTeam * 128) {
                    const int h = idx / D, d = idx - h * D;
                    float M = kNone, L = 0.f;
                    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int c0 = c_first; c0 <= c_last; c0 += 6) {   // six parts requested at a time, added in order
                        float2 ml[6];
                        float4 pa[6];
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            const float* const p = part_of(min(c0 + k, c_last));
                            ml[k] = __ldcg(reinterpret_cast<const float2*>(p + kGroup * D + 2 * h));
                            pa[k] = __ldcg(reinterpret_cast<const float4*>(p + idx));
                        }
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            if (c0 + k > c_last) break;
                            const float mn = fmaxf(M, ml[k].x), f0 = exp2_approx(M - mn), f1 = exp2_approx(ml[k].x - mn);
                            L = fmaf(L, f0, ml[k].y * f1);
                            scale_add(A, f0, pa[k], f1);
                            M = mn;
                        }
                    }
                    *reinterpret_cast<float4*>(s_out + h * C::kAccStride + d) = A;
                    if (d == 0) *reinterpret_cast<float2*>(s_out + h * C::kAccStride + D) = make_float2(M, L);
                }
            }
        }
        if (!ok && lane == 0) s_flag[1] = 1u;
        team_sync();   // (also: s_out is written, the publishing places are free)
        const bool stop = s_flag[1] != 0u;
        // ---- un-rotate and write: out = (inv_sqrt * sign_v) o H(inv_scale * acc) / L, a warp per head ----
        for (int h = warp; finish && !stop && h < done.ng; h += C::kTeam) {
            constexpr int E = D / 32;
            const float M = s_out[h * C::kAccStride + D], L = s_out[h * C::kAccStride + D + 1];
            float v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = s_out[h * C::kAccStride + lane * E + j] * a.inv_scale;
            warp_fwht<E>(v, lane);
            const float invL = L > 0.f ? 1.0f / L : 0.f;
            const size_t row = static_cast<size_t>(done.q_row0 + h);
            // log of the softmax denominator: lets a caller merge results over disjoint token ranges
            if (a.lse != nullptr && lane == 0) a.lse[row] = L > 0.f ? M * 0.6931471805599453f + logf(L) : -INFINITY;
#pragma unroll
            for (int j = 0; j < E; ++j)
                a.out[row * D + lane * E + j] = __float2half_rn(v[j] * a.inv_sqrt * sign_value(a.v_seed, static_cast<uint32_t>(lane * E + j)) * invL);
        }
        if (stop || !more) break;
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
    constexpr int kSmem = static_cast<int>(C::kEnd);
    static bool configured[64] = {false};   // the opt-in size is a per-device attribute
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {   // both, so that neither is used for the first time in a capture
        TQ_CUDA(cudaFuncSetAttribute(attn_kernel<D, QJL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        TQ_CUDA(cudaFuncSetAttribute(attn_kernel<D, QJL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    launch_pdl(args.parts != 0 ? attn_kernel<D, QJL, true> : attn_kernel<D, QJL, false>, dim3(static_cast<unsigned>(grid)), dim3(C::kThreads), kSmem, stream,
               args);
}

}  // namespace

long attn_number_tiles(AttnSeq* seqs, int n_seqs, long* longest, long* shortest) {
    long total = 0;
    *longest = 0;
    *shortest = LONG_MAX;
    for (int i = 0; i < n_seqs; ++i) {
        seqs[i].tile0 = static_cast<int>(total);
        const long tiles = (seqs[i].end + kKvTile - 1) / kKvTile - seqs[i].start / kKvTile;
        *longest = std::max(*longest, tiles);
        *shortest = std::min(*shortest, tiles);
        total += tiles;
    }
    return total;
}

size_t attn_scratch_bytes(int dim, int sm_count) { return static_cast<size_t>(2 * sm_count) * 2 * (kGroup * dim + 2 * kGroup) * sizeof(float); }

size_t attn_counters(int n_seqs, int q_heads, int kv_heads) {
    return static_cast<size_t>(n_seqs) * kv_heads * ((q_heads / kv_heads + kGroup - 1) / kGroup);
}

// Or each job is cut into as many parts: a range has one job, so that the parts are as long as each other, end together and are few (an
// equal share's ranges span two jobs each, and it takes all the ranges there are).  The number of parts, 0 where the plan at hand - `ranges` of
// jobs_per_range whole jobs, or equal shares (0) - is as good.  Times of a whole call in ns, fitted to 2000 calls of 1 to 64 sequences of 40 to
// 100 000 tokens, alike and of very different lengths: 5 % off for parts, 9 % for whole jobs, 13 % for shares (more often too low than too high),
// which is why the parts have to be 5 % better than whole jobs, and than shares of 256 dims.  None of those calls is more than 2 % slower for it; chosen
// without that margin, and with costs that left out the call itself, 25 were (64 dims, 4 sequences of up to 550 tokens, 8 / 8 heads 7.8 -> 8.3 us; 32
// dims, 8 of 2400 to 13 000 25.5 -> 29.9).
// Before and with the parts taken, us: 128 dims, 28 / 4 heads, 1 x 1024 tokens 10.5 / 7.9, 1 x 4096 10.2 / 9.5, 1 x 8192 14.4 / 10.9, 1 x 32768 20.6 / 15.6,
// 8 x 1024 10.7 / 9.1, 3494 and 5026 beside each other 17.3 / 10.4; 40 / 8 heads, 1 x 8192 14.8 / 11.6, 8 x 4096 23.7 / 18.8; 8 / 1 heads, 1 x 100000
// 30.7 / 18.6; 64 dims 1 x 16384 15.0 / 12.5, 16 x 4096, 8 / 8 29.4 / 26.1; 32 dims 1 x 16384 11.7 / 9.8; 256 dims 1 x 512 19.9 / 14.6, 4 x 2048 25.2 / 18.6.
// 16 x 32768, whose 64 jobs would be four parts each of the 4.6 that the SMs have room for, 80.3 in equal shares, 85.5 so.  A part has a tile of its job at
// least, so a short sequence beside long ones leaves few parts, one of up to 16 tokens none.
static int attn_parts(int head_dim, long jobs, int ranges, long jobs_per_range, long share, long units, long longest, long shortest, long most, int sm_count) {
    struct {
        int tile, tile_beside, second;   // a tile with one team on the SM, with two; the second team's start
        int part, job;                   // equal shares: a part; the end of a job
        int merge, each;                 // cut at all; for each part of a job that its last one adds (many cost more each)
        int call;                        // what every plan has
    } ns;
    switch (head_dim) {
        case 32: ns = {61, 80, 800, 5800, 4200, 2500, 40, 3900}; break;
        case 64: ns = {98, 141, 1700, 6700, 4200, 2600, 44, 4500}; break;
        case 256: ns = {387, 387, 0, 9400, 7400, 3000, 80, 8300}; break;
        default: ns = {99, 147, 2650, 7200, 5000, 2450, 48, 4800}; break;
    }
    auto tiles_ns = [&](long tiles, long n) { return n > sm_count ? tiles * ns.tile_beside + ns.second : tiles * ns.tile; };
    const long at_hand = jobs_per_range != 0 ? tiles_ns(jobs_per_range * longest, ranges) + (jobs_per_range - 1) * ns.job
                                             : tiles_ns(share, ranges) + ns.part + ns.each * ranges / jobs + ns.job * share * jobs / units;
    long best = (at_hand + ns.call) * (jobs_per_range != 0 || head_dim == 256 ? 95 : 100) / 100 - ns.call;
    int parts = 0;
    // (powers of two, three times them, and as many as there are SMs or ranges: a call's host time is microseconds)
    const long most_parts = std::min(most / jobs, shortest);
    auto consider = [&](long p) {
        if (p < 2 || p > most_parts) return;
        const long cost = tiles_ns(std::max<long>(kTeamWarps, (longest + p - 1) / p), jobs * p) + ns.merge + (ns.each + p / 4) * p;
        if (cost >= best) return;
        best = cost;
        parts = static_cast<int>(p);
    };
    for (long p = 2; p <= most_parts; p *= 2) {
        consider(p);
        consider(p + p / 2);
    }
    consider(sm_count / jobs);
    consider(most_parts);
    return parts;
}

AttnPlan attn_plan(int head_dim, long jobs, long units, long longest, long shortest, int sm_count) {
    // Two ranges per SM while every range has a tile per warp; fewer for short jobs, whose time is the merge of the parts.
    const int team = kTeamWarps, teams = head_dim == 256 ? 1 : 2;
    const long most = std::min<long>(static_cast<long>(teams) * sm_count, head_dim == 32 ? AttnCfg<32>::kMaxParts : kMaxRanges);
    AttnPlan plan{};
    plan.ranges = static_cast<int>(std::min<long>(most, std::max<long>(1, (units + team - 1) / team)));
    // Or whole jobs per range.  An equal share of the tiles cuts most jobs, and the part of a job costs more than a whole one
    // (publish, fence, count, read back); against that stand the tiles that the longest range has more, and the end of every
    // further job of a range.  Costs in ns by head size, from calls forced both ways (28 / 4 heads unless said, cut against
    // whole, us): 32 dims 1 x 4096 tokens 8.2 / 18.0, 8 x 2000, 32 / 8 heads 10.6 / 11.0, 32 x 1000, 32 / 8 18.3 / 14.6;
    // 64 dims 4 x 4096, 8 / 8 heads 17.2 / 27.6, 8 x 2000, 32 / 8 17.1 / 15.9, 64 x 1000, 8 / 8 35.0 / 30.5;
    // 128 dims 1 x 4096 10.0 / 28.5, 8 x 2000, 32 / 8 19.4 / 16.6, 64 x 1000, 8 / 8 38.6 / 33.2, 10 x 10539, 8 / 2 22.4 / 68.3;
    // 256 dims 16 x 2048, 14 / 2 31.1 / 57.2, 32 x 1000, 32 / 8 67.7 / 64.0, 64 x 1000, 8 / 8 124 / 128.
    struct { int tile, tile_beside, part, job; } ns;   // a tile with one team on the SM, with two; a part; the end of a job
    switch (head_dim) {
        case 32: ns = {66, 143, 4000, 6000}; break;
        case 64: ns = {100, 165, 7000, 6000}; break;
        case 256: ns = {400, 400, 9000, 8000}; break;
        default: ns = {100, 190, 10000, 6000}; break;
    }
    const long jobs_per_range = (jobs + most - 1) / most, job_ranges = (jobs + jobs_per_range - 1) / jobs_per_range;
    auto tile_ns = [&](long ranges) { return static_cast<long>(ranges > sm_count ? ns.tile_beside : ns.tile); };
    const long share = (units + plan.ranges - 1) / plan.ranges;
    plan.whole_jobs = jobs_per_range * longest * tile_ns(job_ranges) + (jobs_per_range - 1) * ns.job <=
                   share * tile_ns(plan.ranges) + ns.part + ns.job * share * jobs / units;
    if (plan.whole_jobs) plan.ranges = static_cast<int>(job_ranges);
    plan.parts = attn_parts(head_dim, jobs, plan.ranges, plan.whole_jobs ? jobs_per_range : 0, share, units, longest, shortest, most, sm_count);
    if (plan.parts != 0) {
        plan.whole_jobs = 0;
        plan.ranges = static_cast<int>(jobs * plan.parts);
    }
    return plan;
}

void launch_kv_attention(const AttnSeqs& seqs, int n_seqs, long tiles, long longest, long shortest, const void* q, bool q_is_f16, int q_heads, int kv_heads, int head_dim,
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
    long units = tiles * kv_heads * a.gchunks;
    TQ_REQUIRE(units > 0 && tiles > 0 && units < (1L << 31), "attention: too many tokens for one call");
    a.k_seed = k_seed;
    a.v_seed = v_seed;
    a.qjl_seed = qjl_seed;
    const double d = head_dim;
    a.inv_sqrt = 1.0f / std::sqrt(static_cast<float>(head_dim));
    a.inv_scale = a.inv_sqrt / kAttnCentroidScale;   // of the value sums, whose table is scaled as well
    // softmax scale 1 / sqrt(D) (src/attention_dispatch.cpp:35) and the rotation's 1 / sqrt(D), in units of log2
    a.score_scale = static_cast<float>(1.4426950408889634 / d / kAttnCentroidScale);
    // of the rotated query: the residual's reconstruction, in units of the scaled centroids
    a.qscale = static_cast<float>(std::sqrt(2.0 / (3.14159265358979323846 * d)) * kAttnCentroidScale);
    const AttnPlan plan = attn_plan(head_dim, static_cast<long>(n_seqs) * kv_heads * a.gchunks, units, longest, shortest, sm_count);
    a.ranges = plan.ranges;
    a.parts = plan.parts;
    a.whole_jobs = plan.whole_jobs;
    // 32: five rounds of the team's warps, about 6 us; less where ranges are short and every job ends in several of them
    a.pad = a.parts != 0 ? 0 : static_cast<int>(std::min<long>(32, units / a.ranges / 8));
    units += static_cast<long>(n_seqs) * kv_heads * a.gchunks * a.pad;
    TQ_REQUIRE(units < (1L << 31), "attention: too many tokens for one call");
    a.units = static_cast<int>(units);
    const int grid = std::min(sm_count, a.ranges);
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
