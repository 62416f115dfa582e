// Compressed KV cache kernels: online encoder, range decoder, conversion to and from the reference's arrays.
// The storage layout is described in tq_attn.cuh.
#include <cmath>

#include "tq_attn.cuh"
#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

// 3-bit N(0,1) Lloyd-Max centroids (src/codebook.cpp:24-27); the lower four are these negated.
constexpr float kMag0 = 0.245379f, kMag1 = 0.756130f, kMag2 = 1.344318f, kMag3 = 2.152176f;

template <typename T>
__device__ __forceinline__ float as_f32(T v);
template <>
__device__ __forceinline__ float as_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float as_f32<__half>(__half v) { return __half2float(v); }

// A vector is handled by four neighbouring lanes, lane q holding dims [q N, (q + 1) N), N = D / 4: the quarter whose
// storage words are its own too, so nothing but two butterfly stages crosses lanes.  Pairs of neighbouring dims.
template <int N>
__device__ __forceinline__ void quad_fwht2(unsigned long long (&v)[N / 2], int q) {
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const float2 t = unpack2(v[i]);
        v[i] = pack2(__fadd_rn(t.x, t.y), __fsub_rn(t.x, t.y));
    }
#pragma unroll
    for (int h = 1; h < N / 2; h <<= 1) {
#pragma unroll
        for (int i = 0; i < N / 2; i += 2 * h) {
#pragma unroll
            for (int j = i; j < i + h; ++j) {
                const unsigned long long a = v[j], b = v[j + h];
                v[j] = add2(a, b);
                v[j + h] = sub2(a, b);
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
        // other + v, or other - v in the upper lane: multiply-adds with +-1 round as they do
        const float side = (q & m) != 0 ? -1.0f : 1.0f;
        const unsigned long long side2 = pack2(side, side);
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
            const float2 t = unpack2(v[j]);
            v[j] = fma2(v[j], side2, pack2(__shfl_xor_sync(0xffffffffu, t.x, m), __shfl_xor_sync(0xffffffffu, t.y, m)));
        }
    }
}

// Sums over a vector of v[j]^2, accumulated left to right in fp32 (src/kv_cache.cpp:84-88, 226-231: the order is part of the
// result).  The 32 vectors of a CTA put their squares into shared memory and one warp adds them up, a lane per vector; a
// vector's quarters are kQuarter floats apart and vectors kPitch, so that neither side's 16-byte accesses meet in a bank.
template <int D>
struct SquareSums {
    static constexpr int kQuarter = (D / 4 + 23) / 32 * 32 + 8, kPitch = 4 * kQuarter + 4;
    static constexpr bool kShared = D <= 256;   // (beyond, the running sum goes through the quad's lanes in turn: 32 vectors take 70 KB)
    __align__(16) float sq[kShared ? 32 * kPitch : 4];
    float sum[32];
};
template <int D>
__device__ __forceinline__ void put_squares(const unsigned long long (&v)[D / 8], SquareSums<D>& s) {
    using S = SquareSums<D>;
    float* const mine = s.sq + (threadIdx.x >> 2) * S::kPitch + (threadIdx.x & 3) * S::kQuarter;
#pragma unroll
    for (int j = 0; j < D / 4; j += 4) {
        const float2 a = unpack2(mul2(v[j / 2], v[j / 2])), b = unpack2(mul2(v[j / 2 + 1], v[j / 2 + 1]));
        *reinterpret_cast<float4*>(mine + j) = make_float4(a.x, a.y, b.x, b.y);
    }
}
template <int D>
__device__ __forceinline__ float add_squares(const SquareSums<D>& s, int vector) {
    using S = SquareSums<D>;
    const float* const row = s.sq + vector * S::kPitch;
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll 8
        for (int j = 0; j < D / 4; j += 4) {
            const float4 t = *reinterpret_cast<const float4*>(row + k * S::kQuarter + j);
            acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t.x), t.y), t.z), t.w);
        }
    return acc;
}
template <int N>
__device__ __forceinline__ float quad_square_sum(const unsigned long long (&v)[N / 2], int lane) {
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float t = acc;
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
            const float2 x = unpack2(mul2(v[j], v[j]));
            t = __fadd_rn(__fadd_rn(t, x.x), x.y);
        }
        acc = __shfl_sync(0xffffffffu, t, (lane & 28) + k);
    }
    return acc;
}

// v with its sign flipped where bit j of the word is clear: v * sign_value, without the multiplication.
__device__ __forceinline__ float flip_unless(float v, uint32_t word, int j) {
    return __uint_as_float(__float_as_uint(v) ^ ((~word << (31 - j)) & 0x80000000u));
}

// The code of a rotated, scaled value x and the residual x - centroid.  The boundaries are the centroids' midpoints: +-t1,
// +-t2, +-t3 and zero, and a code is the number of boundaries below the value.  For x > 0 that is 4 + #{t < |x|}, otherwise
// 3 - #{t <= |x|}; one more unit in the last place on |x| turns the second comparison into the first.
__device__ __forceinline__ uint32_t code_of(float x, float& residual) {
    const uint32_t t1 = __float_as_uint(__fmul_rn(__fadd_rn(kMag0, kMag1), 0.5f));
    const uint32_t t2 = __float_as_uint(__fmul_rn(__fadd_rn(kMag1, kMag2), 0.5f));
    const uint32_t t3 = __float_as_uint(__fmul_rn(__fadd_rn(kMag2, kMag3), 0.5f));
    const bool pos = x > 0.0f;
    const uint32_t a = (__float_as_uint(x) & 0x7fffffffu) + (pos ? 0u : 1u);
    const uint32_t m = (a > t1 ? 1u : 0u) + (a > t2 ? 1u : 0u) + (a > t3 ? 1u : 0u);
    const float mag = a > t3 ? kMag3 : (a > t2 ? kMag2 : (a > t1 ? kMag1 : kMag0));
    residual = __fsub_rn(x, pos ? mag : -mag);
    return pos ? 4u + m : 3u - m;
}

// The code alone: 4 + m, or 7 - (4 + m) = (4 + m) ^ 7 for x <= 0, as in code_of, with a comparison less.
__device__ __forceinline__ uint32_t code_only(float x) {
    const uint32_t t1 = __float_as_uint(__fmul_rn(__fadd_rn(kMag0, kMag1), 0.5f));
    const uint32_t t2 = __float_as_uint(__fmul_rn(__fadd_rn(kMag1, kMag2), 0.5f));
    const uint32_t t3 = __float_as_uint(__fmul_rn(__fadd_rn(kMag2, kMag3), 0.5f));
    const bool pos = x > 0.0f;
    const uint32_t a = (__float_as_uint(x) & 0x7fffffffu) + (pos ? 0u : 1u);
    const bool far = a > t2;
    uint32_t c = far ? 6u : 4u;
    if (a > (far ? t3 : t1)) c += 1u;
    return pos ? c : c ^ 7u;
}

struct KvSegments {
    KvSegment seg[kKvMaxSegments];
};

// Eight 3-bit fields at nibble positions (low or high half of a word) to four bytes.
__device__ __forceinline__ uint32_t nibbles_to_bytes(uint32_t four) {
    four = (four | (four << 8)) & 0x00FF00FFu;
    return (four | (four << 4)) & 0x0F0F0F0Fu;
}

// ---- encoder (src/kv_cache.cpp:63-258) ---------------------------------------------------------------
// Eight lanes take a pair of tokens (2p, 2p + 1) of one head, four lanes each; the first half of the units are the keys',
// the second the values'.  A value byte holds both tokens' codes: the two quads exchange half of their words and each
// writes four of the eight groups.  A pair of which only one token is appended keeps the other one's bits.
// Bit-exact: the sums of squares run left to right, every other operation is element-wise or the shared butterfly.
// Bound: issue slots.  2 x 32768 vectors of 128, fp16: 26 us under the profiler with 2175 instructions for a warp's eight
// vectors (a quarter of them for sums that each lane of a quad repeated, and values had residuals that nothing reads);
// 20 with 1445, pairs of dims in one instruction, signs flipped on the halves, the sums as above and
// residuals for keys alone.
template <int D, typename InT>
__global__ void __launch_bounds__(128, D <= 128 ? 7 : (D == 256 ? 3 : 2)) kv_encode_kernel(const InT* __restrict__ keys, const InT* __restrict__ values, int tokens, int n_segs,
                                                        int heads, uint32_t k_seed, uint32_t v_seed, uint32_t qjl_seed,
                                                        float scale, float inv_sqrt, int aligned,
                                                        const __grid_constant__ KvSegments tab) {
    constexpr int N = D / 4, W = N / 8;
    constexpr int kPer = 16 / static_cast<int>(sizeof(InT));   // elements of a 16-byte access
    using B = KvBlock<D>;
    constexpr int kFlips = N / kPer + 1;                   // 16-byte words of a quarter's signs, and one so that the quarters lie in other banks
    __shared__ __align__(16) uint4 s_flip[2][4 * kFlips];  // rotation signs of keys and values, as the elements' sign bits
    __shared__ uint32_t s_qjl[D / 32];                    // residual signs: bit set = +1
    __shared__ float s_cent[8][32];                       // a copy per lane
    __shared__ SquareSums<D> s_sums;
    __shared__ float* s_norm_at[32];                      // where a vector's residual norm goes
    for (int i = threadIdx.x; i < D; i += 128) {
        const uint32_t bits = __ballot_sync(0xffffffffu, qjl_sign_is_positive(qjl_seed, static_cast<uint32_t>(i)));
        if ((i & 31) == 0) s_qjl[i >> 5] = bits;
    }
    {
        constexpr int kPerWord = 4 / static_cast<int>(sizeof(InT));
        for (int i = threadIdx.x; i < 2 * D / kPerWord; i += 128) {
            const int which = i / (D / kPerWord), d = (i - which * (D / kPerWord)) * kPerWord;
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < kPerWord; ++k)
                if (!sign_is_positive(which ? v_seed : k_seed, static_cast<uint32_t>(d + k))) m |= 0x80000000u >> (16 * (kPerWord - 1 - k));
            const int word = d / kPerWord, quarter = word / (N / kPerWord);
            reinterpret_cast<uint32_t*>(&s_flip[which][quarter * kFlips])[word - quarter * (N / kPerWord)] = m;
        }
        for (int i = threadIdx.x; i < 256; i += 128) {
            const int c = i >> 5, m = c < 4 ? 3 - c : c - 4;
            const float mag = m == 3 ? kMag3 : (m == 2 ? kMag2 : (m == 1 ? kMag1 : kMag0));
            s_cent[c][i & 31] = c < 4 ? -mag : mag;
        }
    }
    __syncthreads();
    pdl_wait_release();
    behind_wait(keys, values);

    const int lane = threadIdx.x & 31, q = lane & 3;
    const bool odd = (lane & 4) != 0;
    const int pairs = tokens / 2 + 1;                       // token pairs that `tokens` tokens can touch
    const int per_tensor = n_segs * pairs * heads;
    const bool keys_here = static_cast<long>(blockIdx.x) * 16 < per_tensor;   // whether the CTA has a key (16 pairs per CTA)
    int unit = static_cast<int>((static_cast<long>(blockIdx.x) * 128 + threadIdx.x) >> 3);
    const bool in_range = unit < 2 * per_tensor;
    unit = in_range ? unit : 2 * per_tensor - 1;
    const bool value = unit >= per_tensor;
    const int u = value ? unit - per_tensor : unit;
    const int sidx = u / (pairs * heads), rest = u - sidx * pairs * heads;
    const int pair = rest / heads, head = rest - pair * heads;
    const int first = tab.seg[sidx].first;
    const int token = ((first >> 1) + pair) * 2 + (odd ? 1 : 0), tok = token - first;   // absolute, and within the call
    const bool live = in_range && tok >= 0 && tok < tokens;
    const int src_tok = tok < 0 ? 0 : (tok < tokens ? tok : tokens - 1);
    const InT* const src = (value ? values : keys) + ((static_cast<size_t>(sidx) * tokens + src_tok) * heads + head) * D + q * N;

    unsigned long long v[N / 2];   // pairs of dims; the signs are flipped here (squares do not see them)
#pragma unroll
    for (int i = 0; i < N / kPer; ++i) {
        uint4 raw;
        if (aligned) {
            raw = reinterpret_cast<const uint4*>(src)[i];
        } else {
            InT* const e = reinterpret_cast<InT*>(&raw);
#pragma unroll
            for (int j = 0; j < kPer; ++j) e[j] = src[i * kPer + j];
        }
        const uint4 m = s_flip[value ? 1 : 0][q * kFlips + i];
        raw = make_uint4(raw.x ^ m.x, raw.y ^ m.y, raw.z ^ m.z, raw.w ^ m.w);
        const InT* const e = reinterpret_cast<const InT*>(&raw);
#pragma unroll
        for (int j = 0; j < kPer; j += 2) v[(i * kPer + j) / 2] = pack2(as_f32<InT>(e[j]), as_f32<InT>(e[j + 1]));
    }
    float norm;
    if constexpr (SquareSums<D>::kShared) {
        put_squares<D>(v, s_sums);
        __syncthreads();
        if (threadIdx.x < 32) s_sums.sum[lane] = add_squares<D>(s_sums, lane);
        __syncthreads();
        norm = __fsqrt_rn(s_sums.sum[threadIdx.x >> 2]);
    } else {
        norm = __fsqrt_rn(quad_square_sum<N>(v, lane));
    }
    const float inv_norm = (norm > 1e-10f) ? __fdiv_rn(1.0f, norm) : 0.0f;
    const unsigned long long inv_norm2 = pack2(inv_norm, inv_norm);
#pragma unroll
    for (int j = 0; j < N / 2; ++j) v[j] = mul2(v[j], inv_norm2);
    quad_fwht2<N>(v, q);
    const unsigned long long inv_sqrt2 = pack2(inv_sqrt, inv_sqrt), scale2 = pack2(scale, scale);
#pragma unroll
    for (int j = 0; j < N / 2; ++j) v[j] = mul2(mul2(v[j], inv_sqrt2), scale2);

    uint32_t words[W];   // codes as nibbles
#pragma unroll
    for (int w = 0; w < W; ++w) words[w] = 0u;
#pragma unroll
    for (int j = 0; j < N / 2; ++j) {
        const float2 x = unpack2(v[j]);
        words[j / 4] |= (code_only(x.x) | (code_only(x.y) << 4)) << (8 * (j & 3));
    }
    uint32_t signs[W];   // a key's residual signs, eight bits of a word's dims
    float rnorm = 0.f;   // the residual's norm; only the keys keep it
    if (keys_here) {
        bool plain = true;   // no residual is zero or not a number
#pragma unroll
        for (int w = 0; w < W; ++w) {
            signs[w] = 0u;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                const int i = 4 * w + j;
                const float2 x = unpack2(v[i]);
                const uint32_t two = words[w] >> (8 * j);
                const float r0 = __fsub_rn(x.x, s_cent[two & 7u][lane]), r1 = __fsub_rn(x.y, s_cent[(two >> 4) & 7u][lane]);
                plain = plain && fabsf(r0) > 0.0f && fabsf(r1) > 0.0f;
                signs[w] = __funnelshift_l(__float_as_uint(r1), signs[w], 1);
                signs[w] = __funnelshift_l(__float_as_uint(r0), signs[w], 1);
                v[i] = pack2(r0, r1);
            }
        }
        // a bit is set where the residual's sign is the dim's: r > 0 or r < 0
        auto dims_signs = [&](int w) { return (s_qjl[(q * N + 8 * w) >> 5] >> ((q * N + 8 * w) & 31)) & 0xffu; };
#pragma unroll
        for (int w = 0; w < W; ++w) signs[w] ^= dims_signs(w);
        if (!plain) {
#pragma unroll
            for (int w = 0; w < W; ++w) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 r = unpack2(v[4 * w + j]);
                    if (!(fabsf(r.x) > 0.0f)) signs[w] &= ~(1u << (2 * j));
                    if (!(fabsf(r.y) > 0.0f)) signs[w] &= ~(2u << (2 * j));
                }
            }
        }
        // The last warp adds these up and stores the norms while the others write the codes.
        if constexpr (SquareSums<D>::kShared) put_squares<D>(v, s_sums);
        else rnorm = __fsqrt_rn(quad_square_sum<N>(v, lane));
    }

    // The half of the words that the other quad writes, for the half of its words that this one writes (values).  A
    // group is N / 2 dims; D = 32 has half a word in it.
    constexpr int GW = W >= 2 ? W / 2 : 1;   // nibble words of a group
    uint32_t own[GW], other[GW];
#pragma unroll
    for (int w = 0; w < GW; ++w) {
        const uint32_t lo = W >= 2 ? words[w] : words[0] & 0xFFFFu, hi = W >= 2 ? words[(GW + w) % W] : words[0] >> 16;
        own[w] = odd ? hi : lo;
        other[w] = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 4);
    }
    const bool other_live = __shfl_xor_sync(0xffffffffu, live ? 1 : 0, 4) != 0;
    const int slot = token & (kKvTile - 1);
    unsigned char* const block = tab.seg[sidx].base + (static_cast<size_t>(token / kKvTile) * heads + head) * B::kBytes;
    if constexpr (SquareSums<D>::kShared) {
        if (keys_here) {
            if (q == 0) s_norm_at[threadIdx.x >> 2] = live && !value ? reinterpret_cast<float*>(block + B::kNormOff) + kv_residual_norm(slot) : nullptr;
            __syncthreads();
            if (threadIdx.x >= 96) {
                float* const at = s_norm_at[lane];
                const float sum = add_squares<D>(s_sums, lane);
                if (at != nullptr) *at = __fsqrt_rn(sum);
            }
        }
    }
    if (!live && !(value && other_live)) return;

    if (value) {
        const bool even_live = odd ? other_live : live, odd_live = odd ? live : other_live;
        const int g = 2 * q + (odd ? 1 : 0);
        uint32_t bytes[2 * GW];   // a byte per dim: the even token's code, the odd one's above it
#pragma unroll
        for (int w = 0; w < GW; ++w) {
            const uint32_t e = (even_live ? (odd ? other[w] : own[w]) : 0u), o = (odd_live ? (odd ? own[w] : other[w]) : 0u);
            bytes[2 * w] = nibbles_to_bytes(e & 0xFFFFu) | (nibbles_to_bytes(o & 0xFFFFu) << 3);
            bytes[2 * w + 1] = nibbles_to_bytes(e >> 16) | (nibbles_to_bytes(o >> 16) << 3);
        }
        auto put = [&](uint32_t* p, uint32_t w, int k) { *p = even_live ? w : (*p & ~kv_odd_bits(D, k)) | (w & kv_odd_bits(D, k)); };
        if constexpr (D == 128) {
            const uint32_t spare = bytes[3];
            put(kv_value01(block, slot >> 1, g), bytes[0] | kv_spare_bits(spare, 0), 0);
            put(kv_value01(block, slot >> 1, g) + 1, bytes[1] | kv_spare_bits(spare, 1), 1);
            put(kv_value2(block, slot >> 1, g), bytes[2] | kv_spare_bits(spare, 2), 2);
        } else {
            uint32_t* const dst = kv_value_row(block, D, slot >> 1, g);
#pragma unroll
            for (int w = 0; w < (W >= 2 ? 2 * GW : 1); ++w) put(dst + w, bytes[w], 0);
        }
    } else {
        uint32_t* const dst = reinterpret_cast<uint32_t*>(block) + slot * (D / 8) + q * W;
#pragma unroll
        for (int w = 0; w < W; ++w)   // a byte: two codes, their two signs
            words[w] = (words[w] & 0x07070707u) | ((words[w] >> 1) & 0x38383838u) | ((signs[w] & 0x03u) << 6) | ((signs[w] & 0x0Cu) << 12) |
                       ((signs[w] & 0x30u) << 18) | ((signs[w] & 0xC0u) << 24);
        if constexpr (W % 4 == 0) {
#pragma unroll
            for (int w = 0; w < W; w += 4) *reinterpret_cast<uint4*>(dst + w) = make_uint4(words[w], words[w + 1], words[w + 2], words[w + 3]);
        } else {
#pragma unroll
            for (int w = 0; w < W; ++w) dst[w] = words[w];
        }
    }
    if (q == 0 && live) {
        float* const norms = reinterpret_cast<float*>(block + B::kNormOff);
        norms[value ? kv_value_norm(slot) : kv_key_norm(slot)] = norm;
        if (!SquareSums<D>::kShared && !value) norms[kv_residual_norm(slot)] = rnorm;
    }
}

// The same for a decode step's few vectors, where latency counts: eight dims per lane, so a warp (D = 128) takes one token
// pair of a head.  The quad kernel's straight-line code for 32 dims per lane is 35 KB, which a kernel that runs once
// fetches from L2 as it goes (8.7 us for 16 sequences of 4 heads); this one's is a quarter of it.  The running sums are one
// lane's work, from shared memory.
template <int D, typename InT>
__global__ void __launch_bounds__(64) kv_encode_few_kernel(const InT* __restrict__ keys, const InT* __restrict__ values, int tokens, int n_segs,
                                                           int heads, uint32_t k_seed, uint32_t v_seed, uint32_t qjl_seed, float scale,
                                                           float inv_sqrt, int aligned, const __grid_constant__ KvSegments tab) {
    constexpr int L = D / 8, kUnits = 64 / (2 * L);   // lanes of a vector, token pairs of a CTA
    static_assert(2 * L <= 32, "both tokens of a pair in one warp");
    using B = KvBlock<D>;
    __shared__ __align__(16) float s_sq[2 * kUnits][D + 4];   // a row per vector, rows four banks apart
    const int tid = threadIdx.x, l = tid & (L - 1);
    const bool odd = (tid & L) != 0;
    const int pairs = tokens / 2 + 1, per_tensor = n_segs * pairs * heads;
    int unit = static_cast<int>(blockIdx.x) * kUnits + tid / (2 * L);
    const bool in_range = unit < 2 * per_tensor;
    unit = in_range ? unit : 2 * per_tensor - 1;
    const bool value = unit >= per_tensor;
    const int u = value ? unit - per_tensor : unit;
    const int sidx = u / (pairs * heads), rest = u - sidx * pairs * heads;
    const int pair = rest / heads, head = rest - pair * heads;
    const int first = tab.seg[sidx].first;
    const int token = ((first >> 1) + pair) * 2 + (odd ? 1 : 0), tok = token - first;   // absolute, and within the call
    const bool live = in_range && tok >= 0 && tok < tokens;
    const int src_tok = tok < 0 ? 0 : (tok < tokens ? tok : tokens - 1);
    const InT* src = (value ? values : keys) + ((static_cast<size_t>(sidx) * tokens + src_tok) * heads + head) * D + l * 8;
    uint32_t flips = 0, qflips = 0;   // bit j: dim j's rotation sign, its residual sign (set = +1)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        flips |= sign_is_positive(value ? v_seed : k_seed, static_cast<uint32_t>(l * 8 + j)) ? 1u << j : 0u;
        qflips |= qjl_sign_is_positive(qjl_seed, static_cast<uint32_t>(l * 8 + j)) ? 1u << j : 0u;
    }
    pdl_wait_release();
    behind_wait(src);

    float v[8];
    if (aligned) {
        constexpr int kPer = 16 / static_cast<int>(sizeof(InT));
#pragma unroll
        for (int i = 0; i < 8 / kPer; ++i) {
            const uint4 raw = reinterpret_cast<const uint4*>(src)[i];
            const InT* e = reinterpret_cast<const InT*>(&raw);
#pragma unroll
            for (int j = 0; j < kPer; ++j) v[i * kPer + j] = as_f32<InT>(e[j]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = as_f32<InT>(src[j]);
    }
    float* const row = s_sq[tid / L];
    const int lead = tid & 31 & ~(L - 1);   // the vector's first lane
    auto square_sum = [&] {   // left to right, as in quad_square_sum
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(row + l * 8 + j) =
                make_float4(__fmul_rn(v[j], v[j]), __fmul_rn(v[j + 1], v[j + 1]), __fmul_rn(v[j + 2], v[j + 2]), __fmul_rn(v[j + 3], v[j + 3]));
        __syncwarp();
        float acc = 0.0f;
        if (l == 0) {
#pragma unroll 4
            for (int j = 0; j < D; j += 8) {
                const float4 a = *reinterpret_cast<const float4*>(row + j), b = *reinterpret_cast<const float4*>(row + j + 4);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, a.x), a.y), a.z), a.w);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, b.x), b.y), b.z), b.w);
            }
        }
        __syncwarp();
        return __shfl_sync(0xffffffffu, acc, lead);
    };
    const float norm = __fsqrt_rn(square_sum());
    const float inv_norm = (norm > 1e-10f) ? __fdiv_rn(1.0f, norm) : 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = flip_unless(__fmul_rn(v[j], inv_norm), flips, j);
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int i = 0; i < 8; i += 2 * h)
#pragma unroll
            for (int j = i; j < i + h; ++j) {
                const float a = v[j], b = v[j + h];
                v[j] = __fadd_rn(a, b);
                v[j + h] = __fsub_rn(a, b);
            }
#pragma unroll 1
    for (int m = 1; m < L; m <<= 1) {
        const bool upper = (l & m) != 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, v[j], m);
            v[j] = upper ? __fsub_rn(other, v[j]) : __fadd_rn(v[j], other);
        }
    }
    // the dims' bytes: keys two codes and their signs each, values one code
    uint32_t kword = 0, bytes[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        float r;
        const uint32_t c = code_of(__fmul_rn(__fmul_rn(v[j], inv_sqrt), scale), r);
        v[j] = r;
        const bool bit = ((qflips >> j) & 1u) ? r > 0.0f : r < 0.0f;
        kword |= ((c << (3 * (j & 1))) | (bit ? 64u << (j & 1) : 0u)) << (8 * (j >> 1));
        bytes[j >> 2] |= c << (8 * (j & 3));
    }
    const float rnorm = __fsqrt_rn(square_sum());
    // the other token's codes beside this one's
    const bool other_live = __shfl_xor_sync(0xffffffffu, live ? 1 : 0, L) != 0;
    const bool even_live = odd ? other_live : live, odd_live = odd ? live : other_live;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, bytes[w], L);
        bytes[w] = (even_live ? (odd ? other : bytes[w]) : 0u) | (odd_live ? (odd ? bytes[w] : other) << 3 : 0u);
    }
    const uint32_t spare = __shfl_xor_sync(0xffffffffu, bytes[1], 1);   // D = 128: lanes 2g hold words 0 and 1, lanes 2g + 1 word 2 and the spare dims
    if (!live && !(value && other_live)) return;

    const int slot = token & (kKvTile - 1);
    unsigned char* const block = tab.seg[sidx].base + (static_cast<size_t>(token / kKvTile) * heads + head) * B::kBytes;
    if (value) {
        auto put = [&](uint32_t* p, uint32_t w, int k) { *p = even_live ? w : (*p & ~kv_odd_bits(D, k)) | (w & kv_odd_bits(D, k)); };
        if constexpr (D == 128) {
            const int g = l >> 1;
            if (l & 1) {
                if (!odd) put(kv_value2(block, slot >> 1, g), bytes[0] | kv_spare_bits(bytes[1], 2), 2);
            } else {
                const int k = odd ? 1 : 0;
                put(kv_value01(block, slot >> 1, g) + k, bytes[k] | kv_spare_bits(spare, k), k);
            }
        } else {
            put(kv_value_row(block, D, slot >> 1, 0) + 2 * l + (odd ? 1 : 0), odd ? bytes[1] : bytes[0], 0);
        }
    } else {
        reinterpret_cast<uint32_t*>(block)[slot * L + l] = kword;
    }
    if (l == 0 && live) {
        float* const norms = reinterpret_cast<float*>(block + B::kNormOff);
        norms[value ? kv_value_norm(slot) : kv_key_norm(slot)] = norm;
        if (!value) norms[kv_residual_norm(slot)] = rnorm;
    }
}

// ---- range decoder (src/kv_cache.cpp:292-365) ----------------------------------------------------------
// Four lanes per vector as in the encoder.  The centroids sit in shared memory once per lane: as a constant array they
// were read one lane at a time (86 us for 65536 tokens of 4 heads).  A warp's eight vectors are contiguous in the result: they
// leave through shared memory, in pieces of 16 bytes whose places within a lane's are turned by the lane and the vector
// (no bank conflicts at 128 dims).  8192 tokens of 4 heads of 128: 6.7 us with a dim per instruction and stores 64 bytes apart,
// 5.4 so; heads of 256 17.4 and 6.6.
template <int D>
__global__ void __launch_bounds__(128) kv_decode_kernel(const unsigned char* __restrict__ base, int start, long n_vec, int heads, int values,
                                                        uint32_t wht_seed, float inv_scale, float inv_sqrt, __half* __restrict__ out) {
    constexpr int N = D / 4, W = N / 8;
    using B = KvBlock<D>;
    constexpr int kPieces = N / 8, kFlips = kPieces + 1;    // 16-byte pieces of a lane's result; of a quarter's signs, and one for the banks' sake
    __shared__ float s_cent[8][32];
    __shared__ __align__(16) uint4 s_flip[4 * kFlips];      // rotation signs, as the halves' sign bits
    __shared__ __align__(16) uint4 s_out[4][32 * kPieces];
    for (int i = threadIdx.x; i < 256; i += 128) {
        const int c = i >> 5, m = c < 4 ? 3 - c : c - 4;
        const float mag = m == 3 ? kMag3 : (m == 2 ? kMag2 : (m == 1 ? kMag1 : kMag0));
        s_cent[c][i & 31] = __fmul_rn(c < 4 ? -mag : mag, inv_scale);
    }
    for (int i = threadIdx.x; i < D / 2; i += 128) {
        const int quarter = i / (N / 2);
        reinterpret_cast<uint32_t*>(&s_flip[quarter * kFlips])[i - quarter * (N / 2)] =
            (sign_is_positive(wht_seed, static_cast<uint32_t>(2 * i)) ? 0u : 0x8000u) | (sign_is_positive(wht_seed, static_cast<uint32_t>(2 * i + 1)) ? 0u : 0x80000000u);
    }
    __syncthreads();
    pdl_wait_release();
    behind_wait(base);
    const int lane = threadIdx.x & 31, q = lane & 3;
    const long quad = (static_cast<long>(blockIdx.x) * 128 + threadIdx.x) >> 2;
    const bool live = quad < n_vec;
    const long vec = live ? quad : n_vec - 1;
    const long tok = vec / heads;
    const int head = static_cast<int>(vec - tok * heads);
    const long token = start + tok;
    const int slot = static_cast<int>(token & (kKvTile - 1));
    unsigned char* const block = const_cast<unsigned char*>(base) + (static_cast<size_t>(token / kKvTile) * heads + head) * B::kBytes;
    float v[N];
    if (values) {
        const int sh = (slot & 1) * 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // this lane's two groups of N / 2 dims
            const int g = 2 * q + h;
            if constexpr (D == 128) {
                const uint2 w01 = *reinterpret_cast<const uint2*>(kv_value01(block, slot >> 1, g));
                const uint32_t w[3] = {w01.x, w01.y, *kv_value2(block, slot >> 1, g)};
#pragma unroll
                for (int j = 0; j < 12; ++j) v[h * 16 + j] = s_cent[(w[j / 4] >> (8 * (j & 3) + sh)) & 7u][lane];
                const uint32_t spare = kv_value_spare(w[0], w[1], w[2]);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[(h * 16 + 12 + j) % N] = s_cent[(spare >> (8 * j + sh)) & 7u][lane];
            } else {
                const uint32_t* const src = kv_value_row(block, D, slot >> 1, g);
#pragma unroll
                for (int j = 0; j < N / 2; ++j) v[h * (N / 2) + j] = s_cent[(src[j / 4] >> (8 * (j & 3) + sh)) & 7u][lane];
            }
        }
    } else {
        const uint32_t* const src = reinterpret_cast<const uint32_t*>(block) + slot * (D / 8) + q * W;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t x = src[w];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[8 * w + j] = s_cent[(x >> (8 * (j / 2) + 3 * (j & 1))) & 7u][lane];
        }
    }
    const float norm = reinterpret_cast<const float*>(block + B::kNormOff)[values ? kv_value_norm(slot) : kv_key_norm(slot)];
    unsigned long long p[N / 2];
#pragma unroll
    for (int j = 0; j < N / 2; ++j) p[j] = pack2(v[2 * j], v[2 * j + 1]);
    quad_fwht2<N>(p, q);
    const unsigned long long inv_sqrt2 = pack2(inv_sqrt, inv_sqrt), norm2 = pack2(norm, norm);
    uint4 h[kPieces];
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 t = unpack2(mul2(mul2(p[4 * c + j], inv_sqrt2), norm2));
            const __half2 r = __floats2half2_rn(t.x, t.y);
            w[j] = *reinterpret_cast<const uint32_t*>(&r);
        }
        const uint4 m = s_flip[q * kFlips + c];
        h[c] = make_uint4(w[0] ^ m.x, w[1] ^ m.y, w[2] ^ m.z, w[3] ^ m.w);
    }
    const int in_warp = lane >> 2;   // which of the warp's vectors
    auto place = [](int vector, int quarter, int piece) { return (vector * 4 + quarter) * kPieces + ((piece + quarter + vector) & (kPieces - 1)); };
    if (reinterpret_cast<uintptr_t>(out) % 16 == 0) {
        uint4* const mine = s_out[threadIdx.x >> 5];
#pragma unroll
        for (int c = 0; c < kPieces; ++c) mine[place(in_warp, q, c)] = h[c];
        __syncwarp();
        const long first = quad - in_warp;
        uint4* const dst = reinterpret_cast<uint4*>(out) + first * (4 * kPieces);
#pragma unroll
        for (int k = 0; k < kPieces; ++k) {
            const int i = 32 * k + lane, vector = i / (4 * kPieces), r = i - vector * (4 * kPieces);
            if (first + vector < n_vec) dst[i] = mine[place(vector, r / kPieces, r & (kPieces - 1))];
        }
    } else if (live) {
        const __half* const e = reinterpret_cast<const __half*>(h);
        __half* const dst = out + static_cast<size_t>(vec) * D + q * N;
#pragma unroll
        for (int j = 0; j < N; ++j) dst[j] = e[j];
    }
}

// ---- the reference's arrays ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t stored_code(const unsigned char* block, int dim, int slot, int d, bool value, uint32_t* sign) {
    unsigned char* const b = const_cast<unsigned char*>(block);
    if (value) {
        const int per = dim / 8, g = d / per, r = d - g * per, odd = slot & 1;
        if (dim == 128) {
            const uint32_t w0 = kv_value01(b, slot >> 1, g)[0], w1 = kv_value01(b, slot >> 1, g)[1], w2 = *kv_value2(b, slot >> 1, g);
            const uint32_t w = r < 4 ? w0 : (r < 8 ? w1 : (r < 12 ? w2 : kv_value_spare(w0, w1, w2)));
            return (w >> (8 * (r & 3) + 3 * odd)) & 7u;
        }
        return (kv_value_row(b, dim, slot >> 1, g)[r >> 2] >> (8 * (r & 3) + 3 * odd)) & 7u;
    }
    const uint32_t byte = block[slot * (dim / 2) + (d >> 1)];
    if (sign) *sign = (byte >> (6 + (d & 1))) & 1u;
    return (byte >> (3 * (d & 1))) & 7u;
}

// One thread per word of the reference's records: key words, value words, sign words, norms.
__global__ void __launch_bounds__(128) kv_unpack_kernel(const unsigned char* __restrict__ base, int start, long n_vec, int heads, int dim,
                                                        KvArrays out) {
    const int wph = (dim + 9) / 10, qph = dim / 32, per = 2 * wph + qph + 1;
    const long i = static_cast<long>(blockIdx.x) * 128 + threadIdx.x;
    const long vec = i / per;
    if (vec >= n_vec) return;
    int item = static_cast<int>(i - vec * per);
    const long tok = vec / heads, token = start + tok;
    const int head = static_cast<int>(vec - tok * heads), slot = static_cast<int>(token & (kKvTile - 1));
    const unsigned char* const block = base + (static_cast<size_t>(token / kKvTile) * heads + head) * kv_block_bytes(dim);
    if (item < 2 * wph) {
        const bool value = item >= wph;
        const int w = value ? item - wph : item;
        uint32_t word = 0;
        for (int k = 0; k < 10 && w * 10 + k < dim; ++k) word |= stored_code(block, dim, slot, w * 10 + k, value, nullptr) << (3 * k);
        uint32_t* const dst = value ? out.v_words : out.k_words;
        if (dst) dst[vec * wph + w] = word;
        return;
    }
    item -= 2 * wph;
    if (item < qph) {
        uint32_t word = 0, bit = 0;
        for (int k = 0; k < 32; ++k) {
            stored_code(block, dim, slot, item * 32 + k, false, &bit);
            word |= bit << k;
        }
        if (out.qjl_words) out.qjl_words[vec * qph + item] = word;
        return;
    }
    const float* const norms = reinterpret_cast<const float*>(block + kv_block_bytes(dim) - 3 * kKvTile * 4);
    if (out.k_norms) out.k_norms[vec] = norms[kv_key_norm(slot)];
    if (out.v_norms) out.v_norms[vec] = norms[kv_value_norm(slot)];
    if (out.qjl_norms) out.qjl_norms[vec] = norms[kv_residual_norm(slot)];
}

__device__ __forceinline__ uint32_t array_code(const uint32_t* words, long vec, int wph, int d) {
    return (words[vec * wph + d / 10] >> (3 * (d % 10))) & 7u;
}

// One thread per (token pair, head) and word of the pair's records: the two tokens' key words, the value words, and one
// for the norms.  A token outside [start, start + tokens) keeps its bits.
__global__ void __launch_bounds__(128) kv_pack_kernel(unsigned char* __restrict__ base, int start, int tokens, int heads, int dim, KvArrays in) {
    const int wph = (dim + 9) / 10, qph = dim / 32, kw = dim / 8, vw = dim == 128 ? 8 : dim / 4, per = 2 * kw + vw + 1;
    const long i = static_cast<long>(blockIdx.x) * 128 + threadIdx.x;
    const long unit = i / per;
    const int pair0 = start >> 1, pairs = ((start + tokens - 1) >> 1) - pair0 + 1;
    if (unit >= static_cast<long>(pairs) * heads) return;
    int item = static_cast<int>(i - unit * per);
    const int pair = pair0 + static_cast<int>(unit / heads), head = static_cast<int>(unit % heads);
    auto inside = [&](int odd) { return 2 * pair + odd >= start && 2 * pair + odd < start + tokens; };
    auto vec_of = [&](int odd) { return static_cast<long>(2 * pair + odd - start) * heads + head; };
    const int slot = (2 * pair) & (kKvTile - 1);
    unsigned char* const block = base + (static_cast<size_t>(2 * pair / kKvTile) * heads + head) * kv_block_bytes(dim);
    if (item < 2 * kw) {
        const int odd = item >= kw ? 1 : 0, w = item - odd * kw;
        if (!inside(odd)) return;
        const long vec = vec_of(odd);
        uint32_t word = 0;
        for (int k = 0; k < 8; ++k) {
            const int d = w * 8 + k;
            const uint32_t sign = (in.qjl_words[vec * qph + (d >> 5)] >> (d & 31)) & 1u;
            word |= ((array_code(in.k_words, vec, wph, d) << (3 * (k & 1))) | (sign << (6 + (k & 1)))) << (8 * (k >> 1));
        }
        reinterpret_cast<uint32_t*>(block)[(slot + odd) * kw + w] = word;
        return;
    }
    item -= 2 * kw;
    if (item < vw) {
        // a packed group of 16 dims (three words), or four dims (one word)
        const int d0 = dim == 128 ? item * 16 : item * 4, n_words = dim == 128 ? 3 : 1;
        uint32_t w[4] = {0, 0, 0, 0};
        for (int odd = 0; odd < 2; ++odd) {
            if (!inside(odd)) continue;
            for (int k = 0; k < (dim == 128 ? 16 : 4); ++k) w[k >> 2] |= array_code(in.v_words, vec_of(odd), wph, d0 + k) << (8 * (k & 3) + 3 * odd);
        }
        for (int k = 0; k < n_words; ++k) {
            if (dim == 128) w[k] |= kv_spare_bits(w[3], k);
            const uint32_t keep = (inside(1) ? 0u : kv_odd_bits(dim, k)) | (inside(0) ? 0u : ~kv_odd_bits(dim, k));
            uint32_t* dst;
            if (dim == 128) dst = k < 2 ? kv_value01(block, slot >> 1, item) + k : kv_value2(block, slot >> 1, item);
            else dst = kv_value_row(block, dim, slot >> 1, 0) + item;
            *dst = (*dst & keep) | (w[k] & ~keep);
        }
        return;
    }
    float* const norms = reinterpret_cast<float*>(block + kv_block_bytes(dim) - 3 * kKvTile * 4);
    for (int odd = 0; odd < 2; ++odd) {
        if (!inside(odd)) continue;
        norms[kv_key_norm(slot + odd)] = in.k_norms[vec_of(odd)];
        norms[kv_value_norm(slot + odd)] = in.v_norms[vec_of(odd)];
        norms[kv_residual_norm(slot + odd)] = in.qjl_norms[vec_of(odd)];
    }
}

}  // namespace

#define TQ_D_SWITCH(DIM, MACRO)                                                    \
    switch (DIM) {                                                                 \
        case 32: MACRO(32) break;                                                  \
        case 64: MACRO(64) break;                                                  \
        case 128: MACRO(128) break;                                                \
        case 256: MACRO(256) break;                                                \
        case 512: MACRO(512) break;                                                \
        default: throw Error("head_dim must be a power of two in [32, 512]");      \
    }

void launch_kv_encode(const void* keys, const void* values, bool is_f16, int tokens_per_seg, int heads, int dim, uint32_t k_seed,
                      uint32_t v_seed, uint32_t qjl_seed, const KvSegment* segs, int n_segs, cudaStream_t stream) {
    TQ_REQUIRE(n_segs >= 1 && n_segs <= kKvMaxSegments, "kv encode: 1..32 segments per launch");
    if (tokens_per_seg == 0) return;
    const long units = 2L * n_segs * (tokens_per_seg / 2 + 1) * heads;   // token pairs of a head, keys and values
    TQ_REQUIRE(units < (1L << 28), "kv encode: too many vectors for one call");
    KvSegments tab{};
    for (int i = 0; i < n_segs; ++i) tab.seg[i] = segs[i];
    const float scale = std::sqrt(static_cast<float>(dim));             // src/kv_cache.cpp:72
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(dim));   // src/rotation.cpp:301
    const int aligned = reinterpret_cast<uintptr_t>(keys) % 16 == 0 && reinterpret_cast<uintptr_t>(values) % 16 == 0 ? 1 : 0;
    // Few vectors of 64 or 128 dims: eight dims per lane, up to 16 units per SM.  128 dims, 1040 / 2064 / 4112 units: 3.7 / 4.8 /
    // 8.7 us against 5.4 / 5.6 / 5.9 us with four lanes per vector; 64 dims: 3.0 / 3.3 / 4.4 against 3.3 / 3.4 / 3.7.  (32 dims,
    // 16 to 1040 units: 2.4 to 2.6 against 2.1 to 2.5.)
    if ((dim == 64 || dim == 128) && units <= 16 * 148) {
        const dim3 few(static_cast<unsigned>((units * 2 * (dim / 8) + 63) / 64));
#define TQ_ENC_FEW(DV)                                                                                                                \
    case DV:                                                                                                                          \
        if (is_f16)                                                                                                                   \
            launch_pdl(kv_encode_few_kernel<DV, __half>, few, dim3(64), 0, stream, static_cast<const __half*>(keys),                   \
                       static_cast<const __half*>(values), tokens_per_seg, n_segs, heads, k_seed, v_seed, qjl_seed, scale, inv_sqrt,  \
                       aligned, tab);                                                                                                 \
        else                                                                                                                          \
            launch_pdl(kv_encode_few_kernel<DV, float>, few, dim3(64), 0, stream, static_cast<const float*>(keys),                    \
                       static_cast<const float*>(values), tokens_per_seg, n_segs, heads, k_seed, v_seed, qjl_seed, scale, inv_sqrt,   \
                       aligned, tab);                                                                                                 \
        return;
        switch (dim) { TQ_ENC_FEW(64) TQ_ENC_FEW(128) }
#undef TQ_ENC_FEW
    }
    const dim3 grid(static_cast<unsigned>((units * 8 + 127) / 128));
#define TQ_ENC(DV)                                                                                                                    \
    if (is_f16)                                                                                                                       \
        launch_pdl(kv_encode_kernel<DV, __half>, grid, dim3(128), 0, stream, static_cast<const __half*>(keys),                        \
                   static_cast<const __half*>(values), tokens_per_seg, n_segs, heads, k_seed, v_seed, qjl_seed,           \
                   scale, inv_sqrt, aligned, tab);                                                                                    \
    else                                                                                                                              \
        launch_pdl(kv_encode_kernel<DV, float>, grid, dim3(128), 0, stream, static_cast<const float*>(keys),                          \
                   static_cast<const float*>(values), tokens_per_seg, n_segs, heads, k_seed, v_seed, qjl_seed,           \
                   scale, inv_sqrt, aligned, tab);
    TQ_D_SWITCH(dim, TQ_ENC)
#undef TQ_ENC
}

void launch_kv_decode_f16(const unsigned char* base, int start, int tokens, int heads, int dim, bool values, uint32_t wht_seed,
                          __half* out, cudaStream_t stream) {
    const long n = static_cast<long>(tokens) * heads;
    if (n == 0) return;
    const float inv_scale = 1.0f / std::sqrt(static_cast<float>(dim));  // src/kv_cache.cpp:302
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(dim));
    const dim3 grid(static_cast<unsigned>((n * 4 + 127) / 128));
#define TQ_DEC(DV) launch_pdl(kv_decode_kernel<DV>, grid, dim3(128), 0, stream, base, start, n, heads, values ? 1 : 0, wht_seed, inv_scale, inv_sqrt, out);
    TQ_D_SWITCH(dim, TQ_DEC)
#undef TQ_DEC
}

void launch_kv_unpack(const unsigned char* base, int start, int tokens, int heads, int dim, const KvArrays& out, cudaStream_t stream) {
    const long n = static_cast<long>(tokens) * heads;
    if (n == 0) return;
    const long threads = n * (2 * ((dim + 9) / 10) + dim / 32 + 1);
    kv_unpack_kernel<<<static_cast<unsigned>((threads + 127) / 128), 128, 0, stream>>>(base, start, n, heads, dim, out);
    TQ_CUDA(cudaGetLastError());
}

void launch_kv_pack(unsigned char* base, int start, int tokens, int heads, int dim, const KvArrays& in, cudaStream_t stream) {
    if (tokens == 0) return;
    const long pairs = ((start + tokens - 1) >> 1) - (start >> 1) + 1;
    const long threads = pairs * heads * (2 * (dim / 8) + (dim == 128 ? 8 : dim / 4) + 1);
    kv_pack_kernel<<<static_cast<unsigned>((threads + 127) / 128), 128, 0, stream>>>(base, start, tokens, heads, dim, in);
    TQ_CUDA(cudaGetLastError());
}

}  // namespace tq
