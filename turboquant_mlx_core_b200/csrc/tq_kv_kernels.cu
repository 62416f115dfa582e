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
// storage words are its own too, so nothing but two butterfly stages and the running sums crosses lanes.
template <int N>
__device__ __forceinline__ void quad_fwht(float (&v)[N], int q) {
#pragma unroll
    for (int h = 1; h < N; h <<= 1) {
#pragma unroll
        for (int i = 0; i < N; i += 2 * h) {
#pragma unroll
            for (int j = i; j < i + h; ++j) {
                const float a = v[j], b = v[j + h];
                v[j] = __fadd_rn(a, b);
                v[j + h] = __fsub_rn(a, b);
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
        const bool upper = (q & m) != 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, v[j], m);
            v[j] = upper ? __fsub_rn(other, v[j]) : __fadd_rn(v[j], other);
        }
    }
}

// sum over the vector of v[j]^2, accumulated left to right in fp32 (src/kv_cache.cpp:84-88, 226-231: the order is part of
// the result): the running sum goes through the quad's lanes in turn.
template <int N>
__device__ __forceinline__ float quad_square_sum(const float (&v)[N], int lane) {
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float t = acc;
#pragma unroll
        for (int j = 0; j < N; ++j) t = __fadd_rn(t, __fmul_rn(v[j], v[j]));
        acc = __shfl_sync(0xffffffffu, t, (lane & 28) + k);
    }
    return acc;
}

// v with its sign flipped where bit j of the word is clear: v * sign_value, without the multiplication.
__device__ __forceinline__ float flip_unless(float v, uint32_t word, int j) {
    return __uint_as_float(__float_as_uint(v) ^ ((~word << (31 - j)) & 0x80000000u));
}

struct KvSegments {
    KvSegment seg[kKvMaxSegments];
};

// ---- encoder (src/kv_cache.cpp:63-258) ---------------------------------------------------------------
// Vectors 0 .. n - 1 are the keys, n .. 2 n - 1 the values; segment s takes vec_per_seg vectors.  Bit-exact: the sums of
// squares run left to right, every other operation is element-wise or the shared butterfly.
// Bound: issue slots (about 1100 instructions per lane and vector).  A warp per vector with one lane summing while 31
// waited took 47 us for 2 x 32768 vectors of 128 (two launches), and a batched variant existed beside it for long
// appends; four lanes per vector serve both.
template <int D, typename InT>
__global__ void __launch_bounds__(128) kv_encode_kernel(const InT* __restrict__ keys, const InT* __restrict__ values, int n, int heads,
                                                        int vec_per_seg, uint32_t k_seed, uint32_t v_seed, uint32_t qjl_seed,
                                                        float scale, float inv_sqrt, int aligned,
                                                        const __grid_constant__ KvSegments tab) {
    constexpr int N = D / 4, W = N / 8;
    using B = KvBlock<D>;
    __shared__ uint32_t s_sign[3][D / 32];   // key rotation, value rotation, residual signs: bit set = +1
    for (int i = threadIdx.x; i < 3 * D; i += 128) {
        const int which = i / D, d = i - which * D;
        const bool pos = which == 2 ? qjl_sign_is_positive(qjl_seed, static_cast<uint32_t>(d))
                                    : sign_is_positive(which ? v_seed : k_seed, static_cast<uint32_t>(d));
        const uint32_t bits = __ballot_sync(__activemask(), pos);
        if ((i & 31) == 0) s_sign[which][d >> 5] = bits;
    }
    __syncthreads();
    pdl_wait_release();

    const int lane = threadIdx.x & 31, q = lane & 3;
    const long quad = (static_cast<long>(blockIdx.x) * 128 + threadIdx.x) >> 2;
    const bool live = quad < 2L * n;
    const long vec = live ? quad : 2L * n - 1;
    const bool value = vec >= n;
    const int gvec = static_cast<int>(value ? vec - n : vec);
    const InT* const src = (value ? values : keys) + static_cast<size_t>(gvec) * D + q * N;

    float v[N];
    if (aligned) {
        constexpr int kPer = 16 / static_cast<int>(sizeof(InT));
#pragma unroll
        for (int i = 0; i < N / kPer; ++i) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src) + i);
            const InT* e = reinterpret_cast<const InT*>(&raw);
#pragma unroll
            for (int j = 0; j < kPer; ++j) v[i * kPer + j] = as_f32<InT>(e[j]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = as_f32<InT>(src[j]);
    }
    const float norm = __fsqrt_rn(quad_square_sum<N>(v, lane));
    const float inv_norm = (norm > 1e-10f) ? __fdiv_rn(1.0f, norm) : 0.0f;
    const uint32_t* const signs = s_sign[value ? 1 : 0];
    auto sign_word = [&](const uint32_t* s, int j) { return s[(q * N + j) >> 5]; };   // of this lane's dim j (N >= 8)
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t w = sign_word(signs, j);
        v[j] = flip_unless(__fmul_rn(v[j], inv_norm), N >= 32 ? w : w >> ((q * N) & 31), j & 31);
    }
    quad_fwht<N>(v, q);

    // Codes.  The boundaries are the centroids' midpoints: +-t1, +-t2, +-t3 and zero, and a code is the number of
    // boundaries below the value.  For v > 0 that is 4 + #{t < |v|}, otherwise 3 - #{t <= |v|}; one more unit in the last
    // place on |v| turns the second comparison into the first.
    const uint32_t t1 = __float_as_uint(__fmul_rn(__fadd_rn(kMag0, kMag1), 0.5f));
    const uint32_t t2 = __float_as_uint(__fmul_rn(__fadd_rn(kMag1, kMag2), 0.5f));
    const uint32_t t3 = __float_as_uint(__fmul_rn(__fadd_rn(kMag2, kMag3), 0.5f));
    uint32_t words[W];
#pragma unroll
    for (int w = 0; w < W; ++w) words[w] = 0u;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const float x = __fmul_rn(__fmul_rn(v[j], inv_sqrt), scale);
        const bool pos = x > 0.0f;
        const uint32_t a = (__float_as_uint(x) & 0x7fffffffu) + (pos ? 0u : 1u);
        const uint32_t m = (a > t1 ? 1u : 0u) + (a > t2 ? 1u : 0u) + (a > t3 ? 1u : 0u);
        uint32_t nib = pos ? 4u + m : 3u - m;
        const float mag = a > t3 ? kMag3 : (a > t2 ? kMag2 : (a > t1 ? kMag1 : kMag0));
        const float r = __fsub_rn(x, pos ? mag : -mag);
        v[j] = r;
        if (!value) {
            const uint32_t w = sign_word(s_sign[2], j);
            const bool qpos = ((N >= 32 ? w : w >> ((q * N) & 31)) >> (j & 31)) & 1u;
            if (qpos ? r > 0.0f : r < 0.0f) nib |= 8u;
        }
        words[j / 8] |= nib << (4 * (j & 7));
    }
    const float rnorm = __fsqrt_rn(quad_square_sum<N>(v, lane));   // of the residual; only the keys keep it
    if (!live) return;

    const int sidx = gvec / vec_per_seg, rest = gvec - sidx * vec_per_seg;
    const int tok = rest / heads, head = rest - tok * heads;
    const int token = tab.seg[sidx].first + tok, slot = token & (kKvTile - 1);
    unsigned char* const block = tab.seg[sidx].base + (static_cast<size_t>(token / kKvTile) * heads + head) * B::kBytes;
    if (value && D == 128) {
        uint2 w01;
        w01.x = words[0] | ((words[W - 1] & 0x11111111u) << 3);
        w01.y = words[1 % W] | ((words[W - 1] & 0x22222222u) << 2);
        *reinterpret_cast<uint2*>(kv_value01(block, slot, q)) = w01;
        *kv_value2(block, slot, q) = words[2 % W] | ((words[W - 1] & 0x44444444u) << 1);
    } else {
        uint32_t* const dst = reinterpret_cast<uint32_t*>(block + (value ? B::kValueOff : 0)) + slot * (D / 8) + q * W;
        if constexpr (W % 4 == 0) {
#pragma unroll
            for (int w = 0; w < W; w += 4) *reinterpret_cast<uint4*>(dst + w) = make_uint4(words[w], words[w + 1], words[w + 2], words[w + 3]);
        } else {
#pragma unroll
            for (int w = 0; w < W; ++w) dst[w] = words[w];
        }
    }
    if (q == 0) {
        float* const norms = reinterpret_cast<float*>(block + B::kNormOff);
        norms[(value ? kKvTile : 0) + slot] = norm;
        if (!value) norms[2 * kKvTile + slot] = rnorm;
    }
}

// ---- range decoder (src/kv_cache.cpp:292-365) ----------------------------------------------------------
// Four lanes per vector as in the encoder.  The centroids sit in shared memory once per lane: as a constant array they
// were read one lane at a time (86 us for 65536 tokens of 4 heads).
template <int D>
__global__ void __launch_bounds__(128) kv_decode_kernel(const unsigned char* __restrict__ base, int start, long n_vec, int heads, int values,
                                                        uint32_t wht_seed, float inv_scale, float inv_sqrt, __half* __restrict__ out) {
    constexpr int N = D / 4, W = N / 8;
    using B = KvBlock<D>;
    __shared__ float s_cent[8][32];
    __shared__ uint32_t s_sign[D / 32];
    for (int i = threadIdx.x; i < 256; i += 128) {
        const int c = i >> 5, m = c < 4 ? 3 - c : c - 4;
        const float mag = m == 3 ? kMag3 : (m == 2 ? kMag2 : (m == 1 ? kMag1 : kMag0));
        s_cent[c][i & 31] = __fmul_rn(c < 4 ? -mag : mag, inv_scale);
    }
    for (int i = threadIdx.x; i < D; i += 128) {
        const uint32_t bits = __ballot_sync(__activemask(), sign_is_positive(wht_seed, static_cast<uint32_t>(i)));
        if ((i & 31) == 0) s_sign[i >> 5] = bits;
    }
    __syncthreads();
    pdl_wait_release();
    const int lane = threadIdx.x & 31, q = lane & 3;
    const long quad = (static_cast<long>(blockIdx.x) * 128 + threadIdx.x) >> 2;
    const bool live = quad < n_vec;
    const long vec = live ? quad : n_vec - 1;
    const long tok = vec / heads;
    const int head = static_cast<int>(vec - tok * heads);
    const long token = start + tok;
    const int slot = static_cast<int>(token & (kKvTile - 1));
    unsigned char* const block = const_cast<unsigned char*>(base) + (static_cast<size_t>(token / kKvTile) * heads + head) * B::kBytes;
    uint32_t words[W];
    if (values && D == 128) {
        const uint2 w01 = *reinterpret_cast<const uint2*>(kv_value01(block, slot, q));
        words[0] = w01.x;
        words[1 % W] = w01.y;
        words[2 % W] = *kv_value2(block, slot, q);
        words[W - 1] = kv_value_spare(words[0], words[1 % W], words[2 % W]);
    } else {
        const uint32_t* const src = reinterpret_cast<const uint32_t*>(block + (values ? B::kValueOff : 0)) + slot * (D / 8) + q * W;
#pragma unroll
        for (int w = 0; w < W; ++w) words[w] = src[w];
    }
    const float norm = reinterpret_cast<const float*>(block + B::kNormOff)[(values ? kKvTile : 0) + slot];
    float v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = s_cent[(words[j / 8] >> (4 * (j & 7))) & 7u][lane];
    quad_fwht<N>(v, q);
    __align__(16) __half h[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t w = s_sign[(q * N + j) >> 5];
        h[j] = __float2half_rn(__fmul_rn(flip_unless(__fmul_rn(v[j], inv_sqrt), N >= 32 ? w : w >> ((q * N) & 31), j & 31), norm));
    }
    if (!live) return;
    __half* const dst = out + static_cast<size_t>(vec) * D + q * N;
    if (reinterpret_cast<uintptr_t>(out) % 16 == 0) {
#pragma unroll
        for (int c = 0; c < N / 8; ++c) reinterpret_cast<uint4*>(dst)[c] = reinterpret_cast<const uint4*>(h)[c];
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) dst[j] = h[j];
    }
}

// ---- the reference's arrays ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t stored_code(const unsigned char* block, int dim, int slot, int d, bool value, uint32_t* sign) {
    const int key_bytes = kKvTile * dim / 2;
    if (value && dim == 128) {
        unsigned char* const b = const_cast<unsigned char*>(block);
        const int q = d >> 5, r = d & 31;
        const uint32_t w0 = kv_value01(b, slot, q)[0], w1 = kv_value01(b, slot, q)[1], w2 = *kv_value2(b, slot, q);
        const uint32_t w = r < 8 ? w0 : (r < 16 ? w1 : (r < 24 ? w2 : kv_value_spare(w0, w1, w2)));
        return (w >> (4 * (r & 7))) & 7u;
    }
    const uint32_t* const w = reinterpret_cast<const uint32_t*>(block + (value ? key_bytes : 0)) + slot * (dim / 8);
    const uint32_t nib = w[d >> 3] >> (4 * (d & 7));
    if (sign) *sign = (nib >> 3) & 1u;
    return nib & 7u;
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
    if (out.k_norms) out.k_norms[vec] = norms[slot];
    if (out.v_norms) out.v_norms[vec] = norms[kKvTile + slot];
    if (out.qjl_norms) out.qjl_norms[vec] = norms[2 * kKvTile + slot];
}

__device__ __forceinline__ uint32_t array_code(const uint32_t* words, long vec, int wph, int d) {
    return (words[vec * wph + d / 10] >> (3 * (d % 10))) & 7u;
}

// One thread per word of the storage: key nibbles, value words, and one for the norms.
__global__ void __launch_bounds__(128) kv_pack_kernel(unsigned char* __restrict__ base, int start, long n_vec, int heads, int dim, KvArrays in) {
    const int wph = (dim + 9) / 10, qph = dim / 32, kw = dim / 8, vw = dim == 128 ? 4 : dim / 8, per = kw + vw + 1;
    const long i = static_cast<long>(blockIdx.x) * 128 + threadIdx.x;
    const long vec = i / per;
    if (vec >= n_vec) return;
    int item = static_cast<int>(i - vec * per);
    const long tok = vec / heads, token = start + tok;
    const int head = static_cast<int>(vec - tok * heads), slot = static_cast<int>(token & (kKvTile - 1));
    unsigned char* const block = base + (static_cast<size_t>(token / kKvTile) * heads + head) * kv_block_bytes(dim);
    const int key_bytes = kKvTile * dim / 2;
    if (item < kw) {
        uint32_t word = 0;
        for (int k = 0; k < 8; ++k) {
            const int d = item * 8 + k;
            const uint32_t sign = (in.qjl_words[vec * qph + (d >> 5)] >> (d & 31)) & 1u;
            word |= (array_code(in.k_words, vec, wph, d) | (sign << 3)) << (4 * k);
        }
        reinterpret_cast<uint32_t*>(block)[slot * kw + item] = word;
        return;
    }
    item -= kw;
    if (item < vw) {
        if (dim == 128) {
            uint32_t w[4] = {0, 0, 0, 0};
            for (int k = 0; k < 32; ++k) w[k >> 3] |= array_code(in.v_words, vec, wph, item * 32 + k) << (4 * (k & 7));
            kv_value01(block, slot, item)[0] = w[0] | ((w[3] & 0x11111111u) << 3);
            kv_value01(block, slot, item)[1] = w[1] | ((w[3] & 0x22222222u) << 2);
            *kv_value2(block, slot, item) = w[2] | ((w[3] & 0x44444444u) << 1);
        } else {
            uint32_t word = 0;
            for (int k = 0; k < 8; ++k) word |= array_code(in.v_words, vec, wph, item * 8 + k) << (4 * k);
            reinterpret_cast<uint32_t*>(block + key_bytes)[slot * kw + item] = word;
        }
        return;
    }
    float* const norms = reinterpret_cast<float*>(block + kv_block_bytes(dim) - 3 * kKvTile * 4);
    norms[slot] = in.k_norms[vec];
    norms[kKvTile + slot] = in.v_norms[vec];
    norms[2 * kKvTile + slot] = in.qjl_norms[vec];
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
    const long n = static_cast<long>(tokens_per_seg) * heads * n_segs;
    if (n == 0) return;
    TQ_REQUIRE(n < (1L << 31), "kv encode: too many vectors for one call");
    KvSegments tab{};
    for (int i = 0; i < n_segs; ++i) tab.seg[i] = segs[i];
    const float scale = std::sqrt(static_cast<float>(dim));             // src/kv_cache.cpp:72
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(dim));   // src/rotation.cpp:301
    const int aligned = reinterpret_cast<uintptr_t>(keys) % 16 == 0 && reinterpret_cast<uintptr_t>(values) % 16 == 0 ? 1 : 0;
    const dim3 grid(static_cast<unsigned>((2 * n * 4 + 127) / 128));
#define TQ_ENC(DV)                                                                                                                    \
    if (is_f16)                                                                                                                       \
        launch_pdl(kv_encode_kernel<DV, __half>, grid, dim3(128), 0, stream, static_cast<const __half*>(keys),                        \
                   static_cast<const __half*>(values), static_cast<int>(n), heads, tokens_per_seg * heads, k_seed, v_seed, qjl_seed,  \
                   scale, inv_sqrt, aligned, tab);                                                                                    \
    else                                                                                                                              \
        launch_pdl(kv_encode_kernel<DV, float>, grid, dim3(128), 0, stream, static_cast<const float*>(keys),                          \
                   static_cast<const float*>(values), static_cast<int>(n), heads, tokens_per_seg * heads, k_seed, v_seed, qjl_seed,   \
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
    const long n = static_cast<long>(tokens) * heads;
    if (n == 0) return;
    const long threads = n * (dim / 8 + (dim == 128 ? 4 : dim / 8) + 1);
    kv_pack_kernel<<<static_cast<unsigned>((threads + 127) / 128), 128, 0, stream>>>(base, start, n, heads, dim, in);
    TQ_CUDA(cudaGetLastError());
}

}  // namespace tq
