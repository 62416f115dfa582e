// Activation rows of a caller without device buffers.
//
// A decode call hands over 8 KB and waits for 8 KB.  Through cudaMemcpyAsync from pageable memory, a conversion kernel and
// a copy back the 4096 x 4096 layer took 45 us, 8 of them in the layer's kernel.  Up to 31 KB of rows now ride in the
// parameters of a kernel, which the launch delivers with no copy engine and no staging in between; the host
// rounds fp32 to fp16 on the way (half the bytes, no conversion kernel).  One row that the decode kernel rotates itself is a
// parameter of that kernel (gemv_takes_host_row); several rows and other blocks go through the one-CTA kernel here.
#include <cstring>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

// fp32 -> fp16, round to nearest even: the bits __float2half_rn gives.  (The steps are the well-known ones: rebias and add
// half a unit less a tie's bit, add 0.5 for subnormal results; F. Giesen's public float_to_half collection has them.)  A loop
// of one value at a time, as the compiler makes of this, takes 4 us for 4096 values, and where it came to lie moved a call by
// 1.3 of 34 us; the processor's own conversion does eight at a time.
static void f32_to_f16_portable(const float* src, uint16_t* dst, size_t n) {
    for (size_t i = 0; i < n; ++i) {
        uint32_t u;
        std::memcpy(&u, src + i, 4);
        const uint32_t sign = (u >> 16) & 0x8000u, a = u & 0x7fffffffu;
        // normal results: drop 13 bits with a tie to even, rebias the exponent
        const uint32_t normal = (a + 0xfffu + ((a >> 13) & 1u) - (112u << 23)) >> 13;
        // results below 2^-14: adding 0.5 puts the result's last bit at the sum's last bit
        float f;
        std::memcpy(&f, &a, 4);
        f += 0.5f;
        uint32_t small;
        std::memcpy(&small, &f, 4);
        small -= 0x3f000000u;
        uint32_t h = a < (113u << 23) ? small : normal;
        h = a >= 0x477ff000u ? 0x7c00u : h;   // 65520 and above round to infinity
        h = a > 0x7f800000u ? 0x7fffu : h;    // NaN
        dst[i] = static_cast<uint16_t>(h > 0x7ffeu ? 0x7fffu : (h | sign));
    }
}
#if defined(__x86_64__)
__attribute__((target("avx,f16c"))) static void f32_to_f16_eight(const float* src, uint16_t* dst, size_t n) {
    size_t i = 0;
    for (; i + 8 <= n; i += 8) {
        const __m256 v = _mm256_loadu_ps(src + i);
        if (_mm256_movemask_ps(_mm256_cmp_ps(v, v, _CMP_UNORD_Q)) != 0) f32_to_f16_portable(src + i, dst + i, 8);   // a NaN: 0x7fff, whatever its bits
        else _mm_storeu_si128(reinterpret_cast<__m128i*>(dst + i), _mm256_cvtps_ph(v, _MM_FROUND_TO_NEAREST_INT));
    }
    f32_to_f16_portable(src + i, dst + i, n - i);
}
#endif
void host_f32_to_f16(const float* src, uint16_t* dst, size_t n) {
#if defined(__x86_64__)
    static const bool eight = __builtin_cpu_supports("avx") && __builtin_cpu_supports("f16c");
    if (eight) return f32_to_f16_eight(src, dst, n);
#endif
    f32_to_f16_portable(src, dst, n);
}

namespace {

template <int N>
struct ParamRows {
    uint4 v[N];
};

template <int N>
__global__ void __launch_bounds__(256) rows_from_params_kernel(const __grid_constant__ ParamRows<N> rows, uint4* __restrict__ dst, int n) {
    pdl_wait_release();
    for (int i = threadIdx.x; i < n; i += 256) dst[i] = rows.v[i];
}

template <int N>
void launch_n(const void* host_x, bool is_f16, size_t n, __half* dst, cudaStream_t stream) {
    ParamRows<N> rows;
    if (is_f16) std::memcpy(rows.v, host_x, n * 2);
    else host_f32_to_f16(static_cast<const float*>(host_x), reinterpret_cast<uint16_t*>(rows.v), n);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    uint4* out = reinterpret_cast<uint4*>(dst);
    int pieces = static_cast<int>((n * 2 + 15) / 16);
    void* args[] = {&rows, &out, &pieces};   // by address: the rows are copied once, into the launch
    TQ_CUDA(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(rows_from_params_kernel<N>), args));
}

}  // namespace

// dst holds n fp16 values rounded up to 16 bytes.
void launch_rows_from_params(const void* host_x, bool is_f16, size_t n, __half* dst, cudaStream_t stream) {
    const size_t bytes = n * 2;
    TQ_REQUIRE(bytes <= kMaxParamRowBytes, "activation rows do not fit a launch's parameters");
    // the launch copies its whole parameter block: sizes in steps of two
    if (bytes <= 2048) launch_n<128>(host_x, is_f16, n, dst, stream);
    else if (bytes <= 4096) launch_n<256>(host_x, is_f16, n, dst, stream);
    else if (bytes <= 8192) launch_n<512>(host_x, is_f16, n, dst, stream);
    else if (bytes <= 16384) launch_n<1024>(host_x, is_f16, n, dst, stream);
    else launch_n<kMaxParamRowBytes / 16>(host_x, is_f16, n, dst, stream);
}

}  // namespace tq
