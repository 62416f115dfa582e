// The element-wise glue of a decoder layer around the quantised linears and the compressed-cache
// attention: RMSNorm, rotary position embedding, SwiGLU.  The reference leaves these to MLX
// (mlx::core::fast::rms_norm / rope and plain array arithmetic in the host application); they are here
// so that a whole tensor-parallel decode step can be timed.  fp16 in and out, fp32 arithmetic;
// every kernel is memory-bound (a few bytes per element) and carries the programmatic-launch wait
// so that it can follow the kernels of this library without a launch gap.
#include <cmath>
#include <cstdint>

#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

__device__ __forceinline__ void ops_dependency_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

// y[r, :] = x[r, :] * rsqrt(mean(x[r, :]^2) + eps) * w      one CTA per row
template <bool WIDE, int KEEP>
__global__ void __launch_bounds__(kRowNormThreads, row_ctas(KEEP)) rmsnorm_kernel(const __half* __restrict__ x, const __half* __restrict__ w, __half* __restrict__ y,
                                                      int cols, float eps) {
    ops_dependency_sync();
    behind_wait(x, w);
    rmsnorm_row<WIDE, KEEP>(x + static_cast<size_t>(blockIdx.x) * cols, w, y + static_cast<size_t>(blockIdx.x) * cols, cols, eps);
}

// Rotary embedding, "rotate half" convention: element i of a head pairs with element i + d/2;
// angle = position * theta^(-2 i / d).  x: [rows, heads, d] in place, positions: [rows].
// A second tensor x2 [rows, heads2, d] (the keys beside the queries) rides in the same launch: pairs beyond x's.
__global__ void __launch_bounds__(128) rope_kernel(__half* __restrict__ x, const int* __restrict__ positions, int heads, int dim,
                                                   float log2_theta, long total_pairs, __half* __restrict__ x2, int heads2, long total_pairs2) {
    ops_dependency_sync();
    behind_wait(x, positions, x2);
    const int half = dim >> 1;
    for (long i0 = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < total_pairs + total_pairs2;
         i0 += static_cast<long>(gridDim.x) * blockDim.x) {
        const bool second = i0 >= total_pairs;
        const long i = second ? i0 - total_pairs : i0;
        __half* const xb = second ? x2 : x;
        const int hh = second ? heads2 : heads;
        const int p = static_cast<int>(i % half);
        const long vec = i / half;               // (row, head)
        const long row = vec / hh;
        const float inv_freq = exp2f(-log2_theta * (2.0f * static_cast<float>(p) / static_cast<float>(dim)));
        float s, c;
        sincosf(static_cast<float>(positions[row]) * inv_freq, &s, &c);
        __half* v = xb + vec * dim;
        const float a = __half2float(v[p]), b = __half2float(v[p + half]);
        v[p] = __float2half_rn(a * c - b * s);
        v[p + half] = __float2half_rn(b * c + a * s);
    }
}

// The same for heads of a multiple of 16 elements, 16-byte aligned: a CTA per row.  The angles of a row are the same for all
// its heads: dim / 2 threads take the sines and cosines once, to shared memory, and a thread rotates eight pairs at a time
// (2048 rows of 28 + 4 heads of 128: 34 us with a sine and a cosine per pair and 2-byte accesses).
constexpr int kRopeThreads = 256, kRopeHalfMax = 256;
__global__ void __launch_bounds__(kRopeThreads) rope_rows_kernel(__half* __restrict__ x, const int* __restrict__ positions, int heads, int dim,
                                                                 float log2_theta, __half* __restrict__ x2, int heads2) {
    ops_dependency_sync();
    behind_wait(x, positions, x2);
    __shared__ __align__(16) float s_cos[kRopeHalfMax], s_sin[kRopeHalfMax];
    const int half = dim >> 1, per_head = half / 8, items = (heads + heads2) * per_head;
    const long row = blockIdx.x;
    for (int p = threadIdx.x; p < half; p += kRopeThreads) {
        const float inv_freq = exp2f(-log2_theta * (2.0f * static_cast<float>(p) / static_cast<float>(dim)));
        sincosf(static_cast<float>(positions[row]) * inv_freq, &s_sin[p], &s_cos[p]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < items; i += kRopeThreads) {
        const int h = i / per_head, p = (i - h * per_head) * 8;
        __half* const v = (h < heads ? x + (row * heads + h) * dim : x2 + (row * heads2 + (h - heads)) * dim) + p;
        float a[8], b[8], lo[8], hi[8];
        unpack_halves(*reinterpret_cast<const uint4*>(v), a);
        unpack_halves(*reinterpret_cast<const uint4*>(v + half), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float c = s_cos[p + j], s = s_sin[p + j];
            lo[j] = a[j] * c - b[j] * s;
            hi[j] = b[j] * c + a[j] * s;
        }
        *reinterpret_cast<uint4*>(v) = pack_halves(lo);
        *reinterpret_cast<uint4*>(v + half) = pack_halves(hi);
    }
}

// act[r, j] = silu(gate_up[r, j]) * gate_up[r, inter + j]      (gate rows first, then up rows)
__device__ __forceinline__ float swiglu(float g, float u) { return g / (1.0f + __expf(-g)) * u; }
// Rows of a multiple of eight elements, 16-byte aligned: eight per thread, a row per blockIdx.y (2048 x 18944: 77 us with
// two per thread and a 64-bit division for each pair).
__global__ void __launch_bounds__(256) swiglu_wide_kernel(const __half* __restrict__ gate_up, __half* __restrict__ act, int inter, long rows) {
    ops_dependency_sync();
    behind_wait(gate_up);
    const int j = (blockIdx.x * 256 + threadIdx.x) * 8;
    if (j >= inter) return;
    for (long r = blockIdx.y; r < rows; r += gridDim.y) {
        const __half* const src = gate_up + r * 2 * inter + j;
        float g[8], u[8];
        unpack_halves(*reinterpret_cast<const uint4*>(src), g);
        unpack_halves(*reinterpret_cast<const uint4*>(src + inter), u);
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] = swiglu(g[k], u[k]);
        *reinterpret_cast<uint4*>(act + r * inter + j) = pack_halves(g);
    }
}
__global__ void __launch_bounds__(256) swiglu_kernel(const __half* __restrict__ gate_up, __half* __restrict__ act, int inter, long rows) {
    ops_dependency_sync();
    behind_wait(gate_up);
    const long total = rows * inter;
    for (long i = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) * 2; i < total; i += static_cast<long>(gridDim.x) * blockDim.x * 2) {
        const long r = i / inter, j = i - r * inter;
        const float2 g = __half22float2(*reinterpret_cast<const __half2*>(gate_up + r * 2 * inter + j));
        const float2 u = __half22float2(*reinterpret_cast<const __half2*>(gate_up + r * 2 * inter + inter + j));
        *reinterpret_cast<__half2*>(act + i) = __floats2half2_rn(swiglu(g.x, u.x), swiglu(g.y, u.y));
    }
}

cudaLaunchConfig_t ops_config(unsigned grid, unsigned block, cudaStream_t stream, cudaLaunchAttribute* attr) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

void launch_rmsnorm_f16(const __half* x, const __half* weight, __half* y, long rows, int cols, float eps, cudaStream_t stream) {
    TQ_REQUIRE(x && weight && y, "rmsnorm: NULL argument");
    TQ_REQUIRE(cols > 0 && cols % 2 == 0, "rmsnorm: an even number of columns");
    if (rows == 0) return;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = ops_config(static_cast<unsigned>(rows), kRowNormThreads, stream, attr);
    decltype(&rmsnorm_kernel<true, 1>) kernel;
    TQ_ROW_KERNEL(kernel, rmsnorm_kernel, rows_wide(cols, x, weight, y), cols)
    TQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, x, weight, y, cols, eps));
}

// Whether the row kernel took the call: head sizes up to 512 in sixteens, aligned tensors.
static bool launch_rope_rows(__half* x, __half* x2, const int* positions, long rows, int heads, int heads2, int dim, float theta,
                             cudaStream_t stream) {
    if (dim % 16 != 0 || dim / 2 > kRopeHalfMax || (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x2)) % 16 != 0 || rows >= (1L << 31) ||
        (static_cast<long>(heads) + heads2) * dim >= (1L << 31))
        return false;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = ops_config(static_cast<unsigned>(rows), kRopeThreads, stream, attr);
    TQ_CUDA(cudaLaunchKernelEx(&cfg, rope_rows_kernel, x, positions, heads, dim, std::log2(theta), x2, heads2));
    return true;
}

void launch_rope_f16(__half* x, const int* positions, long rows, int heads, int dim, float theta, cudaStream_t stream) {
    TQ_REQUIRE(x && positions, "rope: NULL argument");
    TQ_REQUIRE(dim > 0 && dim % 2 == 0 && heads > 0 && theta > 1.0f, "rope: bad shape");
    if (rows == 0) return;
    if (launch_rope_rows(x, nullptr, positions, rows, heads, 0, dim, theta, stream)) return;
    const long pairs = rows * heads * (dim / 2);
    long blocks = (pairs + 127) / 128;
    if (blocks > 1184) blocks = 1184;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = ops_config(static_cast<unsigned>(blocks), 128, stream, attr);
    TQ_CUDA(cudaLaunchKernelEx(&cfg, rope_kernel, x, positions, heads, dim, std::log2(theta), pairs, static_cast<__half*>(nullptr), 1, 0L));
}

void launch_rope_qk_f16(__half* q, __half* k, const int* positions, long rows, int q_heads, int kv_heads, int dim, float theta,
                        cudaStream_t stream) {
    TQ_REQUIRE(q && k && positions, "rope: NULL argument");
    TQ_REQUIRE(dim > 0 && dim % 2 == 0 && q_heads > 0 && kv_heads > 0 && theta > 1.0f, "rope: bad shape");
    if (rows == 0) return;
    if (launch_rope_rows(q, k, positions, rows, q_heads, kv_heads, dim, theta, stream)) return;
    const long pairs_q = rows * q_heads * (dim / 2), pairs_k = rows * kv_heads * (dim / 2);
    long blocks = (pairs_q + pairs_k + 127) / 128;
    if (blocks > 1184) blocks = 1184;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = ops_config(static_cast<unsigned>(blocks), 128, stream, attr);
    TQ_CUDA(cudaLaunchKernelEx(&cfg, rope_kernel, q, positions, q_heads, dim, std::log2(theta), pairs_q, k, kv_heads, pairs_k));
}

void launch_swiglu_f16(const __half* gate_up, __half* act, long rows, int inter, cudaStream_t stream) {
    TQ_REQUIRE(gate_up && act, "swiglu: NULL argument");
    TQ_REQUIRE(inter > 0 && inter % 2 == 0, "swiglu: an even intermediate size");
    if (rows == 0) return;
    cudaLaunchAttribute attr[1];
    if (inter % 8 == 0 && (reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(act)) % 16 == 0) {
        cudaLaunchConfig_t wide = ops_config(static_cast<unsigned>((inter / 8 + 255) / 256), 256, stream, attr);
        wide.gridDim.y = static_cast<unsigned>(rows < 65535 ? rows : 65535);
        TQ_CUDA(cudaLaunchKernelEx(&wide, swiglu_wide_kernel, gate_up, act, inter, rows));
        return;
    }
    long blocks = (rows * inter / 2 + 255) / 256;
    if (blocks > 1184) blocks = 1184;
    cudaLaunchConfig_t cfg = ops_config(static_cast<unsigned>(blocks), 256, stream, attr);
    TQ_CUDA(cudaLaunchKernelEx(&cfg, swiglu_kernel, gate_up, act, inter, rows));
}

}  // namespace tq
