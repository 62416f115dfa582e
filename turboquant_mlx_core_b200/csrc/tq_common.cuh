// Shared device/host helpers for the TurboQuant sm_100a kernels.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <stdexcept>
#include <string>

namespace tq {

// ---- errors --------------------------------------------------------------------
// Host code throws; the C boundary catches and turns exceptions into status codes
// plus a thread-local message (no exception crosses the ABI).
struct Error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
    if (e != cudaSuccess) {
        throw Error(std::string(what) + ": " + cudaGetErrorString(e) + " (" + file + ":" + std::to_string(line) + ")");
    }
}
#define TQ_CUDA(x) ::tq::cuda_check((x), #x, __FILE__, __LINE__)
#define TQ_REQUIRE(cond, msg)                    \
    do {                                         \
        if (!(cond)) throw ::tq::Error(msg);     \
    } while (0)

// ---- sign hash -----------------------------------------------------------------
// Same integer hash as the reference's make_signs (src/rotation.cpp:32-42): the index
// is the position inside the WHT block, so one sign vector serves every block and row.
__host__ __device__ __forceinline__ bool sign_is_positive(uint32_t seed, uint32_t i) {
    uint32_t h = seed * 2654435761u + i * 2246822519u;
    h ^= h >> 16;
    h *= 0x45d9f3bu;
    h ^= h >> 16;
    return (h & 1u) != 0u;
}
__host__ __device__ __forceinline__ float sign_value(uint32_t seed, uint32_t i) {
    return sign_is_positive(seed, i) ? 1.0f : -1.0f;
}

// QJL key-side sign (src/kv_cache.cpp:249-250): top bit of the un-avalanched hash.
__host__ __device__ __forceinline__ bool qjl_sign_is_positive(uint32_t seed, uint32_t d) {
    uint32_t h = seed * 2654435761u + d * 2246822519u;
    return (h >> 31) != 0u;
}

// Per-layer KV seeds (src/kv_cache.cpp:32-42). which: 1 = K rotation, 2 = V rotation, 3 = QJL.
__host__ __device__ __forceinline__ uint32_t kv_layer_seed(uint32_t layer, uint32_t which) {
    uint32_t h = layer;
    h ^= which + 0x9e3779b9u + (h << 6) + (h >> 2);
    h = (h ^ (h >> 16)) * 0x45d9f3bu;
    h = (h ^ (h >> 16)) * 0x45d9f3bu;
    h ^= h >> 16;
    return h;
}

// ---- warp-level Walsh-Hadamard butterfly -----------------------------------------
// One warp transforms one block of 32*E values; lane l holds elements [l*E, (l+1)*E).
// The add tree is the reference's (src/rotation.cpp:14-25): for h = 1, 2, 4, ... the
// pair (j, j+h) becomes (a+b, a-b) with a the lower index.  Stages h < E stay in
// registers; stages h >= E exchange with lane ^ (h/E).  Only __fadd_rn/__fsub_rn, and multiply-adds with +-1, which
// round as they do, are used so nothing else can be contracted into an FMA: results are bit-identical to the
// scalar loop.
template <int E>
__device__ __forceinline__ void warp_fwht(float (&v)[E], int lane) {
#pragma unroll
    for (int h = 1; h < E; h <<= 1) {
#pragma unroll
        for (int i = 0; i < E; i += 2 * h) {
#pragma unroll
            for (int j = i; j < i + h; ++j) {
                float a = v[j], b = v[j + h];
                v[j] = __fadd_rn(a, b);
                v[j + h] = __fsub_rn(a, b);
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        // lower lane: mine + other; upper lane: other - mine  (a is the lower index)
        const float side = (lane & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = __fmaf_rn(v[j], side, __shfl_xor_sync(0xffffffffu, v[j], m));
    }
}

// Two fp32 numbers in a register pair: one instruction for both, each rounded as on its own.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// E consecutive values of a lane, in 16-byte accesses where `wide` (all addresses are multiples of 16 bytes then).
template <int E>
__device__ __forceinline__ void load_lane(float (&v)[E], const float* __restrict__ p, bool wide) {
    if constexpr (E % 4 == 0) {
        if (wide) {
#pragma unroll
            for (int j = 0; j < E; j += 4) {
                const float4 t = *reinterpret_cast<const float4*>(p + j);
                v[j] = t.x; v[j + 1] = t.y; v[j + 2] = t.z; v[j + 3] = t.w;
            }
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = p[j];
}
template <int E>
__device__ __forceinline__ void store_lane(float* __restrict__ p, const float (&v)[E], bool wide) {
    if constexpr (E % 4 == 0) {
        if (wide) {
#pragma unroll
            for (int j = 0; j < E; j += 4) *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < E; ++j) p[j] = v[j];
}

// Number of the sorted boundaries below v, as std::lower_bound finds it: `b` holds 31 (more than 15: `five`) or 15 of
// them, +infinity where there are fewer.
__device__ __forceinline__ int bin_of_sorted(float v, const float* b, bool five) {
    int i = 0;
    if (five && b[15] < v) i = 16;
    if (b[i + 7] < v) i += 8;
    if (b[i + 3] < v) i += 4;
    if (b[i + 1] < v) i += 2;
    if (b[i] < v) i += 1;
    return i;
}

__host__ __device__ __forceinline__ bool is_pow2(uint32_t v) { return v && !(v & (v - 1)); }

// ---- layout of the weight codes in HBM ------------------------------------------------
// One "joint" byte per weight, stored in tiles of 16 rows x 64 columns (1 KB, rows of a tile
// contiguous, 64 bytes each); tiles are row-major over the matrix, and the matrix is padded with
// zero bytes to whole tiles.  A warp of the decode kernel reads 16 rows x 16 bytes per load: in
// this order that is 2 x 512 contiguous bytes instead of 16 pieces of 64; a row's 64 columns of
// one tile stay contiguous for the row-wise readers (dequantiser, prefill GEMM).
constexpr int kCodeTileRows = 16, kCodeTileCols = 64, kCodeTileBytes = kCodeTileRows * kCodeTileCols;
__host__ __device__ __forceinline__ size_t code_tiles_per_row(int in) { return (static_cast<size_t>(in) + kCodeTileCols - 1) / kCodeTileCols; }
__host__ __device__ __forceinline__ size_t code_bytes(long out, int in) {
    return (static_cast<size_t>(out) + kCodeTileRows - 1) / kCodeTileRows * code_tiles_per_row(in) * kCodeTileBytes;
}
// Byte offset of (row, col); `tiles_per_row` = code_tiles_per_row(in).
__host__ __device__ __forceinline__ size_t code_offset(long row, int col, size_t tiles_per_row) {
    return ((static_cast<size_t>(row) >> 4) * tiles_per_row + (static_cast<size_t>(col) >> 6)) * kCodeTileBytes +
           (static_cast<size_t>(row) & 15) * kCodeTileCols + (static_cast<size_t>(col) & 63);
}

// Report a failure from a kernel.  The status word may live in page-locked HOST memory (so that
// the host reads it without a copy): a plain store followed by a system-scope fence, no atomic.
// Programmatic dependent launch for the small kernels of a decode step: launched with the attribute, a kernel's CTAs are
// set up while the kernel before it is still draining; they wait here until that kernel has completed (and its
// writes are visible) before they touch anything, and let the kernel after them start setting up in turn.
__device__ __forceinline__ void pdl_wait_release() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}
// Pointers to what kernels in front write, taken up behind the wait.  A load through a const __restrict__ pointer, and any __ldg, is one of memory that
// nothing writes while the kernel runs: the compiler may carry it out in front of the wait, and did (the rotation of blocks of 512 read its
// activation before the kernel in front had written it).  A pointer that comes out of here is nothing the compiler knows, from a place that it does
// not move: plain loads through it stay behind.
template <typename... Pointer>
__device__ __forceinline__ void behind_wait(Pointer&... p) {
    (..., [&] { asm volatile("" : "+l"(p)::"memory"); }());
}
// `carveout`: how much of the SM's memory is to be shared memory while this kernel runs, in percent (0: the driver's choice).  An SM has one division at a
// time and changes it only when it is empty: kernels that are to overlap ask for the same one.
template <typename Kernel, typename... Args>
inline void launch_pdl_carved(Kernel kernel, dim3 grid, dim3 block, size_t smem, int carveout, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = static_cast<unsigned int>(carveout);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = carveout > 0 ? 2 : 1;
    TQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}
template <typename Kernel, typename... Args>
inline void launch_pdl(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    launch_pdl_carved(kernel, grid, block, smem, 0, stream, args...);
}

// Up to 8 halves (n, even, at least 4-byte aligned) from or to memory, 16 bytes at once where they are all there and aligned;
// missing ones read as zero.
__device__ __forceinline__ uint4 load_halves(const __half* p, int n) {
    if (n >= 8 && reinterpret_cast<uintptr_t>(p) % 16 == 0) return *reinterpret_cast<const uint4*>(p);
    const uint32_t* const w = reinterpret_cast<const uint32_t*>(p);
    return make_uint4(n > 0 ? w[0] : 0u, n > 2 ? w[1] : 0u, n > 4 ? w[2] : 0u, n > 6 ? w[3] : 0u);
}
__device__ __forceinline__ void store_halves(__half* p, int n, const uint4& v) {
    if (n >= 8 && reinterpret_cast<uintptr_t>(p) % 16 == 0) {
        *reinterpret_cast<uint4*>(p) = v;
        return;
    }
    uint32_t* const w = reinterpret_cast<uint32_t*>(p);
    if (n > 0) w[0] = v.x;
    if (n > 2) w[1] = v.y;
    if (n > 4) w[2] = v.z;
    if (n > 6) w[3] = v.w;
}
__device__ __forceinline__ void unpack_halves(const uint4& raw, float (&v)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        v[2 * j] = f.x;
        v[2 * j + 1] = f.y;
    }
}
__device__ __forceinline__ uint4 pack_halves(const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Signs of eight columns of a WHT block, `col` and on, as the sign bits of their halves.
__device__ __forceinline__ uint4 chunk_signs(uint32_t seed, uint32_t col, int block) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        w[j] = (sign_is_positive(seed, (col + 2 * j) & static_cast<uint32_t>(block - 1)) ? 0u : 0x8000u) |
               (sign_is_positive(seed, (col + 2 * j + 1) & static_cast<uint32_t>(block - 1)) ? 0u : 0x80000000u);
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// The butterfly stages of a WHT block that a warp holds in chunks of 256 columns, lane l the columns 8 l .. 8 l + 7 of
// each: signs, the stages below 8 in the lane and those of 8 .. 128 (as far as the block goes) between lanes, in the order
// and pairing of warp_fwht.  The stages above 128 are the caller's, between chunks.
__device__ __forceinline__ void rotate_chunk(float (&v)[8], const uint4& raw, const uint4& signs, int block, int lane, unsigned live) {
    unpack_halves(make_uint4(raw.x ^ signs.x, raw.y ^ signs.y, raw.z ^ signs.z, raw.w ^ signs.w), v);
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
    const int lanes = block < 256 ? block >> 3 : 32;
    for (int m = 1; m < lanes; m <<= 1) {
        const float side = (lane & m) != 0 ? -1.0f : 1.0f;   // other + v or other - v, one exact multiply-add
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __fmaf_rn(v[j], side, __shfl_xor_sync(live, v[j], m));
    }
}
// The same with the number of lane exchanges known and their signs at hand (side[k]: -1 where bit k of the lane is set): half of the
// instructions where many rows follow one another.
template <int STAGES>
__device__ __forceinline__ void rotate_chunk_fixed(float (&v)[8], const uint4& raw, const uint4& signs, const float (&side)[STAGES], unsigned live) {
    unpack_halves(make_uint4(raw.x ^ signs.x, raw.y ^ signs.y, raw.z ^ signs.z, raw.w ^ signs.w), v);
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
#pragma unroll
    for (int k = 0; k < STAGES; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __fmaf_rn(v[j], side[k], __shfl_xor_sync(live, v[j], 1 << k));
}

// Threads of a CTA that normalises a row (the RMSNorm kernel and the row-wise all-reduce tails: the same count, so the same
// order of additions).  Eight columns per thread and step: 256 threads take 8192 columns in the four steps that stay in
// registers, and four to eight rows run on an SM at a time (with 1024 threads and two columns per step a row's barriers and
// reduction were most of its time).
constexpr int kRowNormThreads = 256;
constexpr int kRowNormKeep = 4;

// Eight halves of a row; WIDE: all rows are multiples of eight and 16-byte aligned.
template <bool WIDE>
__device__ __forceinline__ uint4 load_row8(const __half* p, int n) {
    if constexpr (WIDE) return *reinterpret_cast<const uint4*>(p);
    else return load_halves(p, n);
}
template <bool WIDE>
__device__ __forceinline__ void store_row8(__half* p, int n, const uint4& v) {
    if constexpr (WIDE) *reinterpret_cast<uint4*>(p) = v;
    else store_halves(p, n, v);
}
__host__ __device__ __forceinline__ bool rows_wide(int cols, const void* a, const void* b, const void* c) {
    return cols % 8 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}
// KEEP: the steps of a row that stay in registers, as many as its columns need, at most kRowNormKeep; kRowNormMore: so many, and others that are
// read twice.  Fewer leave room for more CTAs on an SM, which is what many rows are bound by (row_ctas; 0: the plain sum): with registers for
// four steps whatever the columns, and three CTAs, 512 x 1024 took 2.3 us and the sum of two slots with it 3.5, 1.6 and 2.3 so; 2048 x 3584 6.2 and 11.3, 4.5
// and 7.4.  Rows that are not whole 16-byte pieces keep four steps and ask for the weights late, as many registers as that takes.
constexpr int kRowNormMore = kRowNormKeep + 1;
constexpr int row_ctas(int keep) { return keep == 0 ? 8 : keep == 1 ? 6 : keep == 2 ? 5 : 4; }
#define TQ_ROW_KERNEL(K, KERNEL, WIDE, COLS)                                                        \
    K = KERNEL<false, kRowNormMore>;                                                                \
    if (WIDE) K = (COLS) <= 8 * kRowNormThreads ? KERNEL<true, 1>                                   \
                  : (COLS) <= 16 * kRowNormThreads ? KERNEL<true, 2>                                \
                  : (COLS) <= 8 * kRowNormKeep * kRowNormThreads ? KERNEL<true, kRowNormKeep> : KERNEL<true, kRowNormMore>;

// yr[:] = xr[:] * rsqrt(mean(xr[:]^2) + eps) * w for one row, by the whole CTA (kRowNormThreads threads; cols even).  A
// thread takes the columns 8 (threadIdx.x + k * kRowNormThreads) .. + 7, whatever the alignment, the first KEEP
// steps of them in `keep`; the others (MORE) are read from xr.  Shared by the RMSNorm kernel and the all-reduce tails that
// normalise the row they have just summed, so the fused and the separate form give the same bits.  WIDE: the weights are asked for
// in front of the sum of squares, whose barrier they would otherwise be waited for behind.
template <bool WIDE, bool MORE, int KEEP>
__device__ __forceinline__ void rmsnorm_kept(const uint4 (&keep)[KEEP], const __half* xr, const __half* __restrict__ w, __half* yr, int cols, float eps) {
    constexpr int kStep = 8 * kRowNormThreads;
    const int c0 = threadIdx.x * 8;
    uint4 gain[KEEP];
    if constexpr (WIDE) {
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
            gain[k] = c0 + k * kStep < cols ? load_row8<WIDE>(w + c0 + k * kStep, 8) : make_uint4(0u, 0u, 0u, 0u);
    }
    float ss = 0.f;
    auto add = [&](const uint4& raw) {
        float v[8];
        unpack_halves(raw, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
    };
#pragma unroll
    for (int k = 0; k < KEEP; ++k) add(keep[k]);   // (zero beyond the row)
    if constexpr (MORE)
        for (int c = c0 + KEEP * kStep; c < cols; c += kStep) add(load_row8<WIDE>(xr + c, cols - c));
    __shared__ float s_part[kRowNormThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < kRowNormThreads / 32; ++i) tot += s_part[i];   // fixed order
    const float scale = rsqrtf(tot / static_cast<float>(cols) + eps);
    auto write = [&](int c, const uint4& raw, const uint4& weight) {
        float v[8], g[8];
        unpack_halves(raw, v);
        unpack_halves(weight, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = v[j] * scale * g[j];
        store_row8<WIDE>(yr + c, cols - c, pack_halves(v));
    };
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const int c = c0 + k * kStep;
        if (c < cols) write(c, keep[k], WIDE ? gain[k] : load_row8<WIDE>(w + c, cols - c));
    }
    if constexpr (MORE)
        for (int c = c0 + KEEP * kStep; c < cols; c += kStep) write(c, load_row8<WIDE>(xr + c, cols - c), load_row8<WIDE>(w + c, cols - c));
}
template <bool WIDE, int KEEP>
__device__ __forceinline__ void rmsnorm_row(const __half* xr, const __half* __restrict__ w, __half* yr, int cols, float eps) {
    constexpr int kKeep = KEEP < kRowNormMore ? KEEP : kRowNormKeep;
    uint4 keep[kKeep];
#pragma unroll
    for (int k = 0; k < kKeep; ++k) {
        const int c = 8 * (threadIdx.x + k * kRowNormThreads);
        keep[k] = c < cols ? load_row8<WIDE>(xr + c, cols - c) : make_uint4(0u, 0u, 0u, 0u);
    }
    rmsnorm_kept<WIDE, KEEP == kRowNormMore>(keep, xr, w, yr, cols, eps);
}

__device__ __forceinline__ void raise_status(unsigned int* status, unsigned int code) {
    *reinterpret_cast<volatile unsigned int*>(status) = code;
    __threadfence_system();
}

}  // namespace tq
