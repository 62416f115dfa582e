// Fused TQ8 dequantise + GEMV / skinny GEMM for decode (1..8 activation rows per pass).
//
// Replaces the reference's tq_dequant_mm Metal kernel and its host wrapper
// (metal/turboquant_dequant_mm.metal:152-313, src/dequantizer.cpp:606-721):
//   y[b, r] = fp16( norm[r] * sum_j W~[r, j] * fp16(x[b, j]) ),  fp32 accumulate.
//
// Algebra.  A dequantised row block is  norm * (inv_sqrt*sign) o H(table[codes]*inv_scale)
// and H is symmetric, so   <s o H(c), x> = <c, H(s o x)>.   The activation is therefore
// rotated ONCE per call (forward WHT of every block of x) and the weight side collapses
// to a table lookup per code:
//   y[b, r] = norm[r] * inv_scale * sum_j table[code[r, j]] * xrot[b, j].
//
// Where the rotation happens.  A warp multiplies a fixed 256-column slice, so for WHT
// blocks of up to 256 columns it rotates its own slice of x inside the GEMV kernel (16-byte
// loads, butterflies in registers and lane exchanges, a 1 KB strip of shared memory to reach
// the fragment layout): one kernel per call.  Larger blocks span several warps; for those
// rotate_x_kernel writes xrot (fp32, TF32-rounded, [b, in]) to scratch first, chained with
// programmatic dependent launch.  Either way the GEMV is launched with the programmatic
// attribute: its set-up (table, first code loads) overlaps the tail of whatever precedes it.
//   tq8_gemv_kernel   persistent, one CTA per SM, 16 warps:
//     HBM --(128-bit loads, 16 codes each, two 64-column steps ahead)--> registers
//     --(byte -> address, 1 PRMT)-->
//     shared-memory table (lane-private columns: bank-conflict free by construction)
//     --> TF32 A fragments --> mma.sync m16n8k8 against xrot held in registers as B
//     fragments --> fp32 accumulators --> cross-warp sum in shared memory --> y.
//   The table value a thread fetches IS its A-fragment register, so a weight costs one
//   integer op and one shared load; multiply-adds and the row reduction ride on the
//   tensor pipe.  Roofline: HBM; 1 B per weight + 4 B per row (norm).
//
// Shared-memory table.  256 entries, entry stride 256 B, 32 fp32 copies per entry (one
// per lane), placed at the fixed shared-window address 0x10000 so that the address of
// copy `lane` of entry `code` is a pure byte permutation of (code word, per-lane
// constant): no shift, mask or add.
//
// Work split.  The 16 warps of a CTA are split into groups of wpt warps (a power of two); a group multiplies one
// 16-row tile against a chunk of wpt * 256 columns, so a unit is 16 / wpt row tiles of one chunk (a "slot").  Up to
// 4096 columns there is one chunk and wpt is the fewest warps that cover the row; above, wpt = 16 unless the last
// chunk would leave more than 15 % of the slices empty (5120 columns: five chunks of 1024 with wpt = 4).  Units are
// ordered slot-major and dealt to CTAs in contiguous ranges, so a CTA reloads its B fragments only when its slot
// changes.  A warp's partial tiles are added across the group through a ring in shared memory, one pass of
// log2(wpt) lane exchanges per unit.  With more than one slot (in_features > 4096, or dual rotation) the sums go
// to scratch as fp32; every warp owns the same rows in every slot and counts its arrivals per (row unit, warp) -
// once per 8 units, since the fence before the count stalls the warp - and the warp that completes a row unit adds
// the slots' partial sums in slot order (a fixed order, so results do not depend on scheduling), applies
// norm*inv_scale and writes fp16.
// Dual-rotation weights (separate sign seeds for the primary and residual planes,
// src/dequantizer.cpp:214-246): the activation is rotated with either seed, and a weight is the pair (primary centroid,
// residual centroid) against the pair of rotated values.  A table word holds the pair as two fp16 numbers, and so does a
// word of the activation: one lookup fetches both, and an m16n8k16 product takes eight columns of both planes where the
// single-rotation kernel's m16n8k8 takes eight columns of one; everything else is the same.  (As further partial-sum slots
// the planes took two lookups and a pass each: 3584 x 3584, block 512, 16.5 us at one row, 19.2 at four, 20.9 at eight; as
// pairs 8.4, 11.0 and 12.7.)  fp16 has the ten mantissa bits of TF32, and powers of two bring its range to the values: one for the
// table (its largest entry lies in [2^14, 2^15)) and one for every 256 columns of a rotated row, which rotate_x_pair_kernel
// finds.  The operands are the TF32 numbers they were; what falls below fp16's normal numbers is 2^-28 of the largest beside it.
// Relative error against 64-bit products, 12 draws of 8 rows: 3.772e-4 / 3.772e-4 (3584 columns), 3.633e-4 / 3.633e-4 (18944).
#include <cmath>
#include <cstdint>

#include <cstring>

#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kSlice = 256;               // columns per warp
constexpr uint32_t kLutAddr = 0x10000u;   // shared-window address of the table
constexpr uint32_t kLutBytes = 0x10000u;  // 256 entries * 256 B
// Partial-sum ring: ring * 16 warps * (16 rows * bp + 4) floats.  Eight rows take three slots of 32 KB, which tied the warps to each
// other's pace: seven of 60 KB, 151936 x 2048 75.4 -> 73.9 us, 37888 x 3584 41.1 -> 40.1.  (Fewer rows have seven to sixteen slots as it is, and
// gained nothing from more.  With two rotations a unit takes longer, the sums keep up, and those of the last units, three behind instead of one, come at the
// end: five rows, 11008 x 4096 17.1 us with three slots, 18.5 with seven, 14336 x 4096 21.6 and 22.6, 18944 x 3584 24.7 and 25.3.)
__host__ __device__ constexpr int red_bytes(int bp, bool dual) { return bp == 8 && !dual ? 61440 : 32768; }
constexpr int kMaxRing = 16;
constexpr int kFlushUnits = 8;             // units a warp finishes between two arrival counts (several slots only)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void sts_f32(uint32_t addr, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void sts_v4(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ float to_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}
// Wait for the kernel launched before this one in the stream (no-op without the
// programmatic-serialization launch attribute).
__device__ __forceinline__ void grid_dependency_sync() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Allow the next kernel in the stream to start launching.
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }

// Address of this lane's copy of the table entry selected by byte BYTE of `word`:
//   result byte 0 = lane constant byte 0 (copy offset), byte 1 = the code,
//   bytes 2,3 = lane constant bytes 2,3 (0x0001 -> the 0x10000 base).
template <int BYTE>
__device__ __forceinline__ uint32_t lut_addr(uint32_t word, uint32_t lane_const) {
    return __byte_perm(word, lane_const, 0x7604u | (static_cast<uint32_t>(BYTE) << 4));
}

// ---- activation rotation ---------------------------------------------------------------------
// Where word (row, col) of a rotated activation stands when the decode kernel is to read it: in the order of its B fragments, bp the rows rounded
// up to 1, 4 or 8.  A product takes two columns (2 m and the next) of every 16-column group q of a 64-column block; its eight B columns are
// the bp rows for 8 / bp products m side by side (m = (8 / bp) jj + m', B column g = m' bp + row).  So lane (g, q) has 2 bp words of a block, words 2 jj and the next, and
// they come in pieces of four (two with one row), a piece of all lanes side by side.  Row after row, the 16 bytes of every lane lay in a line of their own, and
// every CTA spent more time on its 128 KB of activations than on a unit of codes: 4096 x 4096 at eight rows 9.6 -> 8.2 us, 3584 x 3584 with two
// rotations at eight 12.0 -> 9.4, 18944 x 3584 at four 24.5 -> 23.7, 27648 x 5120 at eight 46.2 -> 44.3.  (in is a multiple of 32: a last block of 32 columns has two groups q.)
__host__ __device__ __forceinline__ int fragment_groups(int in, int col) {
    const int left = (in - (col & ~63)) >> 4;
    return left < 4 ? left : 4;
}
__host__ __device__ __forceinline__ int row_bits(int bp) { return bp >= 8 ? 3 : bp >> 1; }   // log2
__host__ __device__ __forceinline__ size_t fragment_place(int in, int bp, int row, int col) {
    const int m = (col & 15) >> 1, jj = m >> (3 - row_bits(bp)), g = ((m & (8 / bp - 1)) << row_bits(bp)) + row, r = 2 * jj + (col & 1);
    const int groups = fragment_groups(in, col), lane = g * groups + ((col & 63) >> 4);
    return static_cast<size_t>(col >> 6) * (64 * bp) + static_cast<size_t>(bp == 1 ? 2 * lane + r : ((r >> 2) * 8 * groups + lane) * 4 + (r & 3));
}
// Of the fragments; two rows have those of four (with four products side by side 2048 x 151936 took 81 us instead of 67), and sums of their own (BP).
__host__ __device__ __forceinline__ constexpr int padded_rows(int batch) { return batch <= 1 ? 1 : batch <= 4 ? 4 : 8; }
// One warp per (plane, batch row, WHT block): xrot = FWHT(sign o x) / sqrt(bs), rounded to
// TF32 and stored as fp32, [plane][row][in] or (fragments: the padded rows; one plane) in the decode kernel's order.
template <int E>
__global__ void __launch_bounds__(128) rotate_x_kernel(const __half* __restrict__ x, float* __restrict__ xrot, int in,
                                                       int batch, int n_planes, uint32_t seed_p, uint32_t seed_r,
                                                       float inv_sqrt, int fragments) {
    // Let the GEMV that follows start its set-up right away; it waits for this grid to
    // finish before it reads xrot.
    grid_launch_dependents();
    // x (and the scratch this kernel overwrites) may still be in use by the previous kernel.
    grid_dependency_sync();
    constexpr int BS = 32 * E;
    const int lane = threadIdx.x & 31;
    const int blocks_per_row = in / BS;
    const int total = n_planes * batch * blocks_per_row;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= total) return;
    const int plane = warp / (batch * blocks_per_row);
    const int rem = warp - plane * batch * blocks_per_row;
    const int row = rem / blocks_per_row, blk = rem - row * blocks_per_row;
    const uint32_t seed = plane ? seed_r : seed_p;
    behind_wait(x);
    const __half* src = x + static_cast<size_t>(row) * in + blk * BS + lane * E;
    float v[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = __half2float(src[j]) * sign_value(seed, static_cast<uint32_t>(lane * E + j));
    warp_fwht<E>(v, lane);
    const int col = blk * BS + lane * E;
    float* const dst = xrot + (static_cast<size_t>(plane) * batch + row) * in + col;
#pragma unroll
    for (int j = 0; j < E; ++j) *(fragments ? xrot + fragment_place(in, fragments, row, col + j) : dst + j) = to_tf32(v[j] * inv_sqrt);
}

// The same with 16-byte accesses: a warp takes CHUNKS x 256 columns of a row (a WHT block of 512 or 1024 columns, or the
// smaller blocks of 256 columns).  A lane of the kernel above reads E consecutive halves, 2 bytes at a time: 2 E accesses of
// up to 32 lines each, and as all of its few CTAs land on the first SM that the kernel before it leaves (no other has room
// yet), they serialised there: 13 us of the 31 us of a 3584 x 3584 layer with two rotations, block 512 and 4 rows.  For the
// same reason the launch asks for shared memory it does not use: four CTAs per SM.
template <int CHUNKS>
__global__ void __launch_bounds__(128) rotate_x_wide_kernel(const __half* __restrict__ x, float* __restrict__ xrot, int in, int batch,
                                                            int n_planes, int block, uint32_t seed_p, uint32_t seed_r, float inv_sqrt, int fragments) {
    grid_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int groups_per_row = (in + 256 * CHUNKS - 1) / (256 * CHUNKS);
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= n_planes * batch * groups_per_row) return;
    const int plane = warp / (batch * groups_per_row);
    const int rem = warp - plane * batch * groups_per_row;
    const int row = rem / groups_per_row, col = (rem - row * groups_per_row) * 256 * CHUNKS + 8 * lane;
    const unsigned live = __ballot_sync(0xffffffffu, col < in);   // the lanes that exchange values
    if (col >= in) return;   // a trailing group of less than 256 columns: whole WHT blocks, whole lanes
    const uint32_t seed = plane ? seed_r : seed_p;
    // The signs of one chunk in front of the wait: 4096 x 4096 at eight rows 9.9 -> 9.6 us with the product.  Those of two or four take longer than
    // the loads, behind which they are made: in front, 4096 x 4096, block 512, took 8.8 us at one row instead of 8.3, 1024 x 1024 6.4 instead of 5.9.
    uint4 signs;
    if (CHUNKS == 1) signs = chunk_signs(seed, static_cast<uint32_t>(col), block);
    // A lane's eight columns go out in pairs, 256 columns on at 256 words a row.  (Their places in front of the wait, those of several chunks beside the
    // loads, like the signs: 4096 x 4096, block 512, one row 8.2 us, in front 8.5.)
    float* dst[4];
    const int chunk = fragments ? 256 * fragments : 256;
    auto find_place = [&] {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            dst[i] = xrot + (fragments ? fragment_place(in, fragments, row, col + 2 * i) : (static_cast<size_t>(plane) * batch + row) * in + col + 2 * i);
    };
    if (CHUNKS == 1) find_place();
    grid_dependency_sync();
    behind_wait(x);
    const __half* const src = x + static_cast<size_t>(row) * in + col;
    uint4 raw[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) raw[c] = *reinterpret_cast<const uint4*>(src + 256 * c);
    if (CHUNKS > 1) find_place();
    float v[CHUNKS][8];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        if (CHUNKS > 1) signs = chunk_signs(seed, static_cast<uint32_t>(col + 256 * c), block);
        rotate_chunk(v[c], raw[c], signs, block, lane, live);
    }
#pragma unroll
    for (int h = 1; h < CHUNKS; h <<= 1)
#pragma unroll
        for (int i = 0; i < CHUNKS; i += 2 * h)
#pragma unroll
            for (int c = i; c < i + h; ++c)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float a = v[c][j], b = v[c + h][j];
                    v[c][j] = __fadd_rn(a, b);
                    v[c + h][j] = __fsub_rn(a, b);
                }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float2*>(dst[i] + c * chunk) = make_float2(to_tf32(v[c][2 * i] * inv_sqrt), to_tf32(v[c][2 * i + 1] * inv_sqrt));
}
constexpr size_t kRotateXSmem = 48 * 1024, kRotatePairSmem = 38 * 1024;

// The activation of weights with two rotations: two warps rotate CHUNKS x 256 columns of a row, each with one of the seeds, and write pairs
// of fp16 (primary, residual) in the order of the decode kernel's fragments, each 256 columns times a power of two that brings the largest value of the
// two to [2^14, 2^15), and that power's inverse to xscale[row][columns / 256].  A row that is not 16-byte aligned (`aligned` = 0) is
// read in halves: 2 KB at most per warp.
// The decode kernel waits for the end of this one, few warps alone on their SMs: what counts is the instructions of a warp behind its wait.  So the
// signs are in hand before it, and a warp has one seed, not both: 1.6 us from the wait to the end at four rows of 3584 columns in blocks of 512, 3 to 3.8 with
// both seeds in a warp and the signs behind the wait (3584 x 3584 8.8 -> 8.4, with the order of the fragments 9.7 -> 8.4; eight rows 12.0 -> 8.7).
template <int CHUNKS>
__global__ void __launch_bounds__(128) rotate_x_pair_kernel(const __half* __restrict__ x, uint32_t* __restrict__ pairs, float* __restrict__ xscale,
                                                            int in, int batch, int block, uint32_t seed_p, uint32_t seed_r, float inv_sqrt,
                                                            int aligned) {
    grid_launch_dependents();
    __shared__ __align__(16) float4 s_give[4][CHUNKS][32];   // the half of a lane's columns that the other warp writes
    __shared__ unsigned int s_top[4][CHUNKS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, plane = wib & 1;
    const int slices = (in + kSlice - 1) / kSlice, groups_per_row = (in + 256 * CHUNKS - 1) / (256 * CHUNKS);
    const int item = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 6);
    const int row = item / groups_per_row, col = (item - row * groups_per_row) * 256 * CHUNKS + 8 * lane;
    const bool have = row < batch && col < in;   // (a trailing group of less than 256 columns: whole WHT blocks, whole lanes)
    const unsigned live = __ballot_sync(0xffffffffu, have);   // the lanes that exchange values
    uint4 signs[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) signs[c] = chunk_signs(plane ? seed_r : seed_p, static_cast<uint32_t>(col + 256 * c), block);
    uint32_t* dst[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) dst[i] = pairs + fragment_place(in, padded_rows(batch), row, col + 4 * plane + 2 * i);
    const int chunk = 256 * padded_rows(batch);
    grid_dependency_sync();
    behind_wait(x);
    float v[CHUNKS][8];
    if (have) {
        const __half* const src = x + static_cast<size_t>(row) * in + col;
        uint4 raw[CHUNKS];
        if (aligned) {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) raw[c] = *reinterpret_cast<const uint4*>(src + 256 * c);
        } else {
            const unsigned short* const h = reinterpret_cast<const unsigned short*>(src);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = h[256 * c + 2 * j] | (static_cast<uint32_t>(h[256 * c + 2 * j + 1]) << 16);
                raw[c] = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) rotate_chunk(v[c], raw[c], signs[c], block, lane, live);
#pragma unroll
        for (int h = 1; h < CHUNKS; h <<= 1)
#pragma unroll
            for (int i = 0; i < CHUNKS; i += 2 * h)
#pragma unroll
                for (int c = i; c < i + h; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float a = v[c][j], b = v[c + h][j];
                        v[c][j] = __fadd_rn(a, b);
                        v[c + h][j] = __fsub_rn(a, b);
                    }
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            unsigned int top = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[c][j] = to_tf32(v[c][j] * inv_sqrt);
                top = max(top, __float_as_uint(v[c][j]) & 0x7fffffffu);
            }
            top = __reduce_max_sync(live, top);
            if (lane == 0) s_top[wib][c] = top;
            s_give[wib][c][lane] = plane ? make_float4(v[c][0], v[c][1], v[c][2], v[c][3]) : make_float4(v[c][4], v[c][5], v[c][6], v[c][7]);
        }
    }
    __syncthreads();
    if (!have) return;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        // 2^(14 - exponent), between 2^-113 and 2^126 (its inverse is a normal number); 1 beside an infinity or a NaN
        const unsigned int e = max(s_top[wib][c], s_top[wib ^ 1][c]) >> 23;
        const unsigned int f = e == 255u ? 127u : min(268u - e, 253u);
        const float up = __uint_as_float(f << 23);
        const float4 got = s_give[wib ^ 1][c][lane];
        const float other[4] = {got.x, got.y, got.z, got.w};
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // the warp of the primary seed writes the lower four columns, the other the upper four
            const float mine = plane ? v[c][4 + j] : v[c][j];
            const __half2 h = plane ? __floats2half2_rn(other[j] * up, mine * up) : __floats2half2_rn(mine * up, other[j] * up);
            w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<uint2*>(dst[i] + c * chunk) = make_uint2(w[2 * i], w[2 * i + 1]);
        if (lane == 0 && plane == 0) xscale[row * slices + col / kSlice + c] = __uint_as_float((254u - f) << 23);
    }
}

struct GemvArgs {
    const uint8_t* codes;   // joint bytes in 16 x 64 tiles (code_offset)
    const float* norms;     // [out]
    const float* table;     // [256] fp32; two rotations: [256] pairs of fp16
    const float* xrot;      // [batch, in] fp32 (TF32-rounded) in fragment_place order, used when x == nullptr; two rotations: pairs of fp16
    const float* xscale;    // two rotations: [8, ceil(in / 256)] what the pairs of a row's 256 columns are to be multiplied by
    const __half* x;        // [batch, in] fp16: rotate inside the kernel (WHT block <= 256), else nullptr
    __half* y;              // [batch, y_stride]: row r of activation row n at y[n * y_stride + r]
    float* partial;         // [n_slots, 8, out_pad] (only when n_slots > 1)
    unsigned int* counters; // [n_row_units][16 warps] (only when n_slots > 1)
    unsigned int* status;   // device error word (0 = ok)
    int out, in, batch;
    int n_row_units, n_slots, out_pad;  // n_slots = chunks of a row
    int wpt, tpu;           // warps per row tile, row tiles per unit (wpt * tpu = 16)
    float inv_scale;
    uint32_t seed_p;           // sign seed       (in-kernel rotation)
    int block;                 // WHT block size  (in-kernel rotation)
    float inv_sqrt_block;
};

// Arguments of scattering calls, a kernel parameter of their own: with these fields inside
// GemvArgs the plain kernel (same code otherwise) needed spills within its 128 registers.
struct ScatterArgs {
    __half* y_peer[7];      // further destinations written with the same values (other GPUs' buffers)
    int n_peer;
    long y_stride;
    // Completion signal of a scattering call (n_signal = 0: none): when the whole grid has
    // stored its results, word `signal_slot` of every destination's flag array is set to
    // `signal_value`.  done_counter is a zero-initialised device word owned by the layer.
    unsigned int* signal[8];
    int n_signal, signal_slot;
    unsigned int signal_value;
    unsigned int* done_counter;
    // Fused all-gather (bulk != 0): results are stored locally only; the CTA that completes the grid
    // copies the whole block to the peers with 16-byte stores and then raises the flags with the value
    // ++(*epoch) (signal_value is not used).  With n_wait > 0 every CTA first waits - bounded - until
    // wait_flags[0..n_wait) have reached *wait_epoch + 1 before it reads the activation (the previous
    // exchange has arrived); the completing CTA then advances *wait_epoch.
    int bulk;
    unsigned int* epoch;
    const unsigned int* wait_flags;
    int n_wait;
    unsigned int* wait_epoch;
    // Flag-in-data exchange (ll != 0, with bulk): instead of data, a fence and a flag, the completing CTA
    // writes 16-byte packets {2 halves, epoch, 2 halves, epoch} - each 8-byte half is written atomically
    // by the one store, so a reader that sees the epoch in both halves holds valid data and nothing has to
    // be fenced.  Every rank's packet buffer is [2 halves of the double buffer][ll_world source ranks]
    // [packets] (ll_base[r] = rank r's buffer, ll_base[ll_rank] this rank's own); the half is the parity of
    // the epoch.  With n_wait > 0 every CTA first polls - bounded - the packets all other ranks wrote for
    // epoch *wait_epoch + 1.
    int ll, ll_rank, ll_world;
    uint4* ll_base[8];
};

// One output element goes to the caller's buffer and, when the call scatters, to the same
// position of up to 7 further buffers (peer GPUs' memory mapped into this process: plain stores
// over NVLink, no multicast).
// SCATTER is a compile-time variant: the plain kernel keeps the register budget it had before the
// scattering code existed (with it in the same instantiation the kernel spilled).
template <bool SCATTER>
__device__ __forceinline__ void store_y(const GemvArgs& p, const ScatterArgs& sc, int n, int row, __half h) {
    if constexpr (SCATTER) {
        const size_t o = static_cast<size_t>(n) * sc.y_stride + row;
        p.y[o] = h;
        if (!sc.bulk) {
#pragma unroll
            for (int d = 0; d < 7; ++d)
                if (d < sc.n_peer) sc.y_peer[d][o] = h;
        }
    } else {
        p.y[static_cast<size_t>(n) * p.out + row] = h;
    }
}

// Shared memory holds only the table and the partial-sum ring: the dynamic allocation ends at
// the end of the table (128 KB).  Asking for much more than that shrinks the L1 side of the
// SM's memory and with it the number of global loads the SM keeps in flight (measured: a
// streaming read drops from 5.8 to 3.4 TB/s when a CTA holds 216 KB), so the codes are never
// staged through shared memory: they go from HBM straight into registers.
constexpr size_t kGemvSmem = kLutAddr + kLutBytes;  // dynamic bytes requested (window end)
constexpr int kCtaThreads = kThreads;
constexpr unsigned long long kWaitLimitNs = 200ull * 1000 * 1000;  // bounded waits: give up after 0.2 s and flag it

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Returns false if the phase did not complete within the spin limit.
__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (spin == 64) t0 = global_timer_ns();
        if (spin > 64 && (spin & 63) == 0 && global_timer_ns() - t0 > kWaitLimitNs) return false;
    }
}
// Streaming 16-byte load that leaves `v` untouched when `pred` is false.  Codes outside the
// matrix are never zero-filled: whatever the registers hold indexes a valid table entry, and it
// meets either a zero activation (columns past in_features) or a row that is never written.
__device__ __forceinline__ void ldg_stream_if(uint4& v, const uint8_t* p, bool pred) {
    asm volatile(
        "{ .reg .pred p; setp.ne.u32 p, %5, 0;\n"
        "  @p ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4]; }"
        : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
        : "l"(p), "r"(static_cast<uint32_t>(pred)));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Table lookup.  Not volatile: the table is read-only while lookups run, so the compiler may
// batch and reorder these loads freely (the address depends on codes loaded after the
// barrier that publishes the table, which keeps them below it).
__device__ __forceinline__ uint32_t lut_load(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- flag-in-data exchange (see ScatterArgs) ----
__device__ __forceinline__ void ll_wait_packets(const unsigned int* wait_epoch, const uint4* mine, int rank, int world, long packets,
                                                unsigned int* status) {
    const unsigned int want = *reinterpret_cast<const volatile unsigned int*>(wait_epoch) + 1u;
    const uint4* const half = mine + static_cast<size_t>(want & 1u) * world * packets;
    const unsigned long long t0 = global_timer_ns();
    for (int src = 0; src < world; ++src) {
        if (src == rank) continue;
        const uint4* region = half + static_cast<size_t>(src) * packets;
        for (long i = threadIdx.x; i < packets; i += kCtaThreads) {
            for (unsigned int spin = 0;; ++spin) {
                uint4 pk;
                asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(pk.x), "=r"(pk.y), "=r"(pk.z), "=r"(pk.w)
                             : "l"(region + i)
                             : "memory");
                if (static_cast<int>(pk.y - want) >= 0 && static_cast<int>(pk.w - want) >= 0) break;
                if ((spin & 255u) == 255u && global_timer_ns() - t0 > 5ull * kWaitLimitNs) {   // 1 s: a peer is gone
                    raise_status(status, 10u);
                    return;
                }
            }
        }
    }
}
// Packets c0 .. c1 - 1 (groups of four rows) of every activation row, to every other rank: no fence, no flag -
// the epoch travels with the data.
__device__ __forceinline__ void ll_send_packets(const ScatterArgs& sc, const __half* y, int per_row, int batch, int c0, int c1) {
    const unsigned int value = *reinterpret_cast<const volatile unsigned int*>(sc.epoch) + 1u;
    const long packets = static_cast<long>(batch) * per_row;
    const size_t region = (static_cast<size_t>(value & 1u) * sc.ll_world + sc.ll_rank) * packets;
    const int span = c1 - c0;
    for (long i = threadIdx.x; i < static_cast<long>(batch) * span; i += kCtaThreads) {
        const int n = static_cast<int>(i / span), c = c0 + static_cast<int>(i - static_cast<long>(n) * span);
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(y + static_cast<size_t>(n) * sc.y_stride + static_cast<size_t>(c) * 4));
        const size_t at = region + static_cast<size_t>(n) * per_row + c;
#pragma unroll
        for (int d = 0; d < 8; ++d)
            if (d < sc.ll_world && d != sc.ll_rank)
                asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(sc.ll_base[d] + at), "r"(v.x), "r"(value), "r"(v.y)
                             : "memory");
    }
}

// BP = activation rows padded to 1, 2, 4 or 8 (compile time, so that the partial-sum ring
// geometry and the reduction need no runtime arithmetic).
// MULTI = more than one slot (row units finished through partial sums in scratch); compile time, so that the
// single-slot kernels carry none of that path's state in their 128 registers.
// DUAL = weights with two rotations: table words and activation words are pairs of fp16.
// ROW = the activation row is a kernel parameter, `row` its generic address.
// DEEP = all four steps of a unit's codes in registers, not two (one activation row, many units a CTA).
// AT_FIRST = a new slot is known by its first row unit, not by a number that is kept: a register less, which eight rows of two rotations in several slots turn into
// more lookups in flight (5120 x 27648 at eight rows 53.9 -> 51.2 us, 18944 x 3584 30.8 -> 29.7, 14336 x 4096 27.7 -> 26.8).  The other kernels spill with it (the group's of the same
// rows: twice 5120 x 27648 94 -> 117; one row, four steps: 5120 x 27648 38.6 -> 39.4).
template <int BP, bool SCATTER, bool LL, bool MULTI, bool DUAL, bool ROW = false, bool DEEP = false, bool AT_FIRST = false>
__device__ __forceinline__ void gemv_body(const GemvArgs& p, const ScatterArgs& sargs, const int bid, const int nblk, const __half* row = nullptr) {
    auto load_x = [&](int col) {   // eight columns of the row that is rotated in here
        if constexpr (ROW) return *reinterpret_cast<const uint4*>(row + col);
        else return *reinterpret_cast<const uint4*>(p.x + col);   // (no __ldg: it must stay behind the wait)
    };
    // columns per chunk, derived here: one more field in GemvArgs made ptxas spill within the 128 registers
    const int chunk_cols = p.wpt * kSlice;
    // A warp's partial tile is [16 rows][BP] floats plus 4 floats of padding: the 16 tiles a
    // reduction reads side by side then start 4 banks apart instead of in the same bank.
    constexpr int kTileFloats = 16 * BP + 4;
    constexpr int kRedBytes = red_bytes(BP, DUAL);
    constexpr int kRing = (kRedBytes / (kWarps * kTileFloats * 4)) > kMaxRing ? kMaxRing : (kRedBytes / (kWarps * kTileFloats * 4));
    static_assert(kRing >= 2, "the ring needs a slot to write while another is summed");
    constexpr int kLag = kRing / 2;                       // how many units behind the sums run
    constexpr uint32_t kSlotBytes = kWarps * kTileFloats * 4;  // one ring slot: [warp][16 rows][BP] floats (+ padding)
    constexpr int kPer = BP >= 2 ? BP / 2 : 1;            // floats a lane adds in the reduction
    constexpr int kFrag = padded_rows(BP), kSide = 8 / kFrag, kAcc = kSide < 2 ? 2 : kSide;   // products side by side in the B columns; accumulators
    constexpr int kSteps = DEEP ? 4 : 2;                  // steps of codes in registers

    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ unsigned int s_abort;
    // [0..kRing) "tiles of ring slot written" (one arrival per warp), [kMaxRing..) "slot read"
    __shared__ __align__(8) unsigned long long s_bars[2 * kMaxRing];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- unit range of this CTA: unit = (slot, row unit), a slot is a chunk of columns ----
    // (the first `rem` CTAs take one unit more; one 32-bit division - the prologue runs once per launch on
    // instructions that are not cached yet, and cannot overlap the preceding kernel, whose CTA fills this SM)
    const int n_units = p.n_row_units * p.n_slots;
    const int u_quot = n_units / nblk, u_rem = n_units - u_quot * nblk;   // bid of nblk CTAs work on this matrix
    const int u_begin = u_quot * bid + (bid < u_rem ? bid : u_rem);
    const int n_local = u_quot + (bid < u_rem ? 1 : 0);
    if (n_local <= 0) return;

    // ---- shared-memory map: [partial-sum ring | rotation strips | unused | table at 0x10000] ----
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t red_addr = (base + 127u) & ~127u;
    const uint32_t strip_addr = red_addr + kRedBytes + static_cast<uint32_t>(warp) * (kSlice * 4u);
    if (red_addr + kRedBytes + (BP == 1 ? kWarps * kSlice * 4u : 0u) > kLutAddr) {  // layout assumption broken: refuse to run
        if (tid == 0) raise_status(p.status, 1u);
        return;
    }
    const uint32_t bar_written = smem_u32(&s_bars[0]), bar_read = smem_u32(&s_bars[kMaxRing]);
    if (tid < kRing) {   // one pair of barriers per thread: a single thread took 0.45 us for the 32 of them
        mbar_init(bar_written + 8u * tid, kWarps);
        mbar_init(bar_read + 8u * tid, kWarps);
        if (tid == 0) s_abort = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    const int g = lane >> 2, q = lane & 3;
    const int wpt_shift = 31 - __clz(p.wpt);                    // wpt is a power of two
    const int tile_in_unit = warp >> wpt_shift;                 // which of the unit's row tiles this warp works on
    const int slice0 = (warp & (p.wpt - 1)) * kSlice;           // column of this warp's slice inside the chunk
    const uint32_t lane_const = 0x00010000u | static_cast<uint32_t>(lane * 4);
    // Codes are stored in 16-row x 64-column tiles of 1 KB (code_offset): a step of a warp is one
    // tile, of which lane (g, q) reads bytes g*64 + 16q (row g) and 512 + g*64 + 16q (row g + 8) -
    // 512 contiguous bytes per warp load.  Consecutive steps are consecutive tiles.
    const size_t tiles_per_row = code_tiles_per_row(p.in);
    const size_t unit_stride = static_cast<size_t>(p.tpu) * tiles_per_row * kCodeTileBytes;  // bytes between consecutive row units

    // ---- position of a unit, kept incrementally (no divisions in the loop) ----
    struct Pos {
        int slot, ru;          // slot and row unit
        const uint8_t* ptr;    // this thread's first 16 codes of the unit (row g)
        uint32_t ok;           // bit s: columns of step s exist; bits 4, 5: the row tile exists (padded rows are stored)
    };
    auto make_pos = [&](int unit) {
        Pos u;
        if constexpr (MULTI) {
            u.slot = unit / p.n_row_units;
            u.ru = unit - u.slot * p.n_row_units;
        } else {
            u.slot = 0;
            u.ru = unit;
        }
        const int c = (MULTI ? u.slot * chunk_cols : 0) + slice0;  // first column of this warp's slice
        const int tile = u.ru * p.tpu + tile_in_unit;
        u.ptr = p.codes + (static_cast<size_t>(tile) * tiles_per_row + static_cast<size_t>(c >> 6)) * kCodeTileBytes + g * 64 + 16 * q;
        u.ok = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) u.ok |= (c + 64 * s < p.in) ? (1u << s) : 0u;
        u.ok |= (tile * 16 < p.out) ? 48u : 0u;
        return u;
    };
    auto next_pos = [&](const Pos& u) {
        Pos n = u;
        if (!MULTI || u.ru + 1 < p.n_row_units) {   // same slot, next row unit: only the rows move
            n.ru = u.ru + 1;
            n.ptr = u.ptr + unit_stride;
            n.ok = (u.ok & 15u) | (((n.ru * p.tpu + tile_in_unit) * 16 < p.out) ? 48u : 0u);
            return n;
        }
        return make_pos((u.slot + 1) * p.n_row_units);
    };
    // Codes never depend on the kernel before this one, so the first loads go out before the
    // dependency wait below.  Pieces outside the matrix are simply not loaded.
    auto load_step = [&](const Pos& u, int s, bool live, uint4& lo, uint4& hi) {
        const bool c_ok = live && ((u.ok >> s) & 1u);
        ldg_stream_if(lo, u.ptr + kCodeTileBytes * s, c_ok && (u.ok & 16u));
        ldg_stream_if(hi, u.ptr + kCodeTileBytes * s + 512, c_ok && (u.ok & 32u));
    };
    Pos cur = make_pos(u_begin);
    Pos nxt = (n_local > 1) ? next_pos(cur) : cur;
    // Two register buffers (even / odd step): two steps, 32 KB per SM, in flight.  (Four for one row and many units a CTA, see the launch; several rows are
    // bound by L1 data-pipe wavefronts, table lookups plus the code loads, and gain nothing from more.)
    uint4 blo[kSteps], bhi[kSteps];
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
        blo[s] = make_uint4(0, 0, 0, 0);
        bhi[s] = make_uint4(0, 0, 0, 0);
        load_step(cur, s, true, blo[s], bhi[s]);
    }

    if constexpr (DUAL) {
        // The rest of this unit and the next one on their way into the L2 cache, a line a lane, while the rotation in front is
        // waited for: 3584 x 3584, four rows, 11.1 -> 9.8 us, one row 9.0 -> 8.2; further units in advance gain no more.  (One row of one
        // rotation is rotated in here, and its loads would queue behind this: 7.5 -> 7.6 for 4096 x 4096 even so late as behind them.)
        auto prefetch = [&](const Pos& u, int first, int steps) {
            const int s = first + (lane >> 3);
            if ((lane >> 3) < steps && ((u.ok >> s) & 1u) && (u.ok & 16u))
                asm volatile("prefetch.global.L2 [%0];" ::"l"(u.ptr - (g * 64 + 16 * q) + kCodeTileBytes * s + 128 * (lane & 7)));
        };
        prefetch(cur, 2, 2);
        if (n_local > 1) prefetch(nxt, 0, 4);
    }

    // Prologue order: table entries are fetched into registers (they do not depend on the
    // preceding kernel), then comes the dependency wait, then this warp's activation slice of
    // the first unit is requested, and only then are the table entries written to shared
    // memory - so the activation's latency hides behind the table build.
    float tab_first[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) tab_first[k] = __ldg(p.table + (tid >> 3) + 64 * k);

    // The signs of a row that is rotated in here (a slice is a multiple of the block: the same for all).  A kernel of two units and more waits long enough to
    // have them first (3584 x 3584 7.3 -> 7.15 us, 5120 x 5120 16.0 -> 15.5); one of a unit follows the kernel before it so soon that they are made while the
    // row's loads are on their way (2048 x 4096 5.5, in front 5.8).
    uint4 row_signs = make_uint4(0, 0, 0, 0);
    constexpr bool kMayRotate = ROW || (BP == 1 && !DUAL);
    if (kMayRotate && n_local > 1) row_signs = chunk_signs(p.seed_p, static_cast<uint32_t>(8 * lane), p.block);

    // Everything below reads or writes data the preceding kernels produce or still use.
    grid_dependency_sync();
    if constexpr (SCATTER) {
        if (LL && sargs.n_wait > 0) {
            // the activation comes out of a flag-in-data exchange: every packet of every other rank must carry the epoch
            if constexpr (LL) {
                ll_wait_packets(sargs.wait_epoch, sargs.ll_base[sargs.ll_rank], sargs.ll_rank, sargs.ll_world,
                                static_cast<long>(p.batch) * (p.out / 4), p.status);
            }
            __syncthreads();
        } else if (sargs.n_wait > 0) {
            // the activation comes out of an exchange: wait until every rank's part has arrived
            if (tid < sargs.n_wait) {
                const unsigned int want = *reinterpret_cast<volatile unsigned int*>(sargs.wait_epoch) + 1u;
                const unsigned long long t0 = global_timer_ns();
                for (unsigned int spin = 0;; ++spin) {
                    unsigned int v;
                    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(sargs.wait_flags + tid) : "memory");
                    if (static_cast<int>(v - want) >= 0) break;
                    if ((spin & 255u) == 255u && global_timer_ns() - t0 > 5ull * kWaitLimitNs) {   // 1 s: a peer is gone
                        raise_status(p.status, 10u);
                        break;
                    }
                }
            }
            __syncthreads();
        }
    }
    uint4 x_first = make_uint4(0, 0, 0, 0);
    if (ROW || (!DUAL && p.x != nullptr)) {
        const int cl0 = (MULTI ? cur.slot * chunk_cols : 0) + slice0 + 8 * lane;
        if (cl0 < p.in) x_first = load_x(cl0);
        if (n_local <= 1) row_signs = chunk_signs(p.seed_p, static_cast<uint32_t>(8 * lane), p.block);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float v = DUAL ? tab_first[k] : to_tf32(tab_first[k]);
        sts_v4(kLutAddr + static_cast<uint32_t>((tid >> 3) + 64 * k) * 256u + static_cast<uint32_t>((tid & 7) * 4) * 4u, v, v, v, v);
    }
    __syncthreads();  // table and barriers visible

    // ---- sum of one unit's per-warp partial tiles ----
    // Ring slot layout: [warp][16 rows][BP] floats (+ 4 floats of padding per warp).  Warp w owns the (tile, row) pairs
    // w*tpu .. w*tpu+tpu-1 of the unit.  The 16 lanes of a half warp cover those tpu pairs times the wpt warps that
    // worked on the pair's row tile (tpu * wpt = 16): lane l reads what warp (l & (wpt - 1)) of the group wrote for pair
    // (l & 15) / wpt, activation columns (l >> 4) * kPer .., and a fixed tree of log2(wpt) lane exchanges adds them
    // (fixed order: results do not depend on timing).  One pass per unit whatever the split.
    const int pw = lane & (p.wpt - 1), hv = lane >> 4;
    const int n0 = BP >= 2 ? hv * kPer : 0;
    const int red_pi = warp * p.tpu + ((lane & 15) >> wpt_shift);       // this lane's pair: row tile red_pi >> 4 of the unit, row red_pi & 15
    const int red_row = (red_pi >> 4) * 16 + (red_pi & 15);      // its row inside the row unit
    const uint32_t red_src = red_addr + static_cast<uint32_t>(((red_pi >> 4) * p.wpt + pw) * kTileFloats + (red_pi & 15) * BP + n0) * 4u;
    const bool red_active = BP >= 2 || hv == 0;
    const bool red_writer = pw == 0 && red_active;
    // Counts this warp's last `pend` units (row units ru_last - pend + 1 .. ru_last of one slot) in and finishes the
    // row units it completes.
    int pend = 0;
    auto flush_pending = [&](int ru_last) {
        __threadfence();
        __syncwarp();
        const int ru0 = ru_last - pend + 1;
        unsigned int prev = 0xffffffffu;
        if (lane < pend) prev = atomicAdd(&p.counters[(ru0 + lane) * kWarps + warp], 1u);
        unsigned int done = __ballot_sync(0xffffffffu, prev == static_cast<unsigned int>(p.n_slots) - 1u);
        pend = 0;
        if (done == 0u) return;
        __threadfence();
        if (prev == static_cast<unsigned int>(p.n_slots) - 1u) p.counters[(ru0 + lane) * kWarps + warp] = 0u;  // ready for the next launch
        // the outputs of all completed row units side by side over the lanes; up to 8 slots' partial sums are requested
        // at once (one round trip to L2) and added in slot order
        const int per_unit = p.tpu * BP;
        const int n_done = __popc(done) * per_unit;
        for (int idx = lane; idx < n_done; idx += 32) {
            const int k = idx / per_unit, e = idx - k * per_unit;
            const int ru = ru0 + static_cast<int>(__fns(done, 0u, k + 1));
            const int n = e % BP, pi = warp * p.tpu + e / BP;
            const int row = (ru * p.tpu + (pi >> 4)) * 16 + (pi & 15);
            if (row < p.out && n < p.batch) {
                const float sc = __ldg(p.norms + row) * p.inv_scale;
                const float* src = p.partial + static_cast<size_t>(n) * p.out_pad + row;
                float total = 0.f;
                for (int c0 = 0; c0 < p.n_slots; c0 += 8) {
                    float t[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        t[c] = (c0 + c < p.n_slots) ? __ldcg(src + static_cast<size_t>(c0 + c) * 8 * p.out_pad) : 0.f;
#pragma unroll
                    for (int c = 0; c < 8; ++c) total += t[c];
                }
                store_y<SCATTER>(p, sargs, n, row, __float2half_rn(total * sc));
            }
        }
    };
    auto reduce_unit = [&](int slot, int ru, int rs, uint32_t parity) {
        if (!mbar_wait(bar_written + 8u * rs, parity)) {
            raise_status(p.status, 5u);
            atomicExch(&s_abort, 1u);
        }
        {
            const int row = ru * p.tpu * 16 + red_row;
            const bool wr = red_writer && row < p.out;
            float sc = 0.f;
            // the norm is fetched first so that its latency hides behind the exchanges
            if constexpr (!MULTI) sc = wr ? __ldg(p.norms + row) * p.inv_scale : 0.f;
            float v[kPer];
#pragma unroll
            for (int k = 0; k < kPer; ++k) v[k] = 0.f;
            if (red_active) {
                const uint32_t src = red_src + static_cast<uint32_t>(rs) * kSlotBytes;
                if constexpr (kPer == 4) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(src));
                else if constexpr (kPer == 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(src));
                else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[0]) : "r"(src));
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                if (o < p.wpt) {
#pragma unroll
                    for (int k = 0; k < kPer; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
                }
            }
            if (wr) {
#pragma unroll
                for (int k = 0; k < kPer; ++k) {
                    const int n = n0 + k;
                    if constexpr (!MULTI) {
                        if (n < p.batch) store_y<SCATTER>(p, sargs, n, row, __float2half_rn(v[k] * sc));
                    } else {
                        p.partial[(static_cast<size_t>(slot) * 8 + n) * p.out_pad + row] = v[k];
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_read + 8u * rs);
        if constexpr (MULTI) {
            // Row units spread over several slots.  A warp owns the same rows of a row unit in every slot, so the
            // arrival count is kept per (row unit, warp): the warp that brings it to n_slots adds the slots' partial
            // sums of its rows in slot order and writes y.  The fence between the partial stores and the count makes
            // the warp wait for its memory traffic, code loads in flight included, so it is paid once per
            // kFlushUnits units (consecutive row units of one slot), not per unit.
            ++pend;
            if (pend == kFlushUnits || ru + 1 == p.n_row_units) flush_pending(ru);
        }
    };
    // B fragments.  bp rows fill bp of a product's eight columns: so the columns are 8 / bp products' pieces of the rows side by side (fragment_place), each of
    // those products has an accumulator, and only its own columns of it count.  With a fragment per product, 64 registers whatever the rows and zero columns for those that
    // are missing, fewer lookups were in flight: one row, 4096 x 4096 7.5 -> 6.3 us, 1024 x 1024 5.0 -> 4.0, 18944 x 3584 24.0 -> 22.5.
    uint32_t bfrag[4][2 * kFrag];
    int staged_slot = -1;
    // ring bookkeeping: slot / parity for the unit being written and the unit being summed
    int ws = 0;             // write slot = i % kRing
    uint32_t wpar = 0;      // parity of the "read" phase the writer waits for = ((i / kRing) - 1) & 1
    int rs = 0;             // slot of the unit being summed = (i - kLag) % kRing
    uint32_t rpar = 0;      // parity of its "written" phase = ((i - kLag) / kRing) & 1
    Pos red = cur;          // position of the unit being summed

    // Makes `slot` the current one: rebuilds this warp's B fragments.  x0 is this lane's first-row activation when the
    // caller has already requested it (have_x0).
    float xs[2];   // two rotations: the scales of activation rows 2q and 2q + 1 in this warp's slice
    auto stage_slot = [&](int slot, const uint4& x0, bool have_x0) {
            // B fragment of MMA (s, m): k = q -> column 64 s + 16 q + 2 m, k = q+4 -> the next column; n = g: row and product (see bfrag).
            const int colw = (MULTI ? slot * chunk_cols : 0) + slice0;  // first column of this warp's slice
            const int col0 = colw + 16 * q;
            if (ROW || (BP == 1 && !DUAL && p.x != nullptr)) {
                // One activation row (the launcher rotates in here only then): rotate this warp's 256 columns of it.
                // Lane l holds columns 8l..8l+7 of the slice, stages below 8 stay in the lane, the rest are lane
                // exchanges (same add tree as rotate_x_kernel).  A 1 KB strip of shared memory per warp turns the
                // result into the fragment layout.
                const int cl = colw + 8 * lane;
                uint4 xc = x0;
                if (!have_x0) {
                    xc = make_uint4(0, 0, 0, 0);
                    if (cl < p.in) xc = load_x(cl);
                }
                float v[8];
                const uint4 sg = MULTI && !have_x0 ? chunk_signs(p.seed_p, static_cast<uint32_t>(8 * lane), p.block) : row_signs;
                rotate_chunk(v, xc, sg, p.block, lane, 0xffffffffu);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = to_tf32(v[j] * p.inv_sqrt_block);
                sts_v4(strip_addr + static_cast<uint32_t>(lane) * 32u, v[0], v[1], v[2], v[3]);
                sts_v4(strip_addr + static_cast<uint32_t>(lane) * 32u + 16u, v[4], v[5], v[6], v[7]);
                __syncwarp();
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];"
                                 : "=r"(bfrag[s][0]), "=r"(bfrag[s][1])
                                 : "r"(strip_addr + static_cast<uint32_t>(64 * s + 16 * q + 2 * g) * 4u));
                __syncwarp();
            } else {
            const float* xr = p.xrot + static_cast<size_t>(colw) * kFrag;
            if constexpr (DUAL) {
                const int slices = (p.in + kSlice - 1) / kSlice;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int n = 2 * q + k;
                    xs[k] = (n < BP && n < p.batch && colw < p.in) ? p.xscale[n * slices + colw / kSlice] : 0.f;
                }
            }
            const bool have_row = (g & (kFrag - 1)) < p.batch;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const bool ok = have_row && (col0 + 64 * s) < p.in;
                const int groups = colw + 64 * s + 64 <= p.in ? 4 : 2;   // fragment_groups
                if constexpr (BP == 1) {
                    const float2 t = ok ? *reinterpret_cast<const float2*>(xr + 64 * s + 2 * (g * groups + q)) : make_float2(0.f, 0.f);
                    bfrag[s][0] = __float_as_uint(t.x);
                    bfrag[s][1] = __float_as_uint(t.y);
                } else {
#pragma unroll
                    for (int k = 0; k < 2 * kFrag; k += 4) {
                        const float4 t = ok ? *reinterpret_cast<const float4*>(xr + 64 * kFrag * s + (2 * k + g) * groups * 4 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
                        bfrag[s][k] = __float_as_uint(t.x);
                        bfrag[s][k + 1] = __float_as_uint(t.y);
                        bfrag[s][k + 2] = __float_as_uint(t.z);
                        bfrag[s][k + 3] = __float_as_uint(t.w);
                    }
                }
            }
            }
        staged_slot = slot;
    };
    stage_slot(cur.slot, x_first, ROW || (!DUAL && p.x != nullptr));

    for (int i = 0; i < n_local; ++i) {
        if (AT_FIRST ? i > 0 && cur.ru == 0 : cur.slot != staged_slot) stage_slot(cur.slot, make_uint4(0, 0, 0, 0), false);
        const bool has_next = i + 1 < n_local;

        float acc[kAcc][4];
#pragma unroll
        for (int m = 0; m < kAcc; ++m)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[m][k] = 0.f;
        float(&acc0)[4] = acc[0];
        float(&acc1)[4] = acc[1];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            uint4& lo = blo[s % kSteps];
            uint4& hi = bhi[s % kSteps];
            // Eight independent lookups (a word of each row), then the two MMAs they feed (bytes 0, 1 of the words feed one, bytes 2, 3 the next), kAcc
            // accumulator chains.  Once the last words' addresses are formed the code registers are free: the step kSteps ahead is loaded into them.
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint32_t l = w == 0 ? lo.x : (w == 1 ? lo.y : (w == 2 ? lo.z : lo.w));
                const uint32_t u = w == 0 ? hi.x : (w == 1 ? hi.y : (w == 2 ? hi.z : hi.w));
                uint32_t ad[8];
                ad[0] = lut_addr<0>(l, lane_const);
                ad[1] = lut_addr<0>(u, lane_const);
                ad[2] = lut_addr<1>(l, lane_const);
                ad[3] = lut_addr<1>(u, lane_const);
                ad[4] = lut_addr<2>(l, lane_const);
                ad[5] = lut_addr<2>(u, lane_const);
                ad[6] = lut_addr<3>(l, lane_const);
                ad[7] = lut_addr<3>(u, lane_const);
                if (w == 3) {
                    if (s + kSteps < 4) load_step(cur, (s + kSteps) % 4, true, lo, hi);
                    else load_step(nxt, (s + kSteps) % 4, has_next, lo, hi);
                }
                uint32_t av[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) av[k] = lut_load(ad[k]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int m = 2 * w + h, b = 2 * (m / kSide);
                    if constexpr (DUAL) mma_f16(acc[m % kAcc], av[4 * h], av[4 * h + 1], av[4 * h + 2], av[4 * h + 3], bfrag[s][b], bfrag[s][b + 1]);
                    else mma_tf32(acc[m % kAcc], av[4 * h], av[4 * h + 1], av[4 * h + 2], av[4 * h + 3], bfrag[s][b], bfrag[s][b + 1]);
                }
            }
        }
        if (!has_next) grid_launch_dependents();  // the next kernel may start setting up

        // ---- cross-warp sum without a CTA-wide barrier, kLag units behind ----
        // Every warp drops its partial tile of unit i into ring slot i % kRing and signals
        // "written"; the sum is done kLag units later by all warps symmetrically, followed by
        // "read".  With a deep ring (16 slots for one activation row) warps drift apart by
        // several units, so a slow memory response delays one warp, not the CTA.
        if (i >= kLag) {
            reduce_unit(red.slot, red.ru, rs, rpar);
            red = next_pos(red);
            if (++rs == kRing) { rs = 0; rpar ^= 1u; }
        }
        if (i >= kRing && !mbar_wait(bar_read + 8u * ws, wpar)) {
            raise_status(p.status, 4u);
            atomicExch(&s_abort, 1u);
        }
        {
            // C fragment: (row g, columns 2q, 2q+1) and (row g+8, same columns)
            const uint32_t dst = red_addr + static_cast<uint32_t>(ws) * kSlotBytes + static_cast<uint32_t>(warp * kTileFloats) * 4u;
            const int n = 2 * q;
            // Lane q has columns 2q and 2q + 1: of accumulator m' those that are rows for product m' count, and the products' sums meet in the lanes of the rows.
            if constexpr (BP == 1) {
                float top = q == 0 ? acc[0][0] + acc[1][1] : q == 1 ? acc[2][0] + acc[3][1] : q == 2 ? acc[4][0] + acc[5][1] : acc[6][0] + acc[7][1];
                float low = q == 0 ? acc[0][2] + acc[1][3] : q == 1 ? acc[2][2] + acc[3][3] : q == 2 ? acc[4][2] + acc[5][3] : acc[6][2] + acc[7][3];
                top += __shfl_xor_sync(0xffffffffu, top, 1);
                low += __shfl_xor_sync(0xffffffffu, low, 1);
                acc0[0] = top + __shfl_xor_sync(0xffffffffu, top, 2);
                acc0[2] = low + __shfl_xor_sync(0xffffffffu, low, 2);
                acc1[0] = acc1[2] = 0.f;
            } else if constexpr (kFrag == 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float v = q < 2 ? acc[0][k] : acc[1][k];
                    acc0[k] = v + __shfl_xor_sync(0xffffffffu, v, 2);
                    acc1[k] = 0.f;
                }
            }
            if constexpr (DUAL) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    acc0[k] *= xs[k & 1];
                    acc1[k] *= xs[k & 1];
                }
            }
            if (n < BP) {
                sts_f32(dst + static_cast<uint32_t>(g * BP + n) * 4u, acc0[0] + acc1[0]);
                sts_f32(dst + static_cast<uint32_t>((g + 8) * BP + n) * 4u, acc0[2] + acc1[2]);
                if (n + 1 < BP) {
                    sts_f32(dst + static_cast<uint32_t>(g * BP + n + 1) * 4u, acc0[1] + acc1[1]);
                    sts_f32(dst + static_cast<uint32_t>((g + 8) * BP + n + 1) * 4u, acc0[3] + acc1[3]);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_written + 8u * ws);
        if (++ws == kRing) { ws = 0; if (i >= kRing) wpar ^= 1u; }

        cur = nxt;
        if (i + 2 < n_local) nxt = next_pos(nxt);
    }
    // the last kLag units (or all of them, for a short range) are still to be summed
    for (int k = (n_local > kLag ? n_local - kLag : 0); k < n_local; ++k) {
        reduce_unit(red.slot, red.ru, rs, rpar);
        if constexpr (MULTI) if (k + 1 == n_local && pend > 0) flush_pending(red.ru);
        red = next_pos(red);
        if (++rs == kRing) { rs = 0; rpar ^= 1u; }
    }

    // ---- completion signal to the destinations' owners ----
    // Every thread orders its (possibly remote) result stores system-wide, the CTA counts in, and
    // the CTA that completes the grid publishes the flag everywhere.  Whoever then reads the flag
    // with acquire semantics sees all of this launch's results.
    if constexpr (SCATTER) {
    if (sargs.n_signal > 0 || LL) {
        __shared__ unsigned int s_last;
        // Packets, one slot: every row of this CTA's units was stored by this CTA, so it sends its own rows as soon
        // as it is done - the sends of the grid run side by side and nothing waits for the slowest CTA.  (With several
        // slots the CTA that completes a row tile is not known in advance: the completing CTA of the grid sends all.)
        const bool own_rows = LL && !MULTI;
        if constexpr (LL) if (own_rows) {
            __syncthreads();   // this CTA's stores are ordered before the loads below (read back through L2)
            const int per_row = p.out / 4;
            ll_send_packets(sargs, p.y, per_row, p.batch, u_begin * p.tpu * 4, min(per_row, (u_begin + n_local) * p.tpu * 4));
        }
        // results that went to other GPUs need a system-scope fence; with the bulk copy every CTA's
        // results are local and only the copying CTA pays for one
        if (sargs.bulk) __threadfence();
        else __threadfence_system();
        __syncthreads();
        if (tid == 0) {
            const unsigned int prev = atomicAdd(sargs.done_counter, 1u);
            s_last = (prev == static_cast<unsigned int>(nblk) - 1u) ? 1u : 0u;
        }
        __syncthreads();
        if (LL && s_last) {
            __threadfence();
            if constexpr (LL) if (!own_rows) ll_send_packets(sargs, p.y, p.out / 4, p.batch, 0, p.out / 4);
            __syncthreads();
            if (tid == 0) {
                *sargs.done_counter = 0u;  // ready for the next launch (stream order)
                atomicAdd(sargs.epoch, 1u);
                if (sargs.n_wait > 0) atomicAdd(sargs.wait_epoch, 1u);   // every CTA has read it by now
            }
        } else if (s_last) {
            __threadfence();
            if (sargs.bulk && sargs.n_peer > 0) {
                // the whole block (batch rows of `out` halves, y_stride apart) to every peer: 16-byte
                // pieces where the rows allow it
                const bool vec = (p.out % 8 == 0) && (sargs.y_stride % 8 == 0) && (reinterpret_cast<uintptr_t>(p.y) % 16 == 0);
                if (vec) {
                    const int per_row = p.out / 8;
                    for (int i = tid; i < per_row * p.batch; i += kCtaThreads) {
                        const int n = i / per_row, c = i - n * per_row;
                        const size_t o = static_cast<size_t>(n) * sargs.y_stride + static_cast<size_t>(c) * 8;
                        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p.y + o));
#pragma unroll
                        for (int d = 0; d < 7; ++d)
                            if (d < sargs.n_peer) *reinterpret_cast<uint4*>(sargs.y_peer[d] + o) = v;
                    }
                } else {
                    for (int i = tid; i < p.out * p.batch; i += kCtaThreads) {
                        const int n = i / p.out, c = i - n * p.out;
                        const size_t o = static_cast<size_t>(n) * sargs.y_stride + c;
                        const __half v = __ldcg(p.y + o);
#pragma unroll
                        for (int d = 0; d < 7; ++d)
                            if (d < sargs.n_peer) sargs.y_peer[d][o] = v;
                    }
                }
                __threadfence_system();
                __syncthreads();
            }
            if (tid == 0) {
                *sargs.done_counter = 0u;  // ready for the next launch (stream order)
                unsigned int value = sargs.signal_value;
                if (sargs.bulk) value = atomicAdd(sargs.epoch, 1u) + 1u;
                if (sargs.n_wait > 0) atomicAdd(sargs.wait_epoch, 1u);   // every CTA has read it by now
                __threadfence_system();
#pragma unroll
                for (int d = 0; d < 8; ++d)
                    if (d < sargs.n_signal)
                        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(sargs.signal[d] + sargs.signal_slot), "r"(value) : "memory");
            }
        }
    }
    }
}

template <int BP, bool MULTI, bool DUAL, bool DEEP = false>
__global__ void __launch_bounds__(kCtaThreads, 1) tq8_gemv_kernel(const GemvArgs p) {
    gemv_body<BP, false, false, MULTI, DUAL, false, DEEP, BP == 8 && MULTI && DUAL>(p, ScatterArgs{}, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
}
// The one activation row of a host caller, which rides in the launch (16 N bytes of fp16): as a kernel of its own in front, which wrote it to
// device memory, it cost a launch and its end.  4096 x 4096 from and to host memory 31.3 us, 29.7 so, 512 x 14336 39.8 and 33.5.
template <int N>
struct GemvRow {
    uint4 v[N];
};
template <int N, bool MULTI>
__global__ void __launch_bounds__(kCtaThreads, 1) tq8_gemv_row_kernel(const GemvArgs p, const __grid_constant__ GemvRow<N> row) {
    gemv_body<1, false, false, MULTI, false, true>(p, ScatterArgs{}, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x),
                                                   reinterpret_cast<const __half*>(row.v));
}
template <int BP, bool MULTI, bool DUAL>
__global__ void __launch_bounds__(kCtaThreads, 1) tq8_gemv_packets_kernel(const GemvArgs p, const ScatterArgs sc) {
    gemv_body<BP, true, true, MULTI, DUAL>(p, sc, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
}
template <int BP, bool MULTI, bool DUAL>
__global__ void __launch_bounds__(kCtaThreads, 1) tq8_gemv_scatter_kernel(const GemvArgs p, const ScatterArgs sc) {
    gemv_body<BP, true, false, MULTI, DUAL>(p, sc, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
}

// Several matrices that multiply the same activation (q / k / v, gate / up) in one launch: the grid is cut into one
// range of CTAs per matrix, in proportion to the matrices' units, and every CTA runs the ordinary body on its matrix
// with its index inside the range.  A decode layer's small projections then pay the launch and the prologue once.
constexpr int kMaxGroup = 4;
struct GemvGroupArgs {
    GemvArgs m[kMaxGroup];
    int cta_start[kMaxGroup + 1];   // CTAs cta_start[i] .. cta_start[i + 1] - 1 work on matrix i
    int n;
};
template <int BP, bool MULTI, bool DUAL>
__global__ void __launch_bounds__(kCtaThreads, 1) tq8_gemv_group_kernel(const __grid_constant__ GemvGroupArgs grp) {
    const int b = static_cast<int>(blockIdx.x);
    int i = 0;
    while (i + 1 < grp.n && b >= grp.cta_start[i + 1]) ++i;
    gemv_body<BP, false, false, MULTI, DUAL>(grp.m[i], ScatterArgs{}, b - grp.cta_start[i], grp.cta_start[i + 1] - grp.cta_start[i]);
}

// Waits (bounded) until flags[0..n) have all reached `value`: the receiving side of the completion
// signal above.  Runs on the GPU that owns the flags; the writers are kernels on other GPUs.
__global__ void peer_wait_kernel(const unsigned int* __restrict__ flags, int n, unsigned int value, unsigned int* status) {
    const int lane = threadIdx.x;
    if (lane >= n) return;
    const unsigned long long t0 = global_timer_ns();
    for (unsigned int spin = 0;; ++spin) {
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + lane) : "memory");
        if (static_cast<int>(v - value) >= 0) return;
        if ((spin & 255u) == 255u && global_timer_ns() - t0 > 5ull * kWaitLimitNs) {  // 1 s: a peer is gone
            raise_status(status, 10u);
            return;
        }
    }
}

// The wait that the decode kernel makes before it reads an activation that comes out of an exchange (see ScatterArgs), for a
// rotation that runs in front of it: bounded, and the epoch stays for the decode kernel to advance.
__global__ void gather_wait_kernel(const unsigned int* __restrict__ flags, int n, const unsigned int* __restrict__ wait_epoch, unsigned int* status) {
    const int lane = threadIdx.x;
    if (lane >= n) return;
    const unsigned int want = *reinterpret_cast<const volatile unsigned int*>(wait_epoch) + 1u;
    const unsigned long long t0 = global_timer_ns();
    for (unsigned int spin = 0;; ++spin) {
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + lane) : "memory");
        if (static_cast<int>(v - want) >= 0) return;
        if ((spin & 255u) == 255u && global_timer_ns() - t0 > 5ull * kWaitLimitNs) {   // 1 s: a peer is gone
            raise_status(status, 10u);
            return;
        }
    }
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// Warps that share one 16-row tile (a power of two up to 16); a chunk is that many 256-column slices, and
// the 16 / wpt row tiles of a unit run side by side.  Up to 4096 columns: the fewest warps that cover the
// row (one chunk).  Above: 16 warps per tile unless the last chunk would leave more than 15 % of the warps'
// slices empty (5120 columns = 20 slices: 16 + 4, i.e. 62 %); then the split with at most 8 chunks that leaves the
// fewest slices empty (5120: 4 warps, five chunks of 1024 columns; 4608: 4 warps, 90 %; 6144: 8 warps, 100 %).
int warps_per_tile(int in) {
    const int slices = (in + kSlice - 1) / kSlice;
    if (in <= kWarps * kSlice) {
        int w = 1;
        while (w < kWarps && w < slices) w <<= 1;
        return w;
    }
    auto fill = [&](int w) { return static_cast<double>(slices) / (static_cast<double>((slices + w - 1) / w) * w); };
    if (fill(kWarps) >= 0.85) return kWarps;
    // otherwise the split (at most 8 chunks) that leaves the fewest slices empty; the wider one when two are close
    int best = kWarps;
    for (int w = kWarps / 2; w >= 1; w >>= 1)
        if ((slices + w - 1) / w <= 8 && fill(w) > fill(best) + 0.02) best = w;
    return best;
}
int chunk_columns(int in) { return warps_per_tile(in) * kSlice; }

}  // namespace

// Scratch layout: [xrot: n_planes*8*in fp32][partials: n_slots*8*out_pad fp32][counters: n_row_tiles*16 u32]
static size_t scratch_bytes(int out, int in, int n_planes, int n_slots) {
    const int n_row_tiles = (out + 15) / 16;
    const size_t out_pad = static_cast<size_t>(n_row_tiles) * 16;
    size_t bytes = align256(static_cast<size_t>(n_planes) * 8 * in * sizeof(float));
    if (n_slots > 1)
        bytes += align256(static_cast<size_t>(n_slots) * 8 * out_pad * sizeof(float)) +
                 align256(static_cast<size_t>(n_row_tiles) * kWarps * sizeof(unsigned int));
    return bytes;
}
static int chunk_count(int in) { return (in + chunk_columns(in) - 1) / chunk_columns(in); }
size_t gemv_scratch_bytes(int out, int in, int n_planes) { return scratch_bytes(out, in, n_planes, chunk_count(in)); }

// Geometry, rotation mode and scratch pointers of one matrix (codes, norms, table, y and status are the caller's).
// Returns whether the kernel rotates the activation itself; otherwise rotate_x_kernel fills a.xrot first.
static bool fill_gemv_args(GemvArgs& a, const __half* x, int out, int in, int batch, uint32_t block, int n_planes, float pair_unit,
                           uint32_t seed_p, void* scratch) {
    a.out = out; a.in = in; a.batch = batch;
    const int n_row_tiles = (out + 15) / 16;
    a.wpt = warps_per_tile(in);
    a.tpu = kWarps / a.wpt;
    a.n_slots = chunk_count(in);
    a.out_pad = n_row_tiles * 16;
    a.n_row_units = (n_row_tiles + a.tpu - 1) / a.tpu;
    a.inv_scale = 1.0f / std::sqrt(static_cast<float>(in));
    if (n_planes == 2) {
        a.table += 512;          // (the pairs, behind the two tables)
        a.inv_scale *= pair_unit;
    }
    // Blocks that fit a warp's 256-column slice are rotated inside the GEMV kernel (16-byte
    // activation loads); larger blocks, or an unaligned activation, go through rotate_x_kernel.
    // In-kernel rotation handles one activation row after the other (a chain of lane exchanges per row) in every
    // warp, which costs more than the pre-kernel from two rows on (4096 x 4096: 9.0 / 11.3 / 15.3 us in-kernel
    // against 8.3 / 9.2 / 10.8 us with the pre-kernel at 2 / 4 / 8 rows; the same at one row).
    // Two rotations always take the pre-kernel: a warp's strip in here would be two such chains, and the scales must be known
    // before the first product (1024 x 512, block 128, one row: 7.3 us with two chains in every warp, 5.0 with the pre-kernel).
    const bool fused_rotation = n_planes == 1 && block <= static_cast<uint32_t>(kSlice) && in % 8 == 0 &&
                                reinterpret_cast<uintptr_t>(x) % 16 == 0 && batch == 1;
    a.x = fused_rotation ? x : nullptr;
    a.seed_p = seed_p;
    a.block = static_cast<int>(block);
    a.inv_sqrt_block = 1.0f / std::sqrt(static_cast<float>(block));
    uint8_t* sp = static_cast<uint8_t*>(scratch);
    float* xrot = reinterpret_cast<float*>(sp);
    a.xrot = xrot;
    a.xscale = xrot + static_cast<size_t>(8) * in;   // (two rotations: the second plane's room)
    if (a.n_slots > 1) {
        sp += align256(static_cast<size_t>(n_planes) * 8 * in * sizeof(float));
        a.partial = reinterpret_cast<float*>(sp);
        sp += align256(static_cast<size_t>(a.n_slots) * 8 * a.out_pad * sizeof(float));
        a.counters = reinterpret_cast<unsigned int*>(sp);
    }

    return fused_rotation;
}

static void launch_rotate_x_pair(const __half* x, float* xrot, int in, int batch, uint32_t block, uint32_t seed_p, uint32_t seed_r,
                                 cudaStream_t stream);
// Shared-memory opt-in of every instantiation, once per device.
static void configure_gemv_kernels();
void launch_tq8_gemv(const uint8_t* codes, const float* norms, const float* table, const __half* x, __half* y,
                     int out, int in, int batch, uint32_t block, int n_planes, float pair_unit,
                     uint32_t seed_p, uint32_t seed_r, void* scratch, unsigned int* status, int sm_count, cudaStream_t stream) {
    launch_tq8_gemv_scatter(codes, norms, table, x, &y, 1, out, out, in, batch, block, n_planes, pair_unit, seed_p, seed_r, scratch,
                            status, sm_count, stream);
}

void launch_peer_wait(const unsigned int* flags, int n, unsigned int value, unsigned int* status, cudaStream_t stream) {
    TQ_REQUIRE(flags != nullptr && n >= 1 && n <= 32, "peer wait: 1..32 flags");
    peer_wait_kernel<<<1, 32, 0, stream>>>(flags, n, value, status);
    TQ_CUDA(cudaGetLastError());
}

void launch_tq8_gemv_scatter(const uint8_t* codes, const float* norms, const float* table, const __half* x,
                             __half* const* dst, int n_dst, long dst_stride, int out, int in, int batch, uint32_t block,
                             int n_planes, float pair_unit, uint32_t seed_p, uint32_t seed_r, void* scratch, unsigned int* status,
                             int sm_count, cudaStream_t stream, unsigned int* const* signal, int signal_slot,
                             unsigned int signal_value, unsigned int* done_counter, const GemvGather* gather, int n_signal) {
    TQ_REQUIRE(dst != nullptr && n_dst >= 1 && n_dst <= 8, "tq8_gemv: 1..8 destinations");
    TQ_REQUIRE(dst_stride >= out, "tq8_gemv: destination row stride smaller than the layer's rows");
    __half* y = dst[0];
    TQ_REQUIRE(n_planes == 1 || n_planes == 2, "tq8_gemv: one or two rotation planes");
    TQ_REQUIRE(batch >= 1 && batch <= 8, "tq8_gemv handles 1..8 activation rows per launch");
    TQ_REQUIRE(is_pow2(block) && block >= 32 && block <= 1024, "WHT block size must be a power of two in [32, 1024]");
    TQ_REQUIRE(in % static_cast<int>(block) == 0, "in_features must be divisible by block_size");
    TQ_REQUIRE(scratch != nullptr, "tq8_gemv needs its scratch buffer");
    if (out == 0) return;

    GemvArgs a{};
    a.codes = codes; a.norms = norms; a.table = table; a.y = y; a.status = status;
    ScatterArgs sa{};
    sa.n_peer = n_dst - 1;
    for (int d = 1; d < n_dst; ++d) {
        TQ_REQUIRE(dst[d] != nullptr, "tq8_gemv: NULL destination");
        sa.y_peer[d - 1] = dst[d];
    }
    sa.y_stride = dst_stride;
    sa.n_signal = 0;
    if (signal != nullptr) {
        sa.n_signal = n_signal > 0 ? n_signal : n_dst;
        TQ_REQUIRE(sa.n_signal <= 8, "tq8_gemv: at most 8 flag arrays");
        for (int d = 0; d < sa.n_signal; ++d) {
            TQ_REQUIRE(signal[d] != nullptr, "tq8_gemv: NULL signal array");
            sa.signal[d] = signal[d];
        }
        sa.signal_slot = signal_slot;
        sa.signal_value = signal_value;
        TQ_REQUIRE(done_counter != nullptr, "tq8_gemv: signalling needs a completion counter in device memory");
        sa.done_counter = done_counter;
    }
    if (gather != nullptr) {
        TQ_REQUIRE((signal != nullptr || gather->ll_world > 0) && gather->epoch != nullptr,
                   "tq8_gemv: the fused all-gather needs flags (or packet buffers) and an epoch counter");
        TQ_REQUIRE(gather->n_wait >= 0 && gather->n_wait <= 32, "tq8_gemv: 0..32 flags to wait for");
        TQ_REQUIRE(gather->n_wait == 0 || ((gather->wait_flags != nullptr || gather->ll_world > 0) && gather->wait_epoch != nullptr),
                   "tq8_gemv: waiting needs the local flag array and the wait counter");
        sa.bulk = 1;
        if (gather->ll_world > 0) {
            TQ_REQUIRE(gather->ll_world <= 8 && gather->ll_rank >= 0 && gather->ll_rank < gather->ll_world, "tq8_gemv: bad rank / world");
            TQ_REQUIRE(out % 4 == 0 && dst_stride % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 8 == 0,
                       "tq8_gemv: the flag-in-data exchange moves groups of four rows (8-byte aligned)");
            sa.ll = 1;
            sa.ll_rank = gather->ll_rank;
            sa.ll_world = gather->ll_world;
            for (int r = 0; r < gather->ll_world; ++r) {
                TQ_REQUIRE(gather->ll_base[r] != nullptr, "tq8_gemv: NULL packet buffer");
                sa.ll_base[r] = static_cast<uint4*>(gather->ll_base[r]);
            }
            sa.n_peer = 0;   // results are stored locally; the packets carry them to the other ranks
            TQ_REQUIRE(done_counter != nullptr, "tq8_gemv: the exchange needs a completion counter in device memory");
            sa.done_counter = done_counter;
        }
        sa.epoch = gather->epoch;
        sa.wait_flags = gather->wait_flags;
        sa.n_wait = gather->n_wait;
        sa.wait_epoch = gather->wait_epoch;
    }
    const bool fused_rotation = fill_gemv_args(a, x, out, in, batch, block, n_planes, pair_unit, seed_p, scratch);
    float* xrot = const_cast<float*>(a.xrot);
    const int bp = batch <= 1 ? 1 : (batch <= 2 ? 2 : (batch <= 4 ? 4 : 8));   // (of the ring; fragments: padded_rows)

    configure_gemv_kernels();

    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    const int n_attr = 1;

    // 1. rotate the activation, once the exchange that it may come from is complete
    if (!fused_rotation && sa.n_wait > 0 && !sa.ll) {
        gather_wait_kernel<<<1, 32, 0, stream>>>(sa.wait_flags, sa.n_wait, sa.wait_epoch, status);
        TQ_CUDA(cudaGetLastError());
    }
    if (n_planes == 2) launch_rotate_x_pair(x, xrot, in, batch, block, seed_p, seed_r, stream);
    else if (!fused_rotation) launch_rotate_x(x, xrot, in, batch, block, 1, seed_p, seed_r, stream, true);
    // 2. the GEMV itself
    {
        const int n_units = a.n_row_units * a.n_slots;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(n_units < sm_count ? n_units : sm_count);
        cfg.blockDim = dim3(kCtaThreads);
        cfg.dynamicSmemBytes = kGemvSmem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = n_attr;
        // One row has the registers for four steps of codes.  They pay from some eight units a CTA on: 2048 x 151936 (32 units) 63.0 -> 61.4 us, 5120 x 55296 70.2 ->
        // 67.7, 18944 x 3584 (8) 22.6 -> 22.1; before, the first unit comes later: 4096 x 4096 (2) 6.3 -> 6.7, 4096 x 11008 (5) 12.4 -> 12.7.
        const bool deep = n_units >= 8 * sm_count - sm_count / 2;
        // one destination with the layer's own row stride and no signal: the plain variant
        const bool scatter = sa.n_peer > 0 || sa.n_signal > 0 || sa.ll != 0 || sa.y_stride != a.out;
#define TQ_GEMV_LAUNCH3(BPV, MV, DV)                                                                  \
    if (sa.ll) TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_packets_kernel<BPV, MV, DV>, a, sa));        \
    else if (scatter) TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_scatter_kernel<BPV, MV, DV>, a, sa)); \
    else if (BPV == 1 && deep) TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_kernel<BPV, MV, DV, BPV == 1>, a)); \
    else TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_kernel<BPV, MV, DV>, a));
#define TQ_GEMV_LAUNCH2(BPV, MV)                         \
    if (n_planes == 2) { TQ_GEMV_LAUNCH3(BPV, MV, true) } \
    else { TQ_GEMV_LAUNCH3(BPV, MV, false) }
#define TQ_GEMV_LAUNCH(BPV)                           \
    if (a.n_slots > 1) { TQ_GEMV_LAUNCH2(BPV, true) } \
    else { TQ_GEMV_LAUNCH2(BPV, false) }
        switch (bp) {
            case 1: TQ_GEMV_LAUNCH(1) break;
            case 2: TQ_GEMV_LAUNCH(2) break;
            case 4: TQ_GEMV_LAUNCH(4) break;
            default: TQ_GEMV_LAUNCH(8) break;
        }
#undef TQ_GEMV_LAUNCH
#undef TQ_GEMV_LAUNCH2
#undef TQ_GEMV_LAUNCH3
    }
}

bool gemv_takes_host_row(int in, uint32_t block, int n_planes) {
    return n_planes == 1 && block <= static_cast<uint32_t>(kSlice) && in % 8 == 0 && static_cast<size_t>(in) * 2 <= kMaxParamRowBytes;
}
template <int N, bool MULTI>
static void launch_gemv_row(const GemvArgs& a, const void* host_x, bool is_f16, int sm_count, cudaStream_t stream) {
    GemvRow<N> row;
    if (is_f16) std::memcpy(row.v, host_x, static_cast<size_t>(a.in) * 2);
    else host_f32_to_f16(static_cast<const float*>(host_x), reinterpret_cast<uint16_t*>(row.v), static_cast<size_t>(a.in));
    static bool configured[64] = {false};   // the opt-in shared-memory size is a per-device function attribute
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute((tq8_gemv_row_kernel<N, MULTI>), cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemvSmem)));
        if (dev < 64) configured[dev] = true;
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    const int n_units = a.n_row_units * a.n_slots;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n_units < sm_count ? n_units : sm_count);
    cfg.blockDim = dim3(kCtaThreads);
    cfg.dynamicSmemBytes = kGemvSmem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {const_cast<GemvArgs*>(&a), &row};   // by address: the row is copied once, into the launch
    TQ_CUDA(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(tq8_gemv_row_kernel<N, MULTI>), args));
}
void launch_tq8_gemv_host_row(const uint8_t* codes, const float* norms, const float* table, const void* host_x, bool is_f16, __half* y, int out,
                              int in, uint32_t block, uint32_t seed_p, void* scratch, unsigned int* status, int sm_count, cudaStream_t stream) {
    TQ_REQUIRE(gemv_takes_host_row(in, block, 1), "tq8_gemv: the activation row does not fit a launch's parameters");
    TQ_REQUIRE(is_pow2(block) && block >= 32, "WHT block size must be a power of two in [32, 1024]");
    TQ_REQUIRE(in % static_cast<int>(block) == 0, "in_features must be divisible by block_size");
    TQ_REQUIRE(scratch != nullptr, "tq8_gemv needs its scratch buffer");
    if (out == 0) return;
    GemvArgs a{};
    a.codes = codes; a.norms = norms; a.table = table; a.y = y; a.status = status;
    fill_gemv_args(a, nullptr, out, in, 1, block, 1, 1.0f, seed_p, scratch);
    // the launch copies its whole parameter block: sizes in steps of two
    if (a.n_slots == 1) {   // 4096 columns at most
        if (in <= 2048) launch_gemv_row<256, false>(a, host_x, is_f16, sm_count, stream);
        else launch_gemv_row<512, false>(a, host_x, is_f16, sm_count, stream);
    } else {
        if (in <= 8192) launch_gemv_row<1024, true>(a, host_x, is_f16, sm_count, stream);
        else launch_gemv_row<kMaxParamRowBytes / 16, true>(a, host_x, is_f16, sm_count, stream);
    }
}

static void configure_gemv_kernels() {
    // the opt-in shared-memory size is a per-device function attribute
    static bool configured[64] = {false};
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && configured[dev]) return;
#define TQ_GEMV_ATTR1(K) TQ_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemvSmem)));
#define TQ_GEMV_ATTR2(BPV, DV)                               \
    TQ_GEMV_ATTR1((tq8_gemv_kernel<BPV, false, DV>))         \
    TQ_GEMV_ATTR1((tq8_gemv_kernel<BPV, true, DV>))          \
    TQ_GEMV_ATTR1((tq8_gemv_scatter_kernel<BPV, false, DV>)) \
    TQ_GEMV_ATTR1((tq8_gemv_scatter_kernel<BPV, true, DV>))  \
    TQ_GEMV_ATTR1((tq8_gemv_packets_kernel<BPV, false, DV>)) \
    TQ_GEMV_ATTR1((tq8_gemv_packets_kernel<BPV, true, DV>))  \
    TQ_GEMV_ATTR1((tq8_gemv_group_kernel<BPV, false, DV>))   \
    TQ_GEMV_ATTR1((tq8_gemv_group_kernel<BPV, true, DV>))
#define TQ_GEMV_ATTR(BPV)     \
    TQ_GEMV_ATTR2(BPV, false) \
    TQ_GEMV_ATTR2(BPV, true)
    TQ_GEMV_ATTR(1)
    TQ_GEMV_ATTR1((tq8_gemv_kernel<1, false, false, true>))
    TQ_GEMV_ATTR1((tq8_gemv_kernel<1, true, false, true>))
    TQ_GEMV_ATTR1((tq8_gemv_kernel<1, false, true, true>))
    TQ_GEMV_ATTR1((tq8_gemv_kernel<1, true, true, true>))
    TQ_GEMV_ATTR(2)
    TQ_GEMV_ATTR(4)
    TQ_GEMV_ATTR(8)
#undef TQ_GEMV_ATTR
#undef TQ_GEMV_ATTR2
#undef TQ_GEMV_ATTR1
    if (dev < 64) configured[dev] = true;
}

void launch_tq8_gemv_group(const GemvGroupItem* items, int n, const __half* x, int batch, int sm_count, cudaStream_t stream) {
    TQ_REQUIRE(items != nullptr && n >= 1 && n <= kMaxGroup, "tq8_gemv group: 1..4 matrices");
    TQ_REQUIRE(x != nullptr && batch >= 1 && batch <= 8, "tq8_gemv group: 1..8 activation rows");
    GemvGroupArgs grp{};
    grp.n = n;
    int units[kMaxGroup], total_units = 0;
    bool fused[kMaxGroup];
    for (int i = 0; i < n; ++i) {
        const GemvGroupItem& it = items[i];
        TQ_REQUIRE(it.codes && it.norms && it.table && it.y && it.scratch, "tq8_gemv group: NULL argument");
        TQ_REQUIRE(it.out >= 1 && it.in == items[0].in && it.n_planes == items[0].n_planes,
                   "tq8_gemv group: the matrices must share in_features and the rotation mode");
        TQ_REQUIRE(it.n_planes == 1 || it.n_planes == 2, "n_planes must be 1 or 2");
        TQ_REQUIRE(is_pow2(it.block) && it.block >= 32 && it.block <= 1024, "WHT block size must be a power of two in [32, 1024]");
        TQ_REQUIRE(it.in % static_cast<int>(it.block) == 0, "in_features must be divisible by block_size");
        GemvArgs& a = grp.m[i];
        a.codes = it.codes; a.norms = it.norms; a.table = it.table; a.y = it.y; a.status = it.status;
        fused[i] = fill_gemv_args(a, x, it.out, it.in, batch, it.block, it.n_planes, it.pair_unit, it.seed_p, it.scratch);
        units[i] = a.n_row_units * a.n_slots;
        total_units += units[i];
    }
    // CTAs in proportion to the units, at least one per matrix, never more than a matrix has units
    const int total = total_units < sm_count ? total_units : sm_count;
    TQ_REQUIRE(total >= n, "tq8_gemv group: fewer SMs than matrices");
    int ctas[kMaxGroup], given = 0;
    for (int i = 0; i < n; ++i) {
        long c = static_cast<long>(total) * units[i] / total_units;
        ctas[i] = static_cast<int>(c < 1 ? 1 : (c > units[i] ? units[i] : c));
        given += ctas[i];
    }
    while (given > total) {   // the minimum of one pushed the sum over: take from the largest
        int big = 0;
        for (int i = 1; i < n; ++i) if (ctas[i] > ctas[big]) big = i;
        --ctas[big]; --given;
    }
    while (given < total) {   // rounding left CTAs over: to the matrix with the most units per CTA that can still use one
        int best = -1;
        for (int i = 0; i < n; ++i)
            if (ctas[i] < units[i] && (best < 0 || static_cast<long>(units[i]) * ctas[best] > static_cast<long>(units[best]) * ctas[i])) best = i;
        if (best < 0) break;
        ++ctas[best]; ++given;
    }
    grp.cta_start[0] = 0;
    for (int i = 0; i < n; ++i) grp.cta_start[i + 1] = grp.cta_start[i] + ctas[i];
    for (int i = n; i < kMaxGroup; ++i) grp.cta_start[i + 1] = grp.cta_start[n];
    configure_gemv_kernels();
    for (int i = 0; i < n; ++i)
        if (!fused[i]) {
            float* const xrot = const_cast<float*>(grp.m[i].xrot);
            if (items[i].n_planes == 2) launch_rotate_x_pair(x, xrot, items[i].in, batch, items[i].block, items[i].seed_p, items[i].seed_r, stream);
            else launch_rotate_x(x, xrot, items[i].in, batch, items[i].block, 1, items[i].seed_p, items[i].seed_r, stream, true);
        }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grp.cta_start[n]);
    cfg.blockDim = dim3(kCtaThreads);
    cfg.dynamicSmemBytes = kGemvSmem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int bp = batch <= 1 ? 1 : (batch <= 2 ? 2 : (batch <= 4 ? 4 : 8));   // (of the ring; fragments: padded_rows)
    const bool multi = grp.m[0].n_slots > 1;   // the same for all: same in_features and planes
    const bool dual = items[0].n_planes == 2;
#define TQ_GROUP_LAUNCH2(BPV, DV)                                                             \
    if (multi) TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_group_kernel<BPV, true, DV>, grp)); \
    else TQ_CUDA(cudaLaunchKernelEx(&cfg, tq8_gemv_group_kernel<BPV, false, DV>, grp));
#define TQ_GROUP_LAUNCH(BPV)                    \
    if (dual) { TQ_GROUP_LAUNCH2(BPV, true) } \
    else { TQ_GROUP_LAUNCH2(BPV, false) }
    switch (bp) {
        case 1: TQ_GROUP_LAUNCH(1) break;
        case 2: TQ_GROUP_LAUNCH(2) break;
        case 4: TQ_GROUP_LAUNCH(4) break;
        default: TQ_GROUP_LAUNCH(8) break;
    }
#undef TQ_GROUP_LAUNCH
#undef TQ_GROUP_LAUNCH2
}

// The activation rotation alone (the pre-kernel of several rows or WHT blocks above 256 columns), also for the other decode
// kernels: xrot = [n_planes, batch, in] fp32.
void launch_rotate_x(const __half* x, float* xrot, int in, int batch, uint32_t block, int n_planes, uint32_t seed_p,
                     uint32_t seed_r, cudaStream_t stream, bool fragments) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(block));
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (reinterpret_cast<uintptr_t>(x) % 16 == 0) {   // (a row is a multiple of 32 halves)
        const int wide_cols = block <= 256 ? 256 : static_cast<int>(block);
        auto* const wide = wide_cols == 256 ? rotate_x_wide_kernel<1> : (wide_cols == 512 ? rotate_x_wide_kernel<2> : rotate_x_wide_kernel<4>);
        cfg.gridDim = dim3((n_planes * batch * ((in + wide_cols - 1) / wide_cols) + 3) / 4);
        cfg.dynamicSmemBytes = kRotateXSmem;
        TQ_CUDA(cudaLaunchKernelEx(&cfg, wide, x, xrot, in, batch, n_planes, static_cast<int>(block), seed_p, seed_r, inv_sqrt, fragments ? padded_rows(batch) : 0));
        return;
    }
    const int n_warps = n_planes * batch * (in / static_cast<int>(block));
    cfg.gridDim = dim3((n_warps + 3) / 4);
#define TQ_ROT_CASE(EV)                                                                                            \
    case 32 * EV:                                                                                                  \
        TQ_CUDA(cudaLaunchKernelEx(&cfg, rotate_x_kernel<EV>, x, xrot, in, batch, n_planes, seed_p, seed_r, inv_sqrt, fragments ? padded_rows(batch) : 0)); \
        break;
    switch (block) {
        TQ_ROT_CASE(1) TQ_ROT_CASE(2) TQ_ROT_CASE(4) TQ_ROT_CASE(8) TQ_ROT_CASE(16) TQ_ROT_CASE(32)
        default: throw Error("unsupported WHT block size");
    }
#undef TQ_ROT_CASE
}

// The same for weights with two rotations: pairs of fp16 and their scales (see rotate_x_pair_kernel), in the room of
// launch_rotate_x's two planes.
static void launch_rotate_x_pair(const __half* x, float* xrot, int in, int batch, uint32_t block, uint32_t seed_p, uint32_t seed_r,
                                 cudaStream_t stream) {
    const int wide_cols = block <= 256 ? 256 : static_cast<int>(block);
    auto* const kernel = wide_cols == 256 ? rotate_x_pair_kernel<1> : (wide_cols == 512 ? rotate_x_pair_kernel<2> : rotate_x_pair_kernel<4>);
    launch_pdl(kernel, dim3((2 * batch * ((in + wide_cols - 1) / wide_cols) + 3) / 4), dim3(128), kRotatePairSmem, stream, x,
               reinterpret_cast<uint32_t*>(xrot), xrot + static_cast<size_t>(8) * in, in, batch, static_cast<int>(block), seed_p, seed_r,
               1.0f / std::sqrt(static_cast<float>(block)), reinterpret_cast<uintptr_t>(x) % 16 == 0 ? 1 : 0);
}

// ---- allocation-free variant ---------------------------------------------------------------
// Same two kernels, but the scratch (rotated activation, split-K partial sums, arrival
// counters) lives in a fixed array inside the library image instead of a buffer the handle
// allocated.  Every GPU that loads the library carries these bytes until the process exits.
constexpr size_t kStaticScratchBytes = size_t(2) << 20;  // 2 MiB
static __device__ __align__(256) unsigned char g_gemv_static_scratch[kStaticScratchBytes];

size_t gemv_static_scratch_capacity() { return kStaticScratchBytes; }

// Device address of the array on the current device.  In host code the array's name is only
// a handle for the runtime, not an address a kernel could use, so the address is looked up
// once per device (with that device current) and cached.
static void* static_scratch_address() {
    static void* cached[64] = {nullptr};
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && cached[dev]) return cached[dev];
    void* ptr = nullptr;
    TQ_CUDA(cudaGetSymbolAddress(&ptr, g_gemv_static_scratch));
    TQ_REQUIRE(ptr != nullptr, "tq8_gemv: static scratch has no device address");
    if (dev >= 0 && dev < 64) cached[dev] = ptr;
    return ptr;
}

// The same address for the other decode kernel's allocation-free variant.
void* gemv_static_scratch_address() { return static_scratch_address(); }

void launch_tq8_gemv_static(const uint8_t* codes, const float* norms, const float* table, const __half* x, __half* y,
                            int out, int in, int batch, uint32_t block, int n_planes, float pair_unit, uint32_t seed_p,
                            uint32_t seed_r, unsigned int* status, int sm_count, cudaStream_t stream) {
    // Which layers are taken, and what an error counts: those whose planes would fit as partial-sum slots of their own.  (Layers with
    // two rotations need less by now; a layer that was refused here still is.)
    const size_t asked = scratch_bytes(out, in, n_planes, chunk_count(in) * n_planes), need = gemv_scratch_bytes(out, in, n_planes);
    if (asked > kStaticScratchBytes)
        throw Error("allocation-free forward: this layer needs " + std::to_string(asked) +
                    " bytes of scratch, the built-in array holds " + std::to_string(kStaticScratchBytes));
    void* scratch = static_scratch_address();
    // The array is shared by every call and keeps what the last one left.  The arrival
    // counters are the only part that must read zero at kernel start; the kernels re-zero
    // them on exit, but a call cut short (device error, aborted process sharing the context)
    // would leave them dirty, so they are cleared here, in stream order.
    const size_t xrot_bytes = align256(static_cast<size_t>(n_planes) * 8 * in * sizeof(float));
    if (need > xrot_bytes) {
        const int n_row_tiles = (out + 15) / 16;
        const size_t counter_bytes = align256(static_cast<size_t>(n_row_tiles) * kWarps * sizeof(unsigned int));
        TQ_CUDA(cudaMemsetAsync(static_cast<uint8_t*>(scratch) + need - counter_bytes, 0, counter_bytes, stream));
    }
    launch_tq8_gemv(codes, norms, table, x, y, out, in, batch, block, n_planes, pair_unit, seed_p, seed_r, scratch, status, sm_count,
                    stream);
}

}  // namespace tq
