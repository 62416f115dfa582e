// Fused TQ8 dequantise + GEMM for prefill (tens to thousands of activation rows) on the
// 5th-generation tensor cores: tcgen05.mma with the accumulator in tensor memory.
//
// Replaces, for large batches, the reference's tq_dequant_mm Metal kernel and its host wrapper
// (metal/turboquant_dequant_mm.metal:152-313, src/dequantizer.cpp:606-721):
//   y[m, r] = fp16( norm[r] * sum_j W~[r, j] * fp16(x[m, j]) ),  fp32 accumulate.
//
// Same algebra as the decode kernel: the activation is rotated once (forward WHT of every block
// of every row, written as fp16 by rotate_rows_f16_kernel), and the weight side is a table
// lookup per code:   y[m, r] = norm[r] * inv_scale * sum_j table[code[r, j]] * xrot[m, j].
// Dual-rotation weights run as twice the K into the same accumulator (primary centroids
// against x rotated with the primary seed, residual centroids against x rotated with the residual
// seed).
//
// One CTA computes a 128 (weight rows) x 256 (activation rows, or fewer) tile of y^T:
//   D[128 x 256] (TMEM, fp32) += A[128 x 64] (weights, fp16, TMEM) . B[256 x 64]^T (xrot, fp16, smem)
// per 64-column K block, as four tcgen05.mma (M 128, N 256, K 16) issued by one thread.
//   A pipeline stage is 128 K columns (two 64-column K blocks), the ring has up to four stages.
//   warps 0-23 producers in three groups of eight (or two, or one, see gemm_groups); group g takes the stages g, g + 3, ...: codes HBM ->
//              registers (the group's next stage, as the present one's are used up) -> lookup (lane-private fp16 table in
//              shared memory) -> weight tile in TENSOR memory (tcgen05.st, 64 columns of fp16 pairs per
//              stage).  The store's 16x256b shape takes registers in the fragment order (lane / 4 = row,
//              lane % 4 = columns), so a code load of a warp is 512 contiguous bytes; with a row per lane
//              (32x32b) it touched 32 lines of 64 bytes, and the first-level cache, which the lookups
//              also load with a wavefront per 32 weights, was the bound (5120 x 55296: 110 -> 89 us at 32
//              rows, 644 -> 547 us at 1024).  The K order this gives is free: the rotation kernels write
//              the activations in the same one (k_position).
//   warp 25    activation tiles: the rotation kernel stores xrot in operand-tile order, so a K block
//              of a tile is one contiguous bulk copy (cp.async.bulk, mbarrier complete_tx) of 128
//              bytes per activation row of the tile
//   warp 24    waits for a stage (ONE barrier collects the producers' arrivals and the copies' bytes); one
//              elected lane issues its eight MMAs and commits to the stage's "empty" barrier.  This serial
//              chain (wait, fence, issue, commit) bounds the kernel when the MMAs are short, hence few and
//              long stages.
//   warps 26-29 (three groups) epilogue: tcgen05.ld the accumulator, scale by norm * inv_scale, store fp16, beside the
//              next tile's products (up to 128 activation rows: two accumulators in turn; above, the next
//              tile's first MMA waits until this one is read).  A CTA of one or two groups has one tile: its producers drain it, 32 rows each
// A CTA per SM walks the output tiles (of a single matrix; a group's matrices have a CTA per tile) and its ring of stages runs on from tile to tile: with a CTA per
// tile, set-up, first loads and epilogue took 8 to 18 of 47 thousand cycles (5120 x 55296: 89 -> 76 us at
// 32 rows, 544 -> 464 us at 1024).  Up to 64 rows the producers bound it: some 420 cycles per 128 x 64 weights, of which the shared-memory
// pipe is taken for 320 (256 of lookups, 64 of code loads) and 32 to 128 more by the activation tile; it is busy for 63 % of a launch at 32 rows.  At
// 16 rows that is 86 % of what the memory delivers.  At 256 it is that pipe: lookups, code loads, the activation tile's write and its read.  What a call
// costs besides its stages is some 6 us where the next kernel's CTAs are set up beside the last one's (gemm_groups), 8 us otherwise: two or three waits of 1.1 us
// for the end of the kernel in front, the rotation, the first activation tile, the epilogue, the split sums.
// The activation tile is as tall as the rows it really has (in steps of 16): a decode batch of 9..64
// rows costs a short MMA and a short copy, so the codes are streamed once whatever the batch.
// The dequantised weights never touch HBM; a weight tile is looked up once per 256 activation
// rows.  Roofline: tensor pipe (2 * M * out * in flops), with the table lookups (one shared-memory
// load per weight per 256 activation rows) as the competing pipe.
//
// Shared-memory layout of the activation operand (K-major, no swizzle): 8 x 8 fp16 core matrices of
// 128 contiguous bytes (8 rows of 16 bytes); core matrices adjacent in K are 128 bytes apart
// (leading byte offset), 8-row groups are 1024 bytes apart (stride byte offset).
//
// Every wait is bounded: a barrier that does not complete within 0.2 s sets the status word and
// an abort flag, after which all warps fall through to the exit path (which still frees the
// tensor memory).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "tq_common.cuh"
#include "tq_kernels.cuh"

namespace tq {

namespace {

constexpr int kTileRows = 128;  // weight rows per CTA (MMA M)
constexpr int kTileTok = 256;   // activation rows per CTA (MMA N)
constexpr int kBlockK = 64;     // columns of a K block
constexpr int kSubPerStage = 2; // K blocks per pipeline stage: a stage is 128 K columns
constexpr int kStagesMax = 4;   // ring of stages: weight tiles in tensor memory (4 x 64 columns), activation tiles in shared memory (as many as fit)
constexpr int kGroupsMax = 3;   // producer groups of eight warps: group g dequantises the stages g, g + groups, ...
constexpr int kEpilogueWarps = 4;
// With three groups four more warps drain the accumulators beside the next tile's products; a CTA of one or two groups has one tile, which its producers
// drain when they are through with it.
__host__ __device__ constexpr int gemm_threads(int groups) { return groups * 256 + 64 + (groups == kGroupsMax ? 32 * kEpilogueWarps : 0); }
constexpr uint32_t kLutBytes = 256 * 32 * 4;           // 256 entries x 32 lane copies x two fp16
constexpr uint32_t kTmemCols = 512;   // accumulators: columns 0..255 (two of up to 128 columns, or one); weight tiles: 4 stages x 64 columns from 256 on
constexpr uint32_t kTmemAColumn = 256;
constexpr uint32_t kTmemASubCols = kBlockK / 2;                    // one K block: two fp16 per 32-bit column
constexpr uint32_t kTmemAStageCols = kSubPerStage * kTmemASubCols;
// One group: 256 columns, so that two CTAs share an SM: an accumulator of 64 or 128 columns, the rest weight tiles (three stages or two).
__host__ __device__ constexpr uint32_t one_group_a_column(uint32_t rows) { return rows <= 64 ? 64 : 128; }
__host__ __device__ constexpr uint32_t one_group_stages(uint32_t rows) { return (256 - one_group_a_column(rows)) / kTmemAStageCols; }
constexpr uint32_t kLutWin = 0x800u;  // window address of the lookup tables (an immediate of the lookup's load)
// Everything an SM can give one CTA: tables at kLutWin, then three 64 KB stages for a 256-row tile.
constexpr size_t kGemmSmemBytes = 232448 - 512;
// What a launch of m activation rows needs of it (an SM is set up faster for less: 3584 x 37888 at 16 rows 32.9 us with all of it, 32.4 so).
size_t gemm_smem_bytes(long m, int groups) {
    const int rows = static_cast<int>(std::min<long>(kTileTok, (m + 15) / 16 * 16));
    const int stages = groups == 1 ? static_cast<int>(one_group_stages(static_cast<uint32_t>(rows))) : kStagesMax;
    return std::min(kGemmSmemBytes, kLutWin + kLutBytes + static_cast<size_t>(stages) * kSubPerStage * rows * kBlockK * 2);
}
// Producer groups of a single product.  Three stream codes fastest (5120 x 55296 at 32 rows 60 us, 66 with two), but 30 warps of 64 registers fill the SM: the
// CTA is set up, makes its table and fetches its first codes only when the rotation in front is gone, and the kernels around it wait for its end in
// turn.  18 warps leave room for CTAs of the rotation and of the split sums, and all of a call's kernels are there when the one in
// front of them ends: what lies between two of them is one wait (1.1 us).  So two groups where a CTA has one tile and few stages, that is less to
// stream than the set-up costs.  Calls in a graph, three groups (one kernel after the other) -> two: 4096 x 4096 at 16 rows (eight stages) 11.5 -> 9.2 us,
// 3584 x 3584 at 64 12.7 -> 11.7 (at 256 20.3 -> 17.4), 3072 x 18944 at 64 (24) 19.0 -> 17.7, 3584 x 18944 at 16 (28) 19.8 -> 19.0, 18944 x 3584 at 16 (30)
// 21.6 -> 20.9; beyond that the other way round, at 64 rows a little earlier: 28672 x 2048 (25) 24.4 -> 25.9, 4096 x 18944 (32) 23.3 -> 24.0.
int gemm_groups(long n_tiles, int k_blocks, long m, int sm_count) {
    const int stages = (k_blocks + kSubPerStage - 1) / kSubPerStage;
    return n_tiles <= sm_count && stages <= (m <= 32 ? 30 : 24) ? 2 : kGroupsMax;
}
// Producer groups of a launch of several matrices, each of them `ctas` CTAs (tiles x K splits) of `stages` stages.  One group (two CTAs to an SM, up to 128 rows: its tensor memory holds an
// accumulator of so many) hides a CTA's beginning and end behind the other's stages, but takes nearly twice as long for a stage.  So where the CTAs outnumber the SMs (otherwise: two) it is
// compared with CTAs that have an SM to themselves, in stages, a CTA's beginning and end as 20 of them: 2 stages + 20 a CTA on 2 x SMs, stages + 20 on the SMs; in waves, or where the matrices' CTAs
// are not equally long by their sum, but no less than the longest.  Three groups and one, 16 rows, weights from memory: 4096 -> 2 x 14080 (220 CTAs of 32 stages) 39.9 and 34.1 us, 2048 -> 2 x 28160 (440 of 16)
// 39.4 and 36.5, 4096 -> 2 x 38400 (600 of 32) 94.0 and 88.9, 5120 -> 5120 + 1024 + 1024 (120 of 13, 160 of 4) 21.0 and 16.6; the other way round 8192 -> 2 x 22528 (352 of 64) 98.3 and 110.8, 4096 ->
// 2 x 28160 (440 of 32) 60.2 and 65.7, two rotations 5120 -> 2 x 22528 (352 of 80) 86.7 and 103.4, 8192 -> 8192 + 1024 + 1024 (128 of 64, 288 of 7) 41.6 and 47.5.
// Of CTAs alone on an SM, three groups stream codes faster, two are set up beside the rotation.  Up to 64 rows (32 of two rotations) three: two would take 104.3 us for the first of those four, 62.1, 92.7 and
// 42.6; above that the tensor cores' share grows and two: two rotations 4096 -> 2 x 19200 at 128 rows 98.1 -> 92.9, 2048 -> 2 x 19200 at 64 48.0 -> 46.2.  Above 128 rows two as well, but three
// where matrices of unequal splits leave long CTAs to a matrix that is split itself, beside short ones of the others: the long ones' codes are the launch's time.  Two groups and three, two
// rotations, weights from memory: 8192 -> 8192 + 1024 + 1024 (64 stages, 7, 7) at 192 rows 86.9 and 82.8 us, 6144 -> 6144 + 1024 + 1024 (32, 5, 5) at 256 77.3 and 73.6, 5120 -> 5120 + 1024 +
// 1024 (27, 4, 4) at 224 62.4 and 59.3, 4096 -> 4096 + 1024 + 1024 (32, 7, 7) at 384 66.9 and 65.4.  The other way round: 14336 -> 2048 + 512 (25, 6) at 192 46.0 and 47.6, 4096 -> 4096 + 1024 +
// 1024 (16, 4, 4) at 192 45.4 and 47.5, 4096 -> 8192 + 2048 (32, 6) at 129 38.1 and 39.3 (at 192 47.4 and 46.1); not split, 5120 -> 5120 + 1024 + 1024 (80, 9, 9) at 512 83.3 and 84.7; equal
// splits, 8192 -> 2 x 4096 (32, 32) at 256 74.7 and 77.3.
constexpr long kGroupOneRows = 128, kCtaEndsInStages = 20;
struct GroupCallCtas {
    long ctas[4];
    int stages[4], n, least;   // least: the smallest count of K splits
    bool unequal;              // splits
};
int group_call_groups(const GroupCallCtas& c, long m, int n_planes, int sm_count) {
    long all = 0, longest = 0;
    for (int i = 0; i < c.n; ++i) {
        all += c.ctas[i];
        longest = std::max<long>(longest, c.stages[i]);
    }
    if (m > kGroupOneRows) return c.unequal && c.least > 1 && longest > 26 ? kGroupsMax : 2;
    if (all <= sm_count) return 2;
    auto time = [&](long per_stage, long slots) {
        if (!c.unequal) return (all + slots - 1) / slots * (per_stage * longest + kCtaEndsInStages);
        long sum = 0;
        for (int i = 0; i < c.n; ++i) sum += c.ctas[i] * (per_stage * c.stages[i] + kCtaEndsInStages);
        return std::max(per_stage * longest + kCtaEndsInStages, sum / slots);
    };
    if (time(2, 2 * sm_count) <= time(1, sm_count)) return 1;
    return m * n_planes <= 64 ? kGroupsMax : 2;
}
// An SM divides its 228 KB between shared memory and first-level cache anew only when it is empty, and small kernels ask for little of it: the product's
// CTA did not come beside them.  So above 32 rows all three kernels of a call with one or two groups ask for what the product (two CTAs of one group) takes and 10 KB (7168 x 2048 at 64
// rows 14.3 -> 12.0 us, 8192 x 1024 12.6 -> 11.5).  Up to 32 rows not: 4096 x 4096 at 16, whose loads of codes then have less of the cache, 8.5 -> 9.1.  Percent; 0: no wish.
int gemm_carveout(long m, int groups) {
    if (m <= 32 || groups == kGroupsMax) return 0;
    const size_t kb = (gemm_smem_bytes(m, groups) / 1024 + 1) * (groups == 1 ? 2 : 1) + 10;
    return std::min(100, static_cast<int>(kb * 100 / 228 + 1));
}
constexpr unsigned long long kGemmWaitLimitNs = 200ull * 1000 * 1000, kGemmCopyLandNs = 1000ull * 1000;

// instruction descriptor: D fp32, A and B fp16, both K-major, M = 128, N = n (a multiple of 16 up to 256)
__host__ __device__ constexpr uint32_t instr_desc(uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | (static_cast<uint32_t>(kTileRows >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ unsigned long long timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait; gives up at once when another thread has already flagged a failure.  Its time begins when it does not find the phase over: a thread whose phase
// ends only when kernels in front are done waits for those first (griddepcontrol.wait), with no limit of its own, or their time would count.  (Without
// a time to sleep: with 20 us of it 3584 x 37888 at 16 rows took 35.3 us instead of 34.2.)
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile unsigned int* abort_flag) {
    unsigned long long t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spin & 15) == 15 && *abort_flag) return false;
        if (spin == 64) t0 = timer_ns();
        if (spin > 64 && (spin & 63) == 0 && timer_ns() - t0 > kGemmWaitLimitNs) return false;
    }
}

// shared-memory matrix descriptor: K-major, no swizzle, LBO 128 B, SBO 1024 B, descriptor version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(128u >> 4) << 16) |
           (static_cast<uint64_t>(1024u >> 4) << 32) | (1ull << 46);
}

// Table lookup: `offset` = scaled code | lane offset; the table's window address is the immediate.
__device__ __forceinline__ uint32_t lut_load(uint32_t offset) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1 + 2048];" : "=r"(v) : "r"(offset));
    return v;
}
static_assert(kLutWin == 2048u, "lut_load's immediate is the tables' window address");

// D[tmem_d] (+)= A[tmem_a] . B[desc_b]^T : A from tensor memory (128 lanes x 8 columns of fp16 pairs),
// B from shared memory.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p; }"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// 16 lanes x 32 columns, four blocks of 8 columns side by side: registers 4 i + (0, 1) are row lane / 4, columns
// 8 i + 2 (lane % 4) and the next; registers 4 i + (2, 3) the same columns of row lane / 4 + 8.
__device__ __forceinline__ void tmem_st_16x256b(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        :
        : "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// The same, two blocks of 8 columns.
__device__ __forceinline__ void tmem_st_16x256b(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :
                 : "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// 16 bytes of codes where `want`, in place: the registers are neither copied nor chosen between.  Codes are read once per 256
// activation rows: they pass by the first-level cache.
__device__ __forceinline__ void load_codes16_if(uint4& v, const uint8_t* p, bool want) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %5, 0; @p ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4]; }"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(p), "r"(static_cast<uint32_t>(want)));
}
// One lane of a converged warp.  The compiler knows that it is one, so that the operands of the tensor and copy instructions behind
// it are uniform; behind `lane == 0` each MMA took some hundred cycles to issue (3584 x 37888 at 16 rows 38.3 us, 35.4 with this).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(p));
    return p != 0;
}
// Waits for this thread's tensor-memory stores and orders them before the barrier arrival that follows.
__device__ __forceinline__ void tmem_st_publish() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
// Arrives on the barrier once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Where column c of a 64-column K block stands in the operands.  A producer lane holds 16 consecutive codes of a row
// (columns 16 q .. of lane quarter q) and the tensor-memory store takes four fp16 of every lane for each block of 16: the
// q-th four of block i are columns 16 q + 4 i and on.  Any order does as long as both operands share it.
__host__ __device__ constexpr int k_position(int c) { return 16 * ((c >> 2) & 3) + 4 * (c >> 4) + (c & 3); }

// ---- activation rotation to fp16, written in operand-tile order --------------------------------
// One warp per (plane, row, WHT block): xrot = fp16( FWHT(sign o fp16(x)) / sqrt(bs) ).
// Output layout: [plane][row tile of 256][K block of 64][32 KB tile], the tile being exactly the
// shared-memory image the GEMM wants (8 x 8 core matrices: [row group 32][core column 8][row 8][8 fp16]),
// so that a CTA fetches an activation tile with ONE contiguous bulk copy.  The order of the 64 columns of a K block is
// the one in which the producers' tensor-memory store lays the weights down (k_position).  Rows past the last
// one are left as they are: they only feed accumulator columns that are never stored.
template <int E>
__global__ void __launch_bounds__(128) rotate_rows_f16_kernel(const __half* __restrict__ x, __half* __restrict__ xrot,
                                                              int in, long rows, int n_planes, uint32_t seed_p,
                                                              uint32_t seed_r, float inv_sqrt) {
    pdl_wait_release();   // x, and the scratch this kernel overwrites, belong to the kernels before it until they are done
    constexpr int BS = 32 * E;
    constexpr int V = E < 4 ? E : 4;  // halves per vector store (k_position keeps groups of four together)
    const int lane = threadIdx.x & 31;
    const long blocks_per_row = in / BS;
    const long total = static_cast<long>(n_planes) * rows * blocks_per_row;
    const long warp = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (warp >= total) return;
    // consecutive warps take consecutive rows of the same block: their stores fill whole lines
    const int plane = static_cast<int>(warp / (rows * blocks_per_row));
    const long rem = warp - static_cast<long>(plane) * rows * blocks_per_row;
    const long blk = rem / rows, row = rem - blk * rows;
    const uint32_t seed = plane ? seed_r : seed_p;
    behind_wait(x);
    const __half* src = x + row * in + blk * BS + lane * E;
    float v[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = __half2float(src[j]) * sign_value(seed, static_cast<uint32_t>(lane * E + j));
    warp_fwht<E>(v, lane);
    const long n_row_tiles = (rows + kTileTok - 1) / kTileTok;
    const long kb_per_plane = in / kBlockK;
    const long rt = row / kTileTok, rin = row - rt * kTileTok;
#pragma unroll
    for (int j0 = 0; j0 < E; j0 += V) {
        const long col = blk * BS + lane * E + j0;
        const long kb = col / kBlockK, pos = k_position(static_cast<int>(col - kb * kBlockK));
        const long tile = (static_cast<long>(plane) * n_row_tiles + rt) * kb_per_plane + kb;
        __half* dst = xrot + tile * (kTileTok * kBlockK) + (((rin >> 3) * 8 + (pos >> 3)) * 8 + (rin & 7)) * 8 + (pos & 7);
        __align__(8) __half h[V];
#pragma unroll
        for (int j = 0; j < V; ++j) h[j] = __float2half_rn(v[j0 + j] * inv_sqrt);
        if constexpr (V == 4) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
        else if constexpr (V == 2) *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(h);
        else dst[0] = h[0];
    }
}

// The butterfly stages of a block above 128 columns, between a lane's chunks.
template <int CHUNKS>
__device__ __forceinline__ void rotate_chunks_above(float (&v)[CHUNKS][8]) {
#pragma unroll
    for (int h = 1; h < CHUNKS; h <<= 1)
#pragma unroll
        for (int i = 0; i < CHUNKS; i += 2 * h)
#pragma unroll
            for (int c = i; c < i + h; ++c)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float a0 = v[c][j], b0 = v[c + h][j];
                    v[c][j] = __fadd_rn(a0, b0);
                    v[c + h][j] = __fsub_rn(a0, b0);
                }
}
// A lane's rotated columns of a row to their places among the 8 rows in shared memory.  The lane's two groups of four columns are 16 positions
// apart; lane ^ 2 holds the ones next to them.  The lanes swap one group each, so that every lane stores a whole core-matrix row of 8.
template <int CHUNKS>
__device__ __forceinline__ void rotated_row_out(float (&v)[CHUNKS][8], float inv_sqrt, int lane, int wib, unsigned live, uint4* s_rows) {
    const bool odd = (lane & 2) != 0;   // of the pair: the upper four of the row
    const int pos = 16 * (2 * (lane & 1) + (odd ? 1 : 0)) + 8 * ((lane >> 2) & 1);   // k_position of the row's first column
    const int cc = pos >> 3;
    uint4* const put = s_rows + (lane >> 3) * 64 + cc * 8 + (wib ^ cc);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[c][j] *= inv_sqrt;
        const uint4 h = pack_halves(v[c]);
        const uint2 keep = odd ? make_uint2(h.z, h.w) : make_uint2(h.x, h.y), give = odd ? make_uint2(h.x, h.y) : make_uint2(h.z, h.w);
        const uint2 got = make_uint2(__shfl_xor_sync(live, give.x, 2), __shfl_xor_sync(live, give.y, 2));
        put[256 * c] = odd ? make_uint4(got.x, got.y, keep.x, keep.y) : make_uint4(keep.x, keep.y, got.x, got.y);
    }
}

// The same with 16-byte accesses, for any WHT block: a warp takes CHUNKS x 256 columns of a row (one block of 512 or
// 1024 columns, or the blocks of 256 columns), lane l the 8 columns 8l..8l+7 of each chunk; butterfly stages below 8 stay in
// the lane, the next are lane exchanges, those above 128 stay in the lane again (the add tree of warp_fwht).  The 8 warps of
// a CTA take 8 consecutive rows, and `row_steps` such groups one after the other: the signs are the same for all rows.  The 8
// rows of a K block are 1 KB of the operand tile: they meet in shared memory (slots of a core matrix's rows permuted by its column: no
// bank conflicts) and leave as contiguous stores; a lane's own 16-byte pieces of a row are 128 bytes apart.
// Instructions bound it, a third of the time the lane exchanges alone: 286 per 256 columns of a row with the exchanges in a loop, 64-bit places
// and the signs of the lanes found anew for every row; 218 so.  2048 x 18944: 53 -> 44 us under the
// profiler, 64 x 18944 with the product behind it 27.5 -> 25.2.  With two columns an instruction (fp32 pairs): 302, the pairs have to be made.
template <int CHUNKS, int STAGES>
__device__ __forceinline__ void rotate_rows_wide_body(const __half* __restrict__ x, __half* __restrict__ xrot, int in, int rows, int block, uint32_t seed,
                                                      unsigned col_group, unsigned row_group, float inv_sqrt, int row_steps, uint4 (*s_rows)[256 * CHUNKS]) {
    // x, and the scratch this kernel overwrites, belong to the kernels before it until they are done.  A CTA of few rows waits first, so that the
    // product's CTAs may come and set themselves up beside it: with the signs in front 8192 x 512, block 512, took 13.6 us at 100 rows instead
    // of 11.8 (with the older loop 13.0), 1024 x 512, block 64, 10.8 at 128 instead of 10.0.  Many rows' CTAs, wave after wave, have them made by then.
    const bool wait_first = CHUNKS == 1 || row_steps == 1;
    if (wait_first) pdl_wait_release();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int col = static_cast<int>(col_group) * 256 * CHUNKS + 8 * lane;
    // in is a multiple of 64 and of the block: whole lanes only, and exchanges stay inside a block.  (A group of several
    // chunks is a whole block, all of it inside the row.)
    const bool have = col < in;
    const unsigned live = __ballot_sync(0xffffffffu, have);
    uint4 signs[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) signs[c] = chunk_signs(seed, static_cast<uint32_t>(col + 256 * c), block);
    float side[STAGES];
#pragma unroll
    for (int k = 0; k < STAGES; ++k) side[k] = (lane & (1 << k)) != 0 ? -1.0f : 1.0f;
    const int kb_per_plane = in / kBlockK;
    // in the other direction: thread -> K block (of four per chunk), core column and row
    const int t = threadIdx.x & 63, tc = t >> 3, tr = t & 7;
    const uint4* get = &s_rows[0][(threadIdx.x >> 6) * 64 + tc * 8 + (tr ^ tc)];
    constexpr int kOther = 256 * CHUNKS;   // to the buffer of the next step
    int flip = kOther;
    const int first = static_cast<int>(row_group) * 8 * row_steps, last = min(rows, first + 8 * row_steps);
    const __half* src = x + static_cast<size_t>(first + wib) * in + col;
    const size_t src_step = static_cast<size_t>(in) * 8;
    const int kb_at = static_cast<int>(col_group) * 4 * CHUNKS + static_cast<int>(threadIdx.x >> 6);
    auto place = [&](int row8) {
        return xrot + (static_cast<size_t>(row8 / kTileTok) * kb_per_plane + kb_at) * (kTileTok * kBlockK) + ((row8 % kTileTok >> 3) * 64 + t) * 8;
    };
    __half* dst = place(first);
    if (!wait_first) pdl_wait_release();
    behind_wait(src);
    // a row's loads are on their way while the one before it is worked on (not of blocks of 1024, which fill the registers)
    constexpr bool kAhead = CHUNKS <= 2;
    uint4 next[CHUNKS];
    auto load = [&](const __half* from, bool there) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) next[c] = there ? *reinterpret_cast<const uint4*>(from + 256 * c) : make_uint4(0, 0, 0, 0);
    };
    if (kAhead) load(src, have && first + wib < rows);
    for (int row8 = first; row8 < last; row8 += 8) {
        if (have && row8 + wib < rows) {
            if (!kAhead) load(src, true);
            uint4 raw[CHUNKS];
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) raw[c] = next[c];
            if (kAhead) load(src + src_step, row8 + 8 + wib < last);
            float v[CHUNKS][8];
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) rotate_chunk_fixed<STAGES>(v[c], raw[c], signs[c], side, live);
            rotate_chunks_above<CHUNKS>(v);
            rotated_row_out<CHUNKS>(v, inv_sqrt, lane, wib, live, &s_rows[flip == kOther ? 0 : 1][0]);
        }
        __syncthreads();   // (the other buffer's readers are past it when it is written again)
        if (row8 + tr < rows) {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c)
                if (kb_at + 4 * c < kb_per_plane) *reinterpret_cast<uint4*>(dst + static_cast<size_t>(4 * c) * (kTileTok * kBlockK)) = get[256 * c];
        }
        get += flip;
        flip = -flip;
        src += src_step;
        dst += 64 * 8;
        if ((row8 + 8) % kTileTok == 0) dst = place(row8 + 8);
    }
}
// The same of one group of 8 rows a CTA, for few rows (FEW): the kernel lies between two others whose ends are waited for, so what counts is the time from one
// wait to the next.  It lets the product's CTAs come at once - beside it they make their tables and fetch their first codes - and has its signs
// in hand when its own wait is over.  32 registers (48 and 64 with two and four chunks): three CTAs of it fit beside a product's, where four with 40 kept it
// away: 8192 x 2048 at 64 rows 14.0 -> 12.4 us, 4096 x 4096 12.8 -> 11.4.
template <int CHUNKS, int STAGES>
__device__ __forceinline__ void rotate_rows_few_body(const __half* __restrict__ x, __half* __restrict__ xrot, int in, int rows, int block, uint32_t seed,
                                                     unsigned col_group, unsigned row_group, float inv_sqrt, uint4* s_rows) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, row8 = 8 * static_cast<int>(row_group);
    const int col = static_cast<int>(col_group) * 256 * CHUNKS + 8 * lane;
    const bool have = col < in;   // (see above)
    const unsigned live = __ballot_sync(0xffffffffu, have);
    uint4 signs[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) signs[c] = chunk_signs(seed, static_cast<uint32_t>(col + 256 * c), block);
    asm volatile("griddepcontrol.wait;" ::: "memory");   // x, and the scratch that is overwritten, belong to the kernels before until they are done
    behind_wait(x);
    if (have && row8 + wib < rows) {
        const __half* const src = x + static_cast<size_t>(row8 + wib) * in + col;
        uint4 raw[CHUNKS];
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) raw[c] = *reinterpret_cast<const uint4*>(src + 256 * c);
        float side[STAGES];
#pragma unroll
        for (int k = 0; k < STAGES; ++k) side[k] = (lane & (1 << k)) != 0 ? -1.0f : 1.0f;
        float v[CHUNKS][8];
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) rotate_chunk_fixed<STAGES>(v[c], raw[c], signs[c], side, live);
        rotate_chunks_above<CHUNKS>(v);
        rotated_row_out<CHUNKS>(v, inv_sqrt, lane, wib, live, s_rows);
    }
    __syncthreads();
    const int t = threadIdx.x & 63, tc = t >> 3, tr = t & 7, kb_per_plane = in / kBlockK;
    const int kb_at = static_cast<int>(col_group) * 4 * CHUNKS + static_cast<int>(threadIdx.x >> 6);
    if (row8 + tr < rows) {
        __half* const dst = xrot + (static_cast<size_t>(row8 / kTileTok) * kb_per_plane + kb_at) * (kTileTok * kBlockK) + ((row8 % kTileTok >> 3) * 64 + t) * 8;
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c)
            if (kb_at + 4 * c < kb_per_plane)
                *reinterpret_cast<uint4*>(dst + static_cast<size_t>(4 * c) * (kTileTok * kBlockK)) = s_rows[256 * c + (threadIdx.x >> 6) * 64 + tc * 8 + (tr ^ tc)];
    }
}
// The lane exchanges of a block as a constant of the loop over rows.
template <int CHUNKS, bool FEW>
__device__ __forceinline__ void rotate_rows_wide(const __half* __restrict__ x, __half* __restrict__ xrot, int in, long rows, int block, uint32_t seed_p,
                                                 uint32_t seed_r, float inv_sqrt, int row_steps) {
    __shared__ __align__(16) uint4 s_rows[FEW ? 1 : 2][256 * CHUNKS];   // [step parity][K block][core column][row slot]
    const unsigned groups_per_row = (static_cast<unsigned>(in) + 256 * CHUNKS - 1) / (256 * CHUNKS);
    const unsigned row_groups = static_cast<unsigned>((rows + 8 * row_steps - 1) / (8 * row_steps));
    // blockIdx.x -> (plane, column group, rows); warp -> row inside a group of 8
    const unsigned rg = blockIdx.x % row_groups, b = blockIdx.x / row_groups, cg = b % groups_per_row, plane = b / groups_per_row;
    const uint32_t seed = plane ? seed_r : seed_p;
    __half* const to = xrot + plane * ((static_cast<size_t>(rows) + kTileTok - 1) / kTileTok * (in / kBlockK) * (kTileTok * kBlockK));
    const int m = static_cast<int>(rows);
#define TQ_ROTATE_BODY(STAGES)                                                                                                        \
    if constexpr (FEW) rotate_rows_few_body<CHUNKS, STAGES>(x, to, in, m, block, seed, cg, rg, inv_sqrt, &s_rows[0][0]);               \
    else rotate_rows_wide_body<CHUNKS, STAGES>(x, to, in, m, block, seed, cg, rg, inv_sqrt, row_steps, s_rows)
    if constexpr (CHUNKS > 1) {
        TQ_ROTATE_BODY(5);
    } else {
        switch (block) {
            case 32: TQ_ROTATE_BODY(2); break;
            case 64: TQ_ROTATE_BODY(3); break;
            case 128: TQ_ROTATE_BODY(4); break;
            default: TQ_ROTATE_BODY(5); break;
        }
    }
#undef TQ_ROTATE_BODY
}
__host__ __device__ constexpr int rotate_ctas(int chunks, bool few) { return chunks == 1 ? (few ? 8 : 5) : !few ? 0 : chunks == 2 ? 5 : 4; }
template <int CHUNKS, bool FEW>
__global__ void __launch_bounds__(256, rotate_ctas(CHUNKS, FEW)) rotate_rows_f16_wide_kernel(const __half* __restrict__ x, __half* __restrict__ xrot,
                                                                   int in, long rows, int block,
                                                                   uint32_t seed_p, uint32_t seed_r, float inv_sqrt, int row_steps) {
    rotate_rows_wide<CHUNKS, FEW>(x, xrot, in, rows, block, seed_p, seed_r, inv_sqrt, row_steps);
}
// The same rows rotated for several matrices at once (their own seeds and destinations): blockIdx.y = matrix.
struct RotateGroupArgs {
    __half* xrot[4];
    uint32_t seed_p[4], seed_r[4];
};
template <int CHUNKS, bool FEW>
__global__ void __launch_bounds__(256, rotate_ctas(CHUNKS, FEW)) rotate_rows_f16_wide_group_kernel(const __half* __restrict__ x, const __grid_constant__ RotateGroupArgs g, int in,
                                                                         long rows, int block, float inv_sqrt, int row_steps) {
    rotate_rows_wide<CHUNKS, FEW>(x, g.xrot[blockIdx.y], in, rows, block, g.seed_p[blockIdx.y], g.seed_r[blockIdx.y], inv_sqrt, row_steps);
}

struct GemmArgs {
    const uint8_t* codes;   // joint bytes in 16 x 64 tiles (code_offset)
    const float* norms;     // [out]
    const float* table;     // [256] fp32; two rotations: [256] pairs of fp16
    const __half* xrot;     // rotated activation in operand-tile order (see rotate_rows_f16_kernel)
    __half* y;              // [m, out], activation rows y_stride elements apart
    long y_stride;
    float* partial;         // [k_splits, m, out] fp32 un-scaled partial sums (only when k_splits > 1)
    unsigned int* status;   // device error word (0 = ok)
    int out, in, m;
    int k_splits;           // CTAs along K per output tile (gridDim.z)
    float inv_scale;
};

// One CTA's work: K split bz of the output tiles t0, t0 + t_step, ... < t_end of matrix p.  Tile t is row tile t / n_tok,
// token tile t % n_tok: CTAs that run side by side share the codes of a few row tiles, which then come from HBM once however
// many token tiles there are.
//
// DUAL: weights with two rotations.  A table word holds both centroids of a byte as a pair of fp16, divided by the unit that inv_scale
// carries, and a stage is ONE 64-column block of codes: its first K block are the primary centroids, against x rotated with the
// primary seed, its second the residual ones.  A lookup serves both (as two planes one after the other the codes were read and looked up
// twice: 3584 x 3584, block 512, 20.2 us at 64 rows, 31.6 at 256 and 116 at 2048; 16.7, 24.8 and 93 so.  18944 x 3584 at 64 rows 50.7
// and 39.6.)
template <bool DUAL, int kGroups>
__device__ __forceinline__ void gemm_body(const GemmArgs& p, const int t0, const int t_step, const int t_end, const int bz) {
    constexpr int kProducerWarps = 8 * kGroups, kGemmThreads = gemm_threads(kGroups);
    constexpr int kMmaWarp = kProducerWarps;       // issues the MMAs, owns the tensor-memory allocation
    constexpr int kCopyWarp = kProducerWarps + 1;  // issues the activation-tile bulk copies
    extern __shared__ __align__(128) uint8_t gemm_smem[];
    __shared__ __align__(8) unsigned long long s_full[kStagesMax], s_empty[kStagesMax], s_accum_full[2], s_accum_empty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ unsigned int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_tok = (p.m + kTileTok - 1) / kTileTok;
    // Activation rows of a tile, rounded up to the MMA's granularity of 16: a short tile (a decode batch of 9..64 rows, or
    // the tail of a prefill) costs a short MMA and a short copy.
    auto tile_rows = [&](int t) { return min(kTileTok, ((p.m - (t % n_tok) * kTileTok) + 15) & ~15); };
    const int n_max = min(kTileTok, (p.m + 15) & ~15);
    const uint32_t tmem_cols = kGroups == 1 ? 256u : kTmemCols;
    const uint32_t a_column = kGroups == 1 ? one_group_a_column(static_cast<uint32_t>(n_max)) : kTmemAColumn;
    const int max_stages = kGroups == 1 ? static_cast<int>(one_group_stages(static_cast<uint32_t>(n_max))) : kStagesMax;
    const int n_acc = kGroups == kGroupsMax && n_max <= kTileTok / 2 ? 2 : 1;   // accumulators: with two, a tile is drained beside the next one's products
    const int n_local = t0 < t_end ? (t_end - t0 + t_step - 1) / t_step : 0;

    // ---- shared-memory map -------------------------------------------------------------------
    // [kLutWin, + 32 KB)            lookup table, at a fixed window address (it is an immediate of
    //                               the lookup's load instruction)
    // [after the table, end)        activation stages of two 64-column pieces, as many as fit, at most kStagesMax
    const uint32_t raw = smem_addr(gemm_smem);
    uint32_t dyn_bytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    const uint32_t stage0 = kLutWin + kLutBytes;
    const uint32_t piece_bytes = static_cast<uint32_t>(n_max) * (kBlockK * 2);   // a 64-column piece: a tile's first n_max rows are contiguous
    const uint32_t stage_bytes = kSubPerStage * piece_bytes;
    const uint32_t smem_end = raw + dyn_bytes;
    int n_st = smem_end > stage0 ? static_cast<int>((smem_end - stage0) / stage_bytes) : 0;
    if (n_st > max_stages) n_st = max_stages;
    if (raw > kLutWin || n_st < kGroups || n_max > (kGroups == 1 ? 128 : kTileTok)) {  // layout does not fit: refuse to run (nothing allocated yet)
        if (tid == 0) raise_status(p.status, 9u);
        return;
    }
    const uint32_t bar_full = smem_addr(&s_full[0]), bar_empty = smem_addr(&s_empty[0]);
    const uint32_t bar_acc_full = smem_addr(&s_accum_full[0]), bar_acc_empty = smem_addr(&s_accum_empty[0]);

    // the table's entries are asked for first: they come while the barriers and the tensor memory are set up
    constexpr int kTableSteps = (256 * 8 + kGemmThreads - 1) / kGemmThreads;
    float table_entry[kTableSteps];
#pragma unroll
    for (int k = 0; k < kTableSteps; ++k) table_entry[k] = __ldg(p.table + min(255, (tid + k * kGemmThreads) >> 3));
    if (tid == 0) {
        for (int s = 0; s < kStagesMax; ++s) {
            bar_init(bar_full + 8u * s, kProducerWarps / kGroups + 1);   // one arrival per producer warp of the group + the copy thread
            bar_init(bar_empty + 8u * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            bar_init(bar_acc_full + 8u * s, 1);
            bar_init(bar_acc_empty + 8u * s, kEpilogueWarps);
        }
        s_abort = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem_base)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        // The kernels behind may come: what they do in front of their waits reads nothing but weights.  Not before this CTA has its tensor memory,
        // which a CTA of the next product beside it may hold while that one waits for this kernel's end.  (With three groups there is no room for
        // them: let go at the end of the copies, small ones go to many SMs; let go here they crowd on the first that are free, 2048 x 37888 at 16 rows 21.3 -> 21.9.)
        if (kGroups < kGroupsMax) asm volatile("griddepcontrol.launch_dependents;");
    }
    // lookup table: entry e, lane copy l at kLutWin + e * 128 + l * 4, value (t, t) or (primary, residual) as fp16
#pragma unroll
    for (int k = 0; k < kTableSteps; ++k) {
        const int i = tid + k * kGemmThreads, e = i >> 3, c4 = (i & 7) * 4;
        const uint32_t v = DUAL ? __float_as_uint(table_entry[k]) : static_cast<uint32_t>(__half_as_ushort(__float2half_rn(table_entry[k]))) * 0x00010001u;
        if (i < 256 * 8)
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(kLutWin + static_cast<uint32_t>(e) * 128u + c4 * 4u), "r"(v)
                         : "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = s_tmem_base;
    volatile unsigned int* abort_flag = &s_abort;

    // Blocks of 64 columns of this CTA: a contiguous range.  A stage is two consecutive ones (the last one may be alone; with
    // two rotations one block and both its K blocks).  The stages of the CTA's tiles follow one another through the ring.
    const int kb_per_plane = p.in / kBlockK;
    constexpr int kBlocksPerStage = DUAL ? 1 : kSubPerStage;
    const int kb_base = static_cast<int>(static_cast<long>(kb_per_plane) * bz / p.k_splits);
    const int n_kb = static_cast<int>(static_cast<long>(kb_per_plane) * (bz + 1) / p.k_splits) - kb_base;
    const int n_it = (n_kb + kBlocksPerStage - 1) / kBlocksPerStage;

    auto epilogue = [&] {
        // ---- epilogue: TMEM lanes 32 * (warp & 3) .. + 31 (a lane = a weight row), 32 activation rows at a time ----
        constexpr int kColStep = kGroups == kGroupsMax ? 32 : 8 * kProducerWarps;   // a quarter of the warps for a quarter of the lanes
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (see bar_wait)
        int acc = 0;
        uint32_t par = 0u;
        for (int j = 0; j < n_local; ++j) {
            const int t = t0 + j * t_step;
            if (!__all_sync(0xffffffffu, bar_wait(bar_acc_full + 8u * acc, par, abort_flag) && !*abort_flag)) {
                raise_status(p.status, 8u);
                atomicExch(&s_abort, 1u);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int r = (t / n_tok) * kTileRows + 32 * (warp & 3) + lane;
            const int tok0 = (t % n_tok) * kTileTok;
            const int rows = min(kTileTok, p.m - tok0);
            const bool r_ok = r < p.out;
            const float scale = r_ok ? __ldg(p.norms + r) * p.inv_scale : 0.f;
            const uint32_t d_tmem = tmem_d + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + static_cast<uint32_t>(acc * (kTileTok / 2));
            const int c_first = kGroups == kGroupsMax ? 0 : 32 * (warp >> 2);
            __half* y = p.y + static_cast<size_t>(tok0 + c_first) * p.y_stride + r;
            float* part = p.partial + (static_cast<size_t>(bz) * p.m + tok0 + c_first) * p.out + r;   // (only used with k_splits > 1)
#pragma unroll 1
            for (int c0 = c_first; c0 < rows; c0 += kColStep) {
                uint32_t v[32];
                tmem_ld32(d_tmem + static_cast<uint32_t>(c0), v);
                if (kGroups == kGroupsMax && c0 + 32 >= rows) {   // the last read: the accumulator is free
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(bar_acc_empty + 8u * acc);
                }
                const int n = r_ok ? min(32, rows - c0) : 0;
                if (p.k_splits == 1) {
                    if (n == 32) {
#pragma unroll
                        for (int k = 0; k < 32; ++k) {
                            *y = __float2half_rn(__uint_as_float(v[k]) * scale);
                            y += p.y_stride;
                        }
                        if (kColStep > 32) y += (kColStep - 32) * p.y_stride;
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (k < n) y[k * p.y_stride] = __float2half_rn(__uint_as_float(v[k]) * scale);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k)
                        if (k < n) part[static_cast<size_t>(k) * p.out] = __uint_as_float(v[k]);
                    part += static_cast<size_t>(kColStep) * p.out;
                }
            }
            if (++acc == n_acc) { acc = 0; par ^= 1u; }
        }
    };

    if (warp < kProducerWarps) {
        // ---- producers ------------------------------------------------------------------------
        // Weight tile in tensor memory: lane = row of the tile, 64 columns per stage (two fp16 per
        // column, 128 K columns).  A warp may touch lanes 32 * (warp % 4) .. + 31.  The 24 producer
        // warps form three groups of eight (warp / 8); inside a group warp w takes the rows of lane
        // quarter w % 4 and the K block (w / 4) % 2 of the stage; group g dequantises the stages g,
        // g + 3, ...  A thread turns 64 codes, 16 of each of four rows, into fp16 pairs.  (With two rotations the two warps
        // of a lane quarter take 16 of its rows each, and 32 codes a thread make as many pairs.)
        // Three groups with one stage in registers each, not two with two: all warps share the pipe of the lookups, and a stage
        // costs a warp some 700 cycles beside them (its turn at the barriers, the tensor-memory stores, the next loads), in which
        // with two groups the pipe was idle half of the time.  5120 x 55296 at 32 rows 66.2 -> 61.6 us, 4096 x 4096 at 16 12.4 -> 12.1.
        const int sub = (warp >> 2) & 1;             // which K block of the stage, or which 16 rows
        constexpr int kLoads = DUAL ? 2 : 4;
        const int grp = warp >> 3;
        // The warp's rows are two code tiles of 16 x 64 bytes; lane (g, q) takes bytes 16 q .. of rows g and g + 8 of each:
        // a load of the warp is 512 contiguous bytes.  Tiles past the matrix repeat the last one (never stored).
        const int last_tile = (p.out - 1) >> 4;
        const size_t tile_row_bytes = static_cast<size_t>(code_tiles_per_row(p.in)) * kCodeTileBytes;
        const uint8_t* const code_lane = p.codes + (lane >> 2) * 64 + 16 * (lane & 3);
        const uint32_t a_taddr = tmem_d + (static_cast<uint32_t>(32 * (warp & 3) + (DUAL ? 16 * sub : 0)) << 16) + a_column +
                                 (DUAL ? 0u : kTmemASubCols * static_cast<uint32_t>(sub));

        // The group's next stage to fetch: its place in its tile, where its codes are, stages left.
        const int full_it = n_it - ((!DUAL && sub != 0 && (n_kb & 1)) ? 1 : 0);   // stages of a tile that have a block for this warp
        int f_it = grp, f_t = t0, left = (n_local * n_it - grp + kGroups - 1) / kGroups, f_lim = left > 0 ? full_it : 0;
        const uint8_t *f_ptr0 = code_lane, *f_ptr1 = code_lane;
        auto fetch_place = [&] {   // past the tile's last stage: the same place of the next tiles
            while (f_it >= n_it) {
                f_it -= n_it;
                f_t += t_step;
            }
            const int tile = (f_t / n_tok) * (kTileRows / 16) + 2 * (warp & 3) + (DUAL ? sub : 0);
            const size_t at = static_cast<size_t>(kb_base + kBlocksPerStage * f_it + (DUAL ? 0 : sub)) * kCodeTileBytes;
            f_ptr0 = code_lane + static_cast<size_t>(min(tile, last_tile)) * tile_row_bytes + at;
            if constexpr (!DUAL) f_ptr1 = code_lane + static_cast<size_t>(min(tile + 1, last_tile)) * tile_row_bytes + at;
        };
        uint4 c[kLoads];
#pragma unroll
        for (int i = 0; i < kLoads; ++i) c[i] = make_uint4(0, 0, 0, 0);
        if (left > 0) {
            fetch_place();
            const bool want = f_it < f_lim;
            load_codes16_if(c[0], f_ptr0, want);
            load_codes16_if(c[1], f_ptr0 + 512, want);
            if constexpr (!DUAL) {
                load_codes16_if(c[2], f_ptr1, want);
                load_codes16_if(c[3], f_ptr1 + 512, want);
            }
        }
        const uint32_t lane_c = static_cast<uint32_t>(lane) * 4u;   // bits outside the scaled code (7..14)
        // byte * 128 + lane offset in one dot-product instruction (a shift and a mask each on the logic pipe before)
        auto entry = [&](uint32_t word, int byte) { return lut_load(__dp4a(word, 128u << (8 * byte), lane_c)); };
        int slot = grp;                                             // ring slot of the stage, and the parity of its "empty" phase
        uint32_t par = 1u;
        bool ok = true;
        for (; left > 0; --left) {
            // The slot must have been read by the MMAs of its previous stage.  Asked for in front of the lookups and used behind them:
            // the answer queues behind the other warps' lookups.
            const uint32_t bar_e = bar_empty + 8u * slot;
            uint32_t ready;
            asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                         : "=r"(ready) : "r"(bar_e), "r"(par) : "memory");
            auto slot_free = [&] {
                if (!__all_sync(0xffffffffu, ready)) {
                    asm volatile("griddepcontrol.wait;" ::: "memory");   // (see bar_wait; a full ring in front of the first activation tile)
                    if (!__all_sync(0xffffffffu, bar_wait(bar_e, par, abort_flag))) {
                        raise_status(p.status, 6u);
                        atomicExch(&s_abort, 1u);
                        return false;
                    }
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");   // the MMAs' reads of the slot before the stores to it
                return true;
            };
            // where the group's next stage is
            f_it += kGroups;
            f_ptr0 += kGroups * kBlocksPerStage * kCodeTileBytes;
            if constexpr (!DUAL) f_ptr1 += kGroups * kBlocksPerStage * kCodeTileBytes;
            if (f_it >= n_it) {
                if (left > 1) fetch_place();
                else f_lim = 0;
            }
            const bool want = f_it < f_lim;
            const uint32_t st_addr = a_taddr + kTmemAStageCols * static_cast<uint32_t>(slot);
            if constexpr (DUAL) {
                // half a block's columns at a time: words i = 2 half and 2 half + 1 of either row, both planes
                const uint32_t w[8] = {c[0].x, c[0].y, c[0].z, c[0].w, c[1].x, c[1].y, c[1].z, c[1].w};
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t first[8], second[8];
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        const uint32_t word = w[4 * ((h >> 1) & 1) + 2 * half + (h >> 2)];
                        const int b0 = (h & 1) * 2;
                        const uint32_t e0 = entry(word, b0), e1 = entry(word, b0 + 1);
                        first[h] = __byte_perm(e0, e1, 0x5410);
                        second[h] = __byte_perm(e0, e1, 0x7632);
                    }
                    if (half == 1) {
                        load_codes16_if(c[0], f_ptr0, want);
                        load_codes16_if(c[1], f_ptr0 + 512, want);
                    }
                    if (half == 0 && !slot_free()) {
                        ok = false;
                        break;
                    }
                    tmem_st_16x256b(st_addr + 16u * half, first);
                    tmem_st_16x256b(st_addr + kTmemASubCols + 16u * half, second);
                }
            } else {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    // code tile `half`: 16 codes of row g and of row g + 8 -> fp16 pairs, word i of a row's four in column block i
                    const uint32_t w[8] = {c[2 * half].x, c[2 * half].y, c[2 * half].z, c[2 * half].w,
                                           c[2 * half + 1].x, c[2 * half + 1].y, c[2 * half + 1].z, c[2 * half + 1].w};
                    uint32_t packed[16];
#pragma unroll
                    for (int h = 0; h < 16; ++h) {
                        const uint32_t word = w[4 * ((h >> 1) & 1) + (h >> 2)];
                        const int b0 = (h & 1) * 2;  // bytes b0, b0 + 1 of the word
                        packed[h] = __byte_perm(entry(word, b0), entry(word, b0 + 1), 0x5410);
                    }
                    // used up: the group's next stage into the same registers
                    load_codes16_if(c[2 * half], half ? f_ptr1 : f_ptr0, want);
                    load_codes16_if(c[2 * half + 1], (half ? f_ptr1 : f_ptr0) + 512, want);
                    if (half == 0 && !slot_free()) {
                        ok = false;
                        break;
                    }
                    // (a tile's last stage may lack its second K block: what its warps store is not read)
                    tmem_st_16x256b(st_addr + (static_cast<uint32_t>(16 * half) << 16), packed);
                }
            }
            if (!ok) break;
            // every lane waits for its own stores, then one arrival per warp
            tmem_st_publish();
            __syncwarp();
            if (lane == 0) bar_arrive(bar_full + 8u * slot);
            slot += kGroups;
            if (slot >= n_st) {
                slot -= n_st;
                par ^= 1u;
            }
        }
        if constexpr (kGroups < kGroupsMax) {
            __syncwarp();
            epilogue();
        }
    } else if (warp == kCopyWarp) {
        // ---- activation tiles: one bulk copy per K block of the stage, as far ahead as the ring allows ----
        // One thread runs the whole loop; ring slot and phase are kept incrementally (no divisions on
        // this serial path).
        if (elect_one()) {
            // The rotated activations are the only input the kernel before this one produces (launched with the
            // programmatic-dependency attribute, the CTA has set up its barriers, tensor memory and tables and the
            // producers are already streaming codes meanwhile): wait for that kernel here.
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int slot = 0, filled = 0;
            uint32_t par = 1u;   // parity of the "empty" phase to wait for
            bool ok = true;
            for (int t = t0; ok && t < t_end; t += t_step) {
                const uint32_t b_bytes = static_cast<uint32_t>(tile_rows(t)) * (kBlockK * 2);
                for (int it = 0; it < n_it; ++it) {
                    ok = !*abort_flag;   // no copy once another thread has given up: it would be on its way when the CTA ends
                    if (!ok) break;
                    if (filled >= n_st && !bar_wait(bar_empty + 8u * slot, par, abort_flag)) {
                        raise_status(p.status, 6u);
                        atomicExch(&s_abort, 1u);
                        ok = false;
                        break;
                    }
                    ++filled;
                    const int nsub = DUAL ? kSubPerStage : min(kSubPerStage, n_kb - kSubPerStage * it);
                    const uint32_t bar = bar_full + 8u * slot;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(b_bytes * nsub) : "memory");
                    for (int sb = 0; sb < nsub; ++sb) {
                        const size_t tile = DUAL ? (static_cast<size_t>(sb) * n_tok + t % n_tok) * kb_per_plane + (kb_base + it)
                                                 : static_cast<size_t>(t % n_tok) * kb_per_plane + (kb_base + kSubPerStage * it + sb);
                        const __half* src = p.xrot + tile * (kTileTok * kBlockK);
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                         stage0 + static_cast<uint32_t>(slot) * stage_bytes + static_cast<uint32_t>(sb) * piece_bytes),
                                     "l"(src), "r"(b_bytes), "r"(bar)
                                     : "memory");
                    }
                    if (++slot == n_st) { slot = 0; par ^= 1u; }
                }
            }
            // every activation tile of this CTA is on its way: the kernel after this one may start setting up
            if (kGroups == kGroupsMax) asm volatile("griddepcontrol.launch_dependents;");
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ---- MMA issuer: the warp waits for a stage, one lane issues its MMAs and one commit ------------------------
        {
            int slot = 0, acc = 0;
            uint32_t par = 0u, acc_par = 1u;   // acc_par: parity of the "drained" phase to wait for
            bool ok = true;
            asm volatile("griddepcontrol.wait;" ::: "memory");   // (see bar_wait)
            for (int j = 0; ok && j < n_local; ++j) {
                const uint32_t idesc = instr_desc(static_cast<uint32_t>(tile_rows(t0 + j * t_step)));
                const uint32_t d_tmem = tmem_d + static_cast<uint32_t>(acc * (kTileTok / 2));
                if (j >= n_acc) {
                    if (!__all_sync(0xffffffffu, bar_wait(bar_acc_empty + 8u * acc, acc_par, abort_flag))) {
                        raise_status(p.status, 7u);
                        atomicExch(&s_abort, 1u);
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                for (int it = 0; it < n_it; ++it) {
                    if (!__all_sync(0xffffffffu, bar_wait(bar_full + 8u * slot, par, abort_flag))) {
                        raise_status(p.status, 7u);
                        atomicExch(&s_abort, 1u);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int nsub = DUAL ? kSubPerStage : min(kSubPerStage, n_kb - kSubPerStage * it);
                    const uint32_t a_tmem = tmem_d + a_column + kTmemAStageCols * static_cast<uint32_t>(slot);
                    const uint32_t b_stage = stage0 + static_cast<uint32_t>(slot) * stage_bytes;
                    if (elect_one()) {
#pragma unroll
                        for (int sb = 0; sb < kSubPerStage; ++sb) {
                            if (sb < nsub) {
                                const uint64_t desc0 = smem_desc(b_stage + static_cast<uint32_t>(sb) * piece_bytes);
#pragma unroll
                                for (int k = 0; k < kBlockK / 16; ++k)   // 256 bytes further along K per step: +16 in the address field
                                    umma_f16_ts(d_tmem, a_tmem + kTmemASubCols * sb + 8u * k, desc0 + static_cast<uint64_t>(16 * k), idesc,
                                                (it | sb | k) != 0 ? 1u : 0u);
                            }
                        }
                        umma_commit(bar_empty + 8u * slot);   // the slot (weights and activation) may be refilled once these MMAs are done
                    }
                    __syncwarp();
                    if (++slot == n_st) { slot = 0; par ^= 1u; }
                }
                if (ok && elect_one()) umma_commit(bar_acc_full + 8u * acc);
                __syncwarp();
                if (++acc == n_acc) { acc = 0; acc_par ^= 1u; }
            }
        }
        __syncwarp();
    } else if constexpr (kGroups == kGroupsMax) {
        epilogue();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // Given up: what the copying lane has started lands before the CTA's shared memory becomes another's.  Its barriers may miss arrivals of warps that are gone
    // and say nothing, so a time: a copy takes microseconds, and no further one starts.
    if (*abort_flag && warp == kCopyWarp) {
        const unsigned long long t0 = timer_ns();
        while (timer_ns() - t0 < kGemmCopyLandNs) {}
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_cols) : "memory");
    }
}

// gridDim.x CTAs walk the output tiles, gridDim.y = K splits.
template <bool DUAL, int GROUPS>
__global__ void __launch_bounds__(gemm_threads(kGroupsMax), 1) tq8_gemm_kernel(const GemmArgs p) {
    const int n_tiles = ((p.out + kTileRows - 1) / kTileRows) * ((p.m + kTileTok - 1) / kTileTok);
    gemm_body<DUAL, GROUPS>(p, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), n_tiles, static_cast<int>(blockIdx.y));
}

// Several matrices that multiply the same activation rows (q / k / v, gate / up) in one launch, a CTA per tile and K split.  Every
// matrix brings its own rotated activations (its own seeds), scratch and status word.  Matrices of one K split: gridDim.x is cut into one
// range of row tiles per matrix, gridDim.y are the token tiles, gridDim.z the splits.  Otherwise (`flat`) the CTAs of a matrix, split by split,
// follow one another in gridDim.x, the matrices with the longest ones first, so that short ones fill what is left of the last wave.  (With
// the largest split as gridDim.z the CTAs beyond a matrix's own left at once, but each took its place on an SM first: 3584 -> 3584 +
// 512 + 512 at 64 rows 20.1 -> 19.6 us, at 2048 96.5 -> 91.3, 5120 -> 5120 + 1024 + 1024 at 32 25.2 -> 22.7.  Matrices of one split in that order, and with
// its division: 3 x 4096 -> 4096 at 16 rows 27.3 -> 27.8.)
constexpr int kMaxGemmGroup = 4;
struct GemmGroupArgs {
    GemmArgs m[kMaxGemmGroup];
    int start[kMaxGemmGroup + 1];   // row tiles, or CTAs, start[i] .. start[i + 1] - 1 belong to matrix i
    int n_tiles[kMaxGemmGroup];     // (flat)
    int n, flat;
};
// CTAs of one group of producers (group_call_groups) go two to an SM, the second half beside the first instead of behind it
// (80 registers: a third one would find no tensor memory).  Two or three groups, one CTA to an SM -> one group: 3584 -> 3584 + 512 + 512 at 16 rows 15.1 -> 9.4 us,
// at 64 17.6 -> 13.4, 5120 -> 5120 + 1024 + 1024 at 32 21.6 -> 19.3, 4096 -> 2 x 11008 at 16 39.1 -> 33.0.  Fewer CTAs than SMs, two groups: 2048 -> 2 x 1024 at 32 rows
// 7.1 -> 6.7, 768 -> 2 x 768 at 100 8.1 -> 6.7 (three 9.6).
// (The bound of two groups is that of three: 64 registers a thread, so that CTAs of the rotation and of the sums fit beside them.)
template <bool DUAL, int GROUPS>
__global__ void __launch_bounds__(GROUPS == 1 ? 384 : gemm_threads(kGroupsMax), GROUPS == 1 ? 2 : 1) tq8_gemm_group_kernel(const __grid_constant__ GemmGroupArgs grp) {
    const int b = static_cast<int>(blockIdx.x);
    int i = 0;
    while (i + 1 < grp.n && b >= grp.start[i + 1]) ++i;
    int t = (b - grp.start[i]) * static_cast<int>(gridDim.y) + static_cast<int>(blockIdx.y), bz = static_cast<int>(blockIdx.z);
    if (grp.flat) {
        bz = t / grp.n_tiles[i];
        t -= bz * grp.n_tiles[i];
    }
    gemm_body<DUAL, GROUPS>(grp.m[i], t, 1, t + 1, bz);
}

// y = fp16(norm * inv_scale * sum over K splits, in split order) - fixed order, run-to-run identical - for the matrices of a call
// that were split (a group's by blockIdx.z).  Latency counts, it follows every split product of a decode batch: a thread takes V weight
// rows, requests their norms before the kernel in front has ended, and then BATCH splits' sums at once.  Behind products that leave room (early) its
// CTAs are there before these end, and let those of the next call's rotation come in turn.  64 registers: eight CTAs to an SM, one or two beside a
// product's.  With 126 (all sums of twelve splits at once) 8192 x 1024 in 16 splits took 11.2 us at 32 rows instead of 8.6, 2048 x 2048 at 512 rows 19.2 instead of 16.2;
// as few CTAs as SMs, with several rows each, crowd on a few of them (3584 x 3584 at 64 rows 12.2 -> 15.0).  Behind a product that fills the SMs four CTAs to an SM
// spread better (18944 x 3584 at 64 rows 25.1 us, 25.6 with eight).
struct FinishOne {
    const float* partial;
    const float* norms;
    __half* y;
    long y_stride;
    int out, k_splits, vec;   // vec: rows of four outputs, aligned
    float inv_scale;
};
struct FinishArgs { FinishOne m[kMaxGemmGroup]; };
constexpr int kFinishThreads = 128;
// V sums side by side in one access.
template <int V>
struct Sums {
    float v[V];
    __device__ __forceinline__ void load(const float* p) {
        if constexpr (V == 4) {
            const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            const float2 t = __ldcg(reinterpret_cast<const float2*>(p));
            v[0] = t.x; v[1] = t.y;
        }
    }
    // `step` apart, those below n.
    __device__ __forceinline__ void load_some(const float* p, int n, int step) {
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = k * step < n ? __ldcg(p + k * step) : 0.f;
    }
};
// V = 4, or 2 where more than eight splits are to be asked for at once.
template <int kBatch, int V>
__device__ __forceinline__ void gemm_finish_body(const FinishOne& f, int m, bool early) {
    const int out = f.out, k_splits = f.k_splits;
    // a thread's V rows: side by side in whole pieces, otherwise a CTA's width apart, so that a warp's accesses are contiguous all the same
    // (side by side in both cases: 3328 x 497 at 160 rows 13.0 us in a CUDA graph, so 11.4; 2816 x 1297 at 56 rows 9.2, so 8.3)
    const int step = f.vec ? 1 : kFinishThreads;
    const int c = f.vec ? V * static_cast<int>(blockIdx.x * kFinishThreads + threadIdx.x) : static_cast<int>(V * blockIdx.x * kFinishThreads + threadIdx.x);
    if (c >= out) return;
    float norm[V];   // (used behind the wait only: a product with it in front of the wait would wait for it there)
#pragma unroll
    for (int k = 0; k < V; ++k) norm[k] = c + k * step < out ? __ldg(f.norms + c + k * step) : 0.f;
    if (early) asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!early) asm volatile("griddepcontrol.launch_dependents;");
    const float* partial = f.partial;
    behind_wait(partial);
    const size_t split = static_cast<size_t>(m) * out;
    for (int row = blockIdx.y; row < m; row += gridDim.y) {
        const float* const src = partial + static_cast<size_t>(row) * out + c;
        __half* const y = f.y + row * f.y_stride + c;
        float acc[V];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] = 0.f;
        for (int z0 = 0; z0 < k_splits; z0 += kBatch) {
            Sums<V> v[kBatch];
            if (f.vec) {
#pragma unroll
                for (int z = 0; z < kBatch; ++z)
                    if (z0 + z < k_splits) v[z].load(src + (z0 + z) * split);
            } else {
#pragma unroll
                for (int z = 0; z < kBatch; ++z)
                    if (z0 + z < k_splits) v[z].load_some(src + (z0 + z) * split, out - c, kFinishThreads);
            }
#pragma unroll
            for (int z = 0; z < kBatch; ++z)
                if (z0 + z < k_splits) {
#pragma unroll
                    for (int k = 0; k < V; ++k) acc[k] += v[z].v[k];
                }
        }
        if (f.vec) {
            uint32_t h[V / 2];
#pragma unroll
            for (int k = 0; k < V; k += 2) {
                const __half2 h2 = __floats2half2_rn(acc[k] * (norm[k] * f.inv_scale), acc[k + 1] * (norm[k + 1] * f.inv_scale));
                h[k / 2] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            if constexpr (V == 4) *reinterpret_cast<uint2*>(y) = make_uint2(h[0], h[1]);
            else *reinterpret_cast<uint32_t*>(y) = h[0];
        } else {
#pragma unroll
            for (int k = 0; k < V; ++k)
                if (c + k * kFinishThreads < out) y[k * kFinishThreads] = __float2half_rn(acc[k] * (norm[k] * f.inv_scale));
        }
    }
}
// (A single matrix as a group of one, its parameters found by an index: 0.2 us more a call.)
template <int BATCH, int V>
__global__ void __launch_bounds__(kFinishThreads, BATCH * V == 32 ? 8 : 0) gemm_finish_kernel(const __grid_constant__ FinishOne f, int m, bool early) { gemm_finish_body<BATCH, V>(f, m, early); }
template <int BATCH, int V>
__global__ void __launch_bounds__(kFinishThreads, BATCH * V == 32 ? 8 : 0) gemm_finish_group_kernel(const __grid_constant__ FinishArgs f, int m, bool early) { gemm_finish_body<BATCH, V>(f.m[blockIdx.z], m, early); }
constexpr size_t kFourCtas = 48 * 1024;   // shared memory that is asked for and not used: so many CTAs to an SM
void finish_add(FinishArgs& f, int& n, const GemmArgs& a) {
    if (a.k_splits <= 1) return;
    f.m[n] = FinishOne{a.partial, a.norms, a.y, a.y_stride, a.out, a.k_splits,
                       a.out % 4 == 0 && a.y_stride % 4 == 0 && reinterpret_cast<uintptr_t>(a.y) % 8 == 0 ? 1 : 0, a.inv_scale};
    ++n;
}
void launch_finish(const FinishArgs& f, int n, int m, int groups, int sm_count, cudaStream_t stream) {
    if (n == 0) return;
    int widest = 0, most = 0;
    for (int i = 0; i < n; ++i) {
        widest = std::max(widest, f.m[i].out);
        most = std::max(most, f.m[i].k_splits);
    }
    const bool few = groups < kGroupsMax;
    const int v = few && most > 8 ? 2 : 4, carveout = gemm_carveout(m, groups);
    const int gx = (widest + v * kFinishThreads - 1) / (v * kFinishThreads);
    const int gy = std::max(1, std::min(m, 16 * sm_count / (gx * n)));   // up to sixteen CTAs per SM
    const dim3 grid(static_cast<unsigned int>(gx), static_cast<unsigned int>(gy), static_cast<unsigned int>(n));
    if (n == 1) launch_pdl_carved(!few ? gemm_finish_kernel<12, 4> : v == 4 ? gemm_finish_kernel<8, 4> : gemm_finish_kernel<16, 2>, grid, dim3(kFinishThreads), few ? 0 : kFourCtas, carveout, stream, f.m[0], m, few);
    else launch_pdl_carved(v == 4 ? gemm_finish_group_kernel<8, 4> : gemm_finish_group_kernel<16, 2>, grid, dim3(kFinishThreads), 0, carveout, stream, f, m, few);
}

// Groups of 8 rows that a CTA of the rotation takes one after the other: as many as leave eight CTAs per SM.
int rotate_row_steps(long groups, int sm_count) { return static_cast<int>(std::max<long>(1, std::min<long>(8, groups / (8L * sm_count)))); }

// The activation rows rotated for n matrices (their own seeds and destinations): one launch, except for an activation that is
// not aligned.  Both kernels add in the order of warp_fwht, in fp32: the operand does not depend on the alignment.  (With four of the
// butterflies as products with +-1 on the tensor cores a 7B layer's projections of 2048 rows took 1100 us instead of 1120, of 64 rows
// 119 instead of 121; but the sums were rounded elsewhere, and the results of the two kernels differed.)
void launch_rotate_rows(const __half* x, const RotateGroupArgs& rot, int n, int in, long m, int n_planes, uint32_t block, int groups_of_product, int carveout, int sm_count, cudaStream_t stream) {
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(block));
    const int bs = static_cast<int>(block);
    if (reinterpret_cast<uintptr_t>(x) % 16 == 0) {
        const int cols = std::max(256, bs);
        const long groups = static_cast<long>(n_planes) * ((in + cols - 1) / cols);
        const int row_steps = rotate_row_steps(n * groups * ((m + 7) / 8), sm_count);
        const long ctas = groups * ((m + 8L * row_steps - 1) / (8L * row_steps));
        if (ctas < (1L << 31)) {
            const dim3 grid(static_cast<unsigned int>(ctas), static_cast<unsigned int>(n));
            const bool few = row_steps == 1 && groups_of_product < kGroupsMax;
#define TQ_ROTATE_WIDE(CHUNKS)                                                                                                                         \
    if (n == 1) launch_pdl_carved(few ? rotate_rows_f16_wide_kernel<CHUNKS, true> : rotate_rows_f16_wide_kernel<CHUNKS, false>, grid, dim3(256), 0, carveout, stream, x, rot.xrot[0], in, m, bs, rot.seed_p[0], rot.seed_r[0], inv_sqrt, row_steps); \
    else launch_pdl_carved(few ? rotate_rows_f16_wide_group_kernel<CHUNKS, true> : rotate_rows_f16_wide_group_kernel<CHUNKS, false>, grid, dim3(256), 0, carveout, stream, x, rot, in, m, bs, inv_sqrt, row_steps);
            switch (cols) {
                case 256: TQ_ROTATE_WIDE(1) break;
                case 512: TQ_ROTATE_WIDE(2) break;
                default: TQ_ROTATE_WIDE(4) break;
            }
#undef TQ_ROTATE_WIDE
            return;
        }
    }
    const long n_warps = static_cast<long>(n_planes) * m * (in / bs);   // a warp per plane, row and block
    const unsigned int grid = static_cast<unsigned int>((n_warps + 3) / 4);
    for (int i = 0; i < n; ++i) {
#define TQ_ROT16_CASE(EV)                                                                                                               \
    case 32 * EV:                                                                                                                       \
        launch_pdl(rotate_rows_f16_kernel<EV>, dim3(grid), dim3(128), 0, stream, x, rot.xrot[i], in, m, n_planes, rot.seed_p[i], rot.seed_r[i], \
                   inv_sqrt);                                                                                                           \
        break;
        switch (block) {
            TQ_ROT16_CASE(1) TQ_ROT16_CASE(2) TQ_ROT16_CASE(4) TQ_ROT16_CASE(8) TQ_ROT16_CASE(16) TQ_ROT16_CASE(32)
            default: throw Error("unsupported WHT block size");
        }
#undef TQ_ROT16_CASE
    }
}

size_t xrot_bytes(int in, long m, int n_planes) {
    const size_t padded = (static_cast<size_t>(m) + kTileTok - 1) / kTileTok * kTileTok;  // whole operand tiles
    return (static_cast<size_t>(n_planes) * padded * static_cast<size_t>(in) * sizeof(__half) + 255) & ~static_cast<size_t>(255);
}

auto gemm_kernel_of(int n_planes, int groups) {
    if (n_planes == 2) return groups == 2 ? tq8_gemm_kernel<true, 2> : tq8_gemm_kernel<true, 3>;
    return groups == 2 ? tq8_gemm_kernel<false, 2> : tq8_gemm_kernel<false, 3>;
}
auto gemm_group_kernel_of(int n_planes, int groups) {
    if (n_planes == 2) return groups == 1 ? tq8_gemm_group_kernel<true, 1> : groups == 2 ? tq8_gemm_group_kernel<true, 2> : tq8_gemm_group_kernel<true, 3>;
    return groups == 1 ? tq8_gemm_group_kernel<false, 1> : groups == 2 ? tq8_gemm_group_kernel<false, 2> : tq8_gemm_group_kernel<false, 3>;
}

}  // namespace

// When the output has too few tiles to occupy the SMs (few activation rows on a matrix with few
// rows and many columns), K is split over several CTAs per tile; every split keeps at least 8 K blocks.  (Splits of four, up to eight of them, are up to
// 12 % faster for a matrix of up to 2048 columns alone, 1024 x 1024 at 32 rows 8.7 -> 7.9 us.  But a matrix has the same splits in a group, for the same bits,
// and the CTAs of a group then outnumber the SMs: 2048 -> 2048 + 256 + 256 at 32 rows 9.2 -> 13.6, 2560 -> 2560 + 512 + 512 9.8 -> 15.1.  And of 512 or 768 columns
// the sums outweigh what the CTAs gain: 512 x 8192 at 128 rows 9.0 -> 14.1.)
int gemm_k_splits(int out, int in, long m, int n_planes, int sm_count) {
    const long tiles = static_cast<long>((out + kTileRows - 1) / kTileRows) * ((m + kTileTok - 1) / kTileTok);
    const int n_kb = in / kBlockK * n_planes;
    long s = sm_count / (tiles > 0 ? tiles : 1);
    if (s > n_kb / 8) s = n_kb / 8;
    return s < 1 ? 1 : static_cast<int>(s);
}

size_t gemm_scratch_bytes(int out, int in, long m, int n_planes, int sm_count) {
    const int splits = gemm_k_splits(out, in, m, n_planes, sm_count);
    size_t bytes = xrot_bytes(in, m, n_planes);
    if (splits > 1) bytes += static_cast<size_t>(splits) * static_cast<size_t>(m) * out * sizeof(float);
    return bytes;
}

bool gemm_supported(int in) { return in % kBlockK == 0; }

void launch_tq8_gemm(const uint8_t* codes, const float* norms, const float* table, const __half* x, __half* y, int out,
                     int in, long m, uint32_t block, int n_planes, float pair_unit, uint32_t seed_p, uint32_t seed_r, void* scratch,
                     unsigned int* status, int sm_count, cudaStream_t stream, long y_stride) {
    if (y_stride <= 0) y_stride = out;
    TQ_REQUIRE(y_stride >= out, "tq8_gemm: output row stride smaller than the layer's rows");
    TQ_REQUIRE(n_planes == 1 || n_planes == 2, "tq8_gemm: one or two rotation planes");
    TQ_REQUIRE(gemm_supported(in), "tq8_gemm: in_features must be a multiple of 64");
    TQ_REQUIRE(is_pow2(block) && block >= 32 && block <= 1024, "WHT block size must be a power of two in [32, 1024]");
    TQ_REQUIRE(in % static_cast<int>(block) == 0, "in_features must be divisible by block_size");
    TQ_REQUIRE(m >= 1 && m < (1L << 30), "tq8_gemm: bad number of activation rows");
    TQ_REQUIRE(scratch != nullptr, "tq8_gemm needs its scratch buffer");
    if (out == 0) return;
    __half* xrot = static_cast<__half*>(scratch);
    const long n_tiles = static_cast<long>((out + kTileRows - 1) / kTileRows) * ((m + kTileTok - 1) / kTileTok);
    TQ_REQUIRE(n_tiles < (1L << 31), "tq8_gemm: too many output tiles");
    const int k_splits = gemm_k_splits(out, in, m, n_planes, sm_count);
    const int groups = gemm_groups(n_tiles, in / kBlockK * n_planes / k_splits, m, sm_count);

    // 1. rotate every activation row
    {
        RotateGroupArgs rot{};
        rot.xrot[0] = xrot; rot.seed_p[0] = seed_p; rot.seed_r[0] = seed_r;
        launch_rotate_rows(x, rot, 1, in, m, n_planes, block, groups, gemm_carveout(m, groups), sm_count, stream);
    }
    // 2. the GEMM
    GemmArgs a{};
    a.codes = codes; a.norms = norms; a.table = table; a.xrot = xrot; a.y = y; a.y_stride = y_stride; a.status = status;
    a.out = out; a.in = in; a.m = static_cast<int>(m);
    a.inv_scale = 1.0f / std::sqrt(static_cast<float>(in));
    if (n_planes == 2) {
        a.table += 512;   // (the pairs, behind the two tables)
        a.inv_scale *= pair_unit;
    }
    a.k_splits = k_splits;
    a.partial = a.k_splits > 1 ? reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + xrot_bytes(in, m, n_planes)) : nullptr;
    static bool configured[64] = {false};
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !configured[dev]) {
        for (auto* const k : {tq8_gemm_kernel<false, 2>, tq8_gemm_kernel<true, 2>, tq8_gemm_kernel<false, 3>, tq8_gemm_kernel<true, 3>})
            TQ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemmSmemBytes)));
        if (dev < 64) configured[dev] = true;
    }
    // a CTA per SM walks the tiles (with a K split there are fewer tiles x splits than SMs)
    const dim3 grid(static_cast<unsigned int>(std::min<long>(n_tiles, sm_count)), static_cast<unsigned int>(a.k_splits));
    launch_pdl_carved(gemm_kernel_of(n_planes, groups), grid, dim3(gemm_threads(groups)), gemm_smem_bytes(m, groups), gemm_carveout(m, groups), stream, a);
    TQ_CUDA(cudaGetLastError());
    FinishArgs fin{};
    int n_fin = 0;
    finish_add(fin, n_fin, a);
    launch_finish(fin, n_fin, static_cast<int>(m), groups, sm_count, stream);
}

void launch_tq8_gemm_group(const GemmGroupItem* items, int n, const __half* x, long m, int sm_count, cudaStream_t stream) {
    TQ_REQUIRE(items != nullptr && n >= 1 && n <= kMaxGemmGroup, "tq8_gemm group: 1..4 matrices");
    TQ_REQUIRE(x != nullptr && m >= 1 && m < (1L << 30), "tq8_gemm group: bad number of activation rows");
    const int in = items[0].in, n_planes = items[0].n_planes;
    const uint32_t block = items[0].block;
    TQ_REQUIRE(n_planes == 1 || n_planes == 2, "tq8_gemm: one or two rotation planes");
    TQ_REQUIRE(gemm_supported(in), "tq8_gemm: in_features must be a multiple of 64");
    TQ_REQUIRE(is_pow2(block) && block >= 32 && block <= 1024, "WHT block size must be a power of two in [32, 1024]");
    TQ_REQUIRE(in % static_cast<int>(block) == 0, "in_features must be divisible by block_size");
    GemmGroupArgs grp{};
    RotateGroupArgs rot{};
    FinishArgs fin{};
    int n_fin = 0;
    grp.n = n;
    long n_ctas = 0;
    GroupCallCtas shape{};
    int order[kMaxGemmGroup], splits[kMaxGemmGroup];
    const long tok_tiles = (m + kTileTok - 1) / kTileTok;
    for (int i = 0; i < n; ++i) {
        // the split a matrix would get alone, not one for the group as a whole: with fewer splits the group ran 7-9 %
        // faster (16 / 64 rows) but the fp32 sums changed their order, and results would no longer be bit-equal to
        // separate calls
        splits[i] = gemm_k_splits(items[i].out, in, m, n_planes, sm_count);
        order[i] = i;
        grp.flat |= splits[i] != splits[0] ? 1 : 0;
    }
    std::stable_sort(order, order + n, [&](int a, int b) { return splits[a] < splits[b]; });
    for (int i = 0; i < n; ++i) {
        const GemmGroupItem& it = items[order[i]];
        TQ_REQUIRE(it.codes && it.norms && it.table && it.y && it.scratch && it.out >= 1, "tq8_gemm group: NULL argument");
        TQ_REQUIRE(it.in == in && it.n_planes == n_planes && it.block == block,
                   "tq8_gemm group: the matrices must share in_features, the WHT block and the rotation mode");
        GemmArgs& a = grp.m[i];
        a.codes = it.codes; a.norms = it.norms; a.table = it.table; a.y = it.y; a.y_stride = it.out; a.status = it.status;
        a.xrot = static_cast<__half*>(it.scratch);
        a.out = it.out; a.in = in; a.m = static_cast<int>(m);
        a.inv_scale = 1.0f / std::sqrt(static_cast<float>(in));
        if (n_planes == 2) {
            a.table += 512;
            a.inv_scale *= it.pair_unit;
        }
        a.k_splits = splits[order[i]];
        a.partial = a.k_splits > 1 ? reinterpret_cast<float*>(static_cast<uint8_t*>(it.scratch) + xrot_bytes(in, m, n_planes)) : nullptr;
        const long row_tiles = (it.out + kTileRows - 1) / kTileRows, n_tiles = row_tiles * tok_tiles;
        grp.n_tiles[i] = static_cast<int>(n_tiles);
        grp.start[i] = static_cast<int>(n_ctas);
        n_ctas += grp.flat ? n_tiles * a.k_splits : row_tiles;
        shape.ctas[i] = n_tiles * a.k_splits;
        shape.stages[i] = (in / kBlockK * n_planes / a.k_splits + kSubPerStage - 1) / kSubPerStage;
        TQ_REQUIRE(n_tiles < (1L << 31) && n_ctas < (1L << 31), "tq8_gemm group: too many output tiles");
        rot.xrot[i] = static_cast<__half*>(it.scratch);
        rot.seed_p[i] = it.seed_p; rot.seed_r[i] = it.seed_r;
        finish_add(fin, n_fin, a);
    }
    for (int i = n; i <= kMaxGemmGroup; ++i) grp.start[i] = static_cast<int>(n_ctas);
    shape.n = n;
    shape.least = splits[order[0]];
    shape.unequal = grp.flat != 0;
    const int groups = group_call_groups(shape, m, n_planes, sm_count);
    // 1. the rotations
    launch_rotate_rows(x, rot, n, in, m, n_planes, block, groups, gemm_carveout(m, groups), sm_count, stream);
    // 2. the GEMMs
    static bool configured[64] = {false};
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !configured[dev]) {
        for (auto* const k : {tq8_gemm_group_kernel<false, 1>, tq8_gemm_group_kernel<true, 1>, tq8_gemm_group_kernel<false, 2>, tq8_gemm_group_kernel<true, 2>, tq8_gemm_group_kernel<false, 3>, tq8_gemm_group_kernel<true, 3>})
            TQ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemmSmemBytes)));
        if (dev < 64) configured[dev] = true;
    }
    const dim3 grid(static_cast<unsigned int>(n_ctas), grp.flat ? 1u : static_cast<unsigned int>(tok_tiles), grp.flat ? 1u : static_cast<unsigned int>(splits[0]));
    launch_pdl_carved(gemm_group_kernel_of(n_planes, groups), grid, dim3(gemm_threads(groups)), gemm_smem_bytes(m, groups), gemm_carveout(m, groups), stream, grp);
    // 3. the split-K sums
    launch_finish(fin, n_fin, static_cast<int>(m), groups, sm_count, stream);
}

}  // namespace tq
