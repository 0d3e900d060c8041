// Fused quantize kernel on the 5th-generation tensor cores (tcgen05 + TMEM) for fp16 / bf16 rows with d in {64, 96, 128, 256}:
//   norm -> rotation (128 rows x d x d contraction per tile) -> Lloyd-Max boundary search -> bit-pack (+ QJL sketch).
//
// The rotation has to be float32-accurate (a code flips whenever a rotated value crosses a boundary), so the rows are
// used UN-normalised as exact MMA operands and R is split into terms that are exact operands too:
//   fp16 rows: R = R_hi + 2^-11 R_lo (fp16 each): one MMA of N = 2 d per k-step against [R_hi ; 2^11 R_lo] fills a
//              high and a low accumulator (two chains of d / 16 dependent MMAs would take as long as one: a dependent
//              step costs about 70 ns whatever its width); the epilogue adds them.  With the sketch on there is room
//              for one accumulator per tile only: the low products are accumulated first and the first high MMA takes
//              the accumulator scaled by 2^-11 (the instruction's scale-input-d).
//   bf16 rows: R = R_1 + R_2 + R_3 (bf16 each, 24 bits together; bf16 has float32's exponent range, so no scaling) into
//              one accumulator.
// Every product is exact in the fp32 accumulator; the normalisation by the row norm is applied afterwards.
//
// Warp roles in a persistent CTA (one per SM; 640 threads for fp16 rows, 704 for bf16 rows and sketches).  Sixteen epilogue warps come first (E of them),
// then one MMA warp, two or four norm warps, one TMA warp:
//   warps 0..E-1 epilogue; thread <-> one row (TMEM lane) and a share of its sixteen-coordinate chunks (tcgen05.ld).
//                fp16 rows: all sixteen warps work on the same tile in step, a quarter of the row each, reading the
//                high and the low accumulator and combining them; two accumulator stages, so the MMAs of the next tile
//                run meanwhile.  bf16 rows: two groups of eight warps take alternate tiles (two stages each), half a row
//                per thread.  With the QJL sketch on, two groups as well and three stages: the quantization residual of
//                every coordinate replaces it in tensor memory, and the MMA warp multiplies the tile by the projections.
//                Up to 3 bits a binary search over boundaries (times the row's norm) held in registers adds its
//                outcome bits straight into the packed word; at 4 bits one lookup in a 513-bin table (bin -> nearest
//                boundary + count below; see build_bins).  Fractional widths: the threads of a row take chunks of
//                either width, so they finish together.
//   warp  E      allocates TMEM, issues the MMAs (in uniform control flow, one elected lane) and commits them to mbarriers
//   next         norms: read each tile back from shared memory for the rows' sums of squares
//   last warp    one thread keeps the operand stages full with tiled TMA copies (cp.async.bulk.tensor, 3-D tensor map
//                (column, row, lane), 128-byte swizzle as the MMA descriptors expect; rows past a lane's end and
//                columns past d read as zeros)
// head_dim 256 (DC = 256, no sketch): R does not fit beside the rows, so four CTAs share a 128-row tile, 64 output columns
// each (a fractional width's halves are two such slices, so every slice has one width).  The contraction runs over 256
// columns in two halves of one operand stage each; all terms of R sit side by side in ONE operand (fp16: [R_hi | R_lo],
// bf16: [R_1 | R_2 | R_3], N = 128 / 192), because sixteen dependent MMAs take the same time at any width, and the epilogue
// adds the accumulators.  The rows' norms have slots of their own, so that stages are free as soon as the MMAs have read
// them.  A tile is fetched from memory once and three times from L2.  (524,288 rows at 4 bits: 4602 us in the CUDA-core row kernel before, 244 here; 3.5 bits 4576 / 254, bf16 4595 / 252.)
// Every mbarrier wait is bounded: on a timeout the kernel raises a status word, drains and frees its TMEM.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace tq {

namespace tc {

constexpr int DMAX = 128, TM = 128;              // largest head_dim, rows per tile
constexpr int A_STAGES_MAX = 3, ACC_STAGES = 4;
constexpr int EPI_WARPS = 16, N_EPI = EPI_WARPS * 32;            // epilogue warps; then the MMA warp, the norm warps, the TMA warp
// Threads that read the rows back for the norms.  fp16 rows without the sketch: two rows each, as with 20 warps in all a thread may have 96
// registers, with 22 only 80, and the epilogue spilled (8 x 65,536 rows: d = 128 at 3 and 2 bits 97.0 / 94.5 us, d = 64 at 4 and 4 bits 88.0 /
// 82.0, 2 x 65,536 of 256 100.8 / 97.0).  The others have fewer operand stages or longer chains of products and want theirs back soon: a row
// each (bf16, d = 64 at 3 bits, 8 x 32,768 rows 39.0 us, with two rows a thread 40.9).
__host__ __device__ constexpr int n_norm(bool splitacc) { return splitacc ? 64 : 128; }
__host__ __device__ constexpr int n_threads(bool splitacc) { return N_EPI + 32 + n_norm(splitacc) + 32; }     // 640 / 704
constexpr int BIN_REP = 16;                      // copies of every lookup-table entry (lane & 15 picks one): the lanes of a half-warp read banks of their own
constexpr int KBLK_BYTES = TM * 128;             // one 64-column K-block of a 128-row operand: 16 KB
constexpr int OPER_BYTES = 2 * KBLK_BYTES;       // 32 KB per operand tile
constexpr int NBINS = 257, BIN0 = 128;           // the table's bins: 1/256 wide around (k - BIN0) / 256
constexpr int QM = 32;                           // projections of the QJL sketch
constexpr uint32_t WAIT_LIMIT = 4u << 20;        // bounded spin: a few hundred milliseconds at most

// shared memory map (bytes).  fp16 rows: three row stages and two terms of R; bf16 rows: two row stages and three terms.
constexpr int OFF_A = 0;                                   // stage s at s * 32 KB, 1024-byte aligned
constexpr int OFF_R3 = OFF_A + 2 * OPER_BYTES;             // bf16: third term of R (fp16: the third row stage)
constexpr int OFF_R1 = OFF_A + 3 * OPER_BYTES;             // R_hi / R_1
constexpr int OFF_R2 = OFF_R1 + OPER_BYTES;                // R_lo / R_2
constexpr int OFF_BINS = OFF_R2 + OPER_BYTES;              // NBINS x BIN_REP x 8 B: the table of the 4-bit codebook (only bits_hi can be 4)
constexpr int OFF_PT = (OFF_BINS + NBINS * BIN_REP * 8 + 1023) / 1024 * 1024;     // QJL: (S R^T) as fp16 high and low parts, operand tiles of 32 rows x 64 columns (PT_KBLK bytes): hi 0, hi 1, lo 0, lo 1
constexpr int PT_KBLK = QM * 128;
constexpr int OFF_BND = OFF_PT + DMAX * QM * 4;            // 2 x 16 floats raw boundaries, 2 x 16 floats centroids
constexpr int OFF_NSQ = OFF_BND + 256;                     // A_STAGES_MAX x 2 x 128 floats: partial sums of squares
constexpr int OFF_BAR = OFF_NSQ + A_STAGES_MAX * 2 * TM * 4;   // mbarriers: 3 full, 3 a_free, 3 norm-ready, 4 acc_full, 4 acc_free
constexpr int OFF_MISC = OFF_BAR + 24 * 8;                 // tmem base, abort flag
constexpr int OFF_EE = (OFF_MISC + 64 + 127) / 128 * 128;   // QJL: squares of the residual, the second half of a row's: SK_STAGES x 128 floats
constexpr int SK_STAGES = 3, SK_COL0 = SK_STAGES * DMAX;    // QJL: accumulator stages; the sketches' 32 TMEM columns a stage lie behind them
constexpr int SMEM_BYTES = OFF_EE + SK_STAGES * TM * 4;
static_assert(SMEM_BYTES <= 227 * 1024, "shared-memory plan");

constexpr int SLICE = 64, NSQ_SLOTS = 8;                   // head_dim 256: output columns of a CTA, norm slots
constexpr int OFF_NSQ256 = OFF_PT, OFF_NRMBAR256 = OFF_NSQ256 + NSQ_SLOTS * TM * 4;     // (there is no sketch)
static_assert(NSQ_SLOTS * TM * 4 + NSQ_SLOTS * 8 <= DMAX * QM * 4, "head_dim 256: norm slots");

struct Params {
    int d, bf16, a_stages;
    int follows;                                 // runs beside the launch before it and ends after it
    int64_t n_rows, n_tiles, tiles_per_lane;     // tiles never cross cache lanes; tile = lane * tiles_per_lane + tile in lane
    const float* rot;
    const float* bnd_hi; const float* bnd_lo; int bits_hi, bits_lo;
    uint8_t* p_hi; uint8_t* p_lo; float* norms; int64_t out_lane_stride;
    const float* qjl_proj_rot; const float* cent_hi; const float* cent_lo; uint32_t* qjl_bits; float* qjl_gamma;
};

__device__ int g_status = 0;   // 0 ok, otherwise the code of the first wait that timed out

// ---- PTX wrappers ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false after WAIT_LIMIT polls (or when another role already gave up).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = code;
    atomicCAS(&g_status, 0, code);
    return false;
}
// What this thread's last copies or products were to complete, also after a wait that ran out (bounded, whatever the flag says):
// nothing may land in shared or tensor memory that the CTA has given up.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try(bar, parity); ++i) {}
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
// Tiled TMA load of a (64 columns x 128 rows x 1 lane) box; the innermost coordinate is 0 or 64 elements (0 or 128 bytes).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D = A.B (+ D when accumulate != 0)
// (issued by one elected lane of a warp in uniform control flow: the operands then come straight from uniform registers, where a
// single thread in a divergent branch moves each of them over one by one)
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// D = A.B (+ D when accumulate != 0), A in tensor memory: row = lane, two fp16 columns a word
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// D = A.B + 2^-11 D
__device__ __forceinline__ void umma_f16_scaled11(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc) {
    const uint32_t one = 1;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(one) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two float32 operations an instruction, and sums of squares that take 16-bit factors as they are: the launch is bound by the instructions
// its warps issue (18.8 a coordinate at 3 bits of fp16 rows, 2 of them the norms').  Keys at 4 bits and values at 2, 8 x 65,536 rows, one
// operation an instruction / now: d = 128 fp16 104.7 / 102.1 us, bf16 114.4 / 111.5, d = 64 at 4 and 4 bits 92.3 / 86.0, d = 96 with
// sketches 134.3 / 127.8, d = 256 (131,072 rows) 106.7 / 101.0.
using u64 = unsigned long long;
__device__ __forceinline__ u64 pk(float a, float b) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void upk(u64 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x)); }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) { u64 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ u64 add2(u64 a, u64 b) { u64 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
// a += the squares of a word's two halves (exact products, one rounding each), low half first
template <bool BF16>
__device__ __forceinline__ void add_squares(float& a, uint32_t x) {
    if (BF16) asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tfma.rn.f32.bf16 %0, l, l, %0;\n\tfma.rn.f32.bf16 %0, h, h, %0;\n\t}" : "+f"(a) : "r"(x));
    else asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tfma.rn.f32.f16 %0, l, l, %0;\n\tfma.rn.f32.f16 %0, h, h, %0;\n\t}" : "+f"(a) : "r"(x));
}

// K-major operand tile in shared memory, 128-byte swizzle: row r of K-block b at  b*16 KB + r*128 B, its 16-byte
// chunk c stored at chunk position c ^ (r & 7).  Descriptor for the 16-column slab `ks` (0..3) of K-block b.
__device__ __forceinline__ uint64_t smem_desc(uint32_t tile_addr, int kblk, int ks) {
    const uint32_t addr = tile_addr + kblk * KBLK_BYTES + ks * 32;
    uint64_t d = 0;
    d |= uint64_t((addr >> 4) & 0x3FFF);          // start address
    d |= uint64_t(1) << 16;                       // leading byte offset (ignored for swizzled K-major)
    d |= uint64_t(1024 >> 4) << 32;               // stride byte offset: 8 rows x 128 B
    d |= uint64_t(1) << 46;                       // descriptor version (Blackwell)
    d |= uint64_t(2) << 61;                       // SWIZZLE_128B
    return d;
}
// kind::f16 instruction descriptor: fp32 accumulate, A and B both fp16 or both bf16, both K-major, M = 128, N = d
__device__ __forceinline__ uint32_t make_idesc(int d, bool bf16) {
    return (1u << 4) | (bf16 ? ((1u << 7) | (1u << 10)) : 0u) | (uint32_t(d >> 3) << 17) | (uint32_t(TM >> 4) << 24);
}

// Lookup table for the boundary search.  Bin k covers normalised values around (k - BIN0) / 256 (width 1/256), the first and the last also
// everything beyond; entry = (boundary to test, number of boundaries below the bin's neighbourhood) where the neighbourhood is the
// bin widened by one bin on each side, so that a bin index that is off by one through rounding still gives the
// exact count.  A neighbourhood holding two boundaries is marked (a flag bit in the count) and handled by the plain
// counting loop.  (Half the bins that |y| <= 1 could use, for twice the copies: the outermost boundary of a 4-bit codebook lies at 0.3 for
// d = 64.  With eight copies of 513 a lookup took 6.6 shared-memory cycles a warp instead of two, and the whole launch 68 % of
// them.  Keys at 4 bits and values at 2, 8 x 65,536 rows of 128, before / now: bf16 122 / 114 us, fp16 108.8 / 104.7; 8 x 4096 rows, where
// the table's set-up counts, 20.1 / 16.5 and 16.5 / 15.7.)
constexpr int MARKED = 0x100;
__device__ void build_bins(float2* bins, const float* bnd, int n_bnd, int tid, int nthreads) {
    for (int k = tid; k < NBINS; k += nthreads) {
        const float lo = k > 0 ? (float(k - BIN0) - 1.5f) / 256.f : -INFINITY, hi = k < NBINS - 1 ? (float(k - BIN0) + 1.5f) / 256.f : INFINITY;
        int below = 0, inside = 0;
        float b_in = 2.0f;                    // no boundary near this bin: |y| <= 1 never exceeds the sentinel
        for (int i = 0; i < n_bnd; ++i) {
            const float b = bnd[i];
            if (b < lo) ++below;
            else if (b <= hi) { ++inside; b_in = b; }
        }
        const float e = __int_as_float(inside > 1 ? (below | MARKED) : below);
#pragma unroll
        for (int r = 0; r < BIN_REP / 2; ++r)                                        // (eight neighbours write eight different 16-byte columns)
            *reinterpret_cast<float4*>(bins + k * BIN_REP + 2 * ((r + tid) % (BIN_REP / 2))) = make_float4(b_in, e, b_in, e);
    }
}

// Up to three bits the code is never formed: the boundaries (times the row's norm) live in registers, a binary search
// (one compare per bit) decides how many of them the value exceeds - the number the counting loop gives for a
// non-decreasing boundary list, NaN included (0) - and each level's outcome adds its bit, already shifted into place,
// to the group word (eight codes per group, so a code never straddles two words while it is being built).
template <int BITS>
__device__ __forceinline__ void add_code(uint32_t& grp, float y, const float (&b)[7], int sh) {
    if (BITS == 1) {
        if (y > b[0]) grp += 1u << sh;
    } else if (BITS == 2) {
        const bool p1 = y > b[1];
        const bool p2 = y > (p1 ? b[2] : b[0]);
        if (p1) grp += 2u << sh;
        if (p2) grp += 1u << sh;
    } else {
        const bool p1 = y > b[3];
        const bool p2 = y > (p1 ? b[5] : b[1]);
        const float lo = p2 ? b[2] : b[0], hi = p2 ? b[6] : b[4];
        const bool p3 = y > (p1 ? hi : lo);
        if (p1) grp += 4u << sh;
        if (p2) grp += 2u << sh;
        if (p3) grp += 1u << sh;
    }
}
// The group word as a float (up to 24 bits: exact), for fp16 rows without the sketch: their launch keeps the pipe of compares and selects 68 %
// busy at 3 bits, and integer adds share it (8 x 65,536 rows of 128 at 3 and 2 bits 97.0 / 93.1 us, at 4 and 2 102.5 / 98.6; bf16 rows, which
// wait for their 24 dependent products, lose: d = 64 at 3 bits 67.8 / 69.4).
template <int BITS>
__device__ __forceinline__ void add_code(float& grp, float y, const float (&b)[7], int sh) {
    const float one = float(1u << sh);
    if (BITS == 1) {
        asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, %2;\n\t@p add.rn.f32 %0, %0, %3;\n\t}" : "+f"(grp) : "f"(y), "f"(b[0]), "f"(one));
    } else if (BITS == 2) {
        asm("{\n\t.reg .pred p, q;\n\t.reg .f32 t;\n\tsetp.gt.f32 p, %1, %3;\n\tselp.f32 t, %4, %2, p;\n\tsetp.gt.f32 q, %1, t;\n\t"
            "@p add.rn.f32 %0, %0, %6;\n\t@q add.rn.f32 %0, %0, %5;\n\t}" : "+f"(grp) : "f"(y), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(one), "f"(2.f * one));
    } else {
        asm("{\n\t.reg .pred p, q, r;\n\t.reg .f32 t, u, v;\n\tsetp.gt.f32 p, %1, %5;\n\tselp.f32 t, %7, %3, p;\n\tsetp.gt.f32 q, %1, t;\n\t"
            "selp.f32 u, %4, %2, q;\n\tselp.f32 v, %8, %6, q;\n\tselp.f32 t, v, u, p;\n\tsetp.gt.f32 r, %1, t;\n\t"
            "@p add.rn.f32 %0, %0, %11;\n\t@q add.rn.f32 %0, %0, %10;\n\t@r add.rn.f32 %0, %0, %9;\n\t}"
            : "+f"(grp) : "f"(y), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]), "f"(b[4]), "f"(b[5]), "f"(b[6]), "f"(one), "f"(2.f * one), "f"(4.f * one));
    }
}
// Plain counting loop, kept out of line: only reached when two boundaries share a bin neighbourhood.
__device__ __noinline__ uint32_t code_slow(float y, const float* raw_bnd, int n_bnd) {
    uint32_t c = 0;
    for (int i = 0; i < n_bnd; ++i) c += (y > raw_bnd[i]) ? 1u : 0u;
    return c;
}

// What a thread needs to know about its row while it walks the coordinates.
struct RowCtx {
    float rinv, rbin;              // 1 / max(|x|, 1e-10) and 256 times that
    const float2* bins;            // this lane's copy of the 4-bit table
};

// Sixteen coordinates (TMEM columns taddr .. + 15) at BITS bits: the codes go into g0 / g1 (eight codes each, BITS bits
// per code).  sb: boundaries times the row's norm (register search); raw: unscaled boundaries (table path's fallback).
// QJL: v[] leaves as 2^8 times the residuals (rbin and the centroids carry the factor); taddr: where v[] came from.
template <int BITS, bool QJL, bool FSUM>
__device__ __forceinline__ void quantize16(uint32_t* v, const RowCtx& rc, const float (&sb)[7], const float* raw, uint32_t& g0, uint32_t& g1, const float* cent, uint32_t taddr) {
    g0 = g1 = 0;
    const auto residual = [&](int i, uint32_t code) { v[i] = __float_as_uint(fmaf(__uint_as_float(v[i]), rc.rbin, -cent[code])); };
    if (BITS <= 3) {
        if constexpr (FSUM) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float grp = 0.f;
#pragma unroll
                for (int i = 8 * h; i < 8 * h + 8; ++i) add_code<BITS>(grp, __uint_as_float(v[i]), sb, BITS * (i & 7));
                (h ? g1 : g0) = __float2uint_rn(grp);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) add_code<BITS>(i < 8 ? g0 : g1, __uint_as_float(v[i]), sb, BITS * (i & 7));
        }
        if constexpr (QJL) {
#pragma unroll
            for (int i = 0; i < 16; ++i) residual(i, ((i < 8 ? g0 : g1) >> (BITS * (i & 7))) & ((1u << BITS) - 1u));
        }
    } else {
        // table path: count-below times 16^k goes in with one multiply-add, the compare adds its bit in place
        uint32_t seen = 0;
        const u64 rbin2 = pk(rc.rbin, rc.rbin), rinv2 = pk(rc.rinv, rc.rinv), bias2 = pk(8388608.f + BIN0, 8388608.f + BIN0);
        float t2[2], yn2[2];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            // bin index from the mantissa of (y * 256 + BIN0 + 2^23): exact rounding to nearest, no convert instruction; a NaN takes the last bin
            if (!(i & 1)) {
                const u64 y2 = pk(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                upk(fma2(y2, rbin2, bias2), t2[0], t2[1]);
                upk(mul2(y2, rinv2), yn2[0], yn2[1]);
            }
            const float yn = yn2[i & 1], tt = fmaxf(fminf(t2[i & 1], 8388608.f + (NBINS - 1)), 8388608.f);
            const float2 en = rc.bins[(__float_as_uint(tt) - 0x4B000000u) * BIN_REP];
            seen |= __float_as_uint(en.y);
            uint32_t& w = i < 8 ? g0 : g1;
            if constexpr (QJL) {
                const uint32_t code = __float_as_uint(en.y) + (yn > en.x ? 1u : 0u);
                w += code * (1u << (4 * (i & 7)));
                residual(i, code & 15u);                                           // (a marked bin's is formed again below)
            } else {
                w += __float_as_uint(en.y) * (1u << (4 * (i & 7)));
                if (yn > en.x) w += 1u << (4 * (i & 7));               // strict >, codebook.py:220-223
            }
        }
        if (__any_sync(0xffffffffu, (seen & MARKED) != 0)) {     // a marked bin was hit: redo the group with the counting loop
            g0 = g1 = 0;
            if constexpr (QJL) {
                tmem_ld16(taddr, *reinterpret_cast<uint32_t (*)[16]>(v));
                tmem_ld_wait();
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t code = code_slow(__uint_as_float(v[i]) * rc.rinv, raw, 15);
                (i < 8 ? g0 : g1) |= code << (4 * (i & 7));
                if constexpr (QJL) residual(i, code);
            }
        }
    }
}

// Appends a group of eight codes (8 * BITS bits) to a row's bit stream held in words[]: group k sits at bit 8 * BITS * k.
template <int BITS, int NW>
__device__ __forceinline__ void put_group(uint32_t (&words)[NW], int k, uint32_t g) {
    constexpr int GB = 8 * BITS;
    const int bit = GB * k, w = bit >> 5, sh = bit & 31;                          // all compile-time after unrolling
    words[w] |= g << sh;
    if (sh + GB > 32 && w + 1 < NW) words[w + 1] |= g >> (32 - sh);
}

// nbytes of words[] to dst with the widest stores the address and the size allow (both known per row only)
template <int NW>
__device__ __forceinline__ void store_words(uint8_t* dst, const uint32_t (&words)[NW], int nbytes) {
    const uint32_t al = uint32_t(reinterpret_cast<uintptr_t>(dst)) | uint32_t(nbytes);
    if ((al & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i)
            if (16 * i < nbytes) reinterpret_cast<uint4*>(dst)[i] = make_uint4(words[4 * i], words[4 * i + 1], words[4 * i + 2], words[4 * i + 3]);
    } else if ((al & 7u) == 0) {
#pragma unroll
        for (int i = 0; i < NW / 2; ++i)
            if (8 * i < nbytes) reinterpret_cast<uint2*>(dst)[i] = make_uint2(words[2 * i], words[2 * i + 1]);
    } else if ((al & 3u) == 0) {
#pragma unroll
        for (int i = 0; i < NW; ++i)
            if (4 * i < nbytes) reinterpret_cast<uint32_t*>(dst)[i] = words[i];
    } else {                                                                      // rows of 6 or 18 bytes: 2-byte aligned
#pragma unroll
        for (int i = 0; i < 2 * NW; ++i)
            if (2 * i < nbytes) reinterpret_cast<uint16_t*>(dst)[i] = uint16_t(words[i >> 1] >> (16 * (i & 1)));
    }
}

struct EpiCtx {
    const Params& p; unsigned char* smem; uint32_t tmem_base, bar_accfull, bar_accfree, bar_afree, bar_nrm, bar_res, bar_proj;
    volatile int* abort_flag; int warp, lane;
    uint8_t* dst; int nb; bool write_norms;        // head_dim 256: the slice's first byte, bytes of a packed row, this slice writes the norms
};

// QJL: the residual of sixteen coordinates (normalised rotated value minus its centroid) enters the residual's sum of squares and goes back
// into tensor memory, into the sixteen columns it came from: it is the A operand of the 32 projections, a product of 128 x d by d x 32 a
// tile.  Only the SIGN of a projection is kept, so the residual is scaled by 2^8 (clear of fp16 subnormals) and split into fp16 high and low
// parts (columns 0-7 and 8-15), as is S R^T: hi x hi + lo x hi + hi x lo reproduces the float32 product to about 2^-21.
// (With mma.sync a thread kept 32 running projections, a warp staged its residuals through shared memory, and the registers allowed eight
// epilogue warps: keys at 4 bits and values at 2 of 1,048,576 rows of 96 took 196 + 168 us, 146 + 118 now; the signs are the same.)
__device__ __forceinline__ void sketch16(const uint32_t* e, uint32_t taddr, u64& ee) {
    uint32_t x[16];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const float e2[2] = {__uint_as_float(e[i]), __uint_as_float(e[i + 1])};
        const u64 ev = pk(e2[0], e2[1]);
        ee = fma2(ev, ev, ee);
        const __half2 h = __floats2half2_rn(e2[0], e2[1]);
        const float2 hf = __half22float2(h);
        float l0, l1;
        upk(add2(ev, pk(-hf.x, -hf.y)), l0, l1);
        const __half2 l = __floats2half2_rn(l0, l1);
        x[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
        x[8 + (i >> 1)] = *reinterpret_cast<const uint32_t*>(&l);
    }
    tmem_st16(taddr, x);
}

// A run of a row's coordinates ([col0, col0 + 16 * nch) at BITS bits) in rolled steps of 32 coordinates, 16 with the sketch; the step's codes
// are assembled in registers and stored at once.  Keeping the loop rolled keeps its body within the instruction cache (with 32 coordinates a
// step the sketch's warps stood 2.7 of 9.4 cycles an instruction without one, with 16 0.5 of 7.8: keys and values of 8 x 65,536 rows of 96
// at 4 and 2 bits 147.7 us before, 134.9 now).  SPLITACC: the high and low products sit in two accumulators lo_off columns apart and are combined
// here (y = hi + 2^-11 lo), sixteen coordinates per pair of loads; otherwise one load per step.
// NCH: the number of chunks when it is known at compile time (1 or 2: a single step whose shape folds), 0 = nch_rt.
template <int BITS, bool QJL, bool SPLITACC, int NCH, int TERMS = 2>
__device__ __forceinline__ void quantize_part(uint32_t t_row, int col0, int nch_rt, int lo_off, const RowCtx& rc, const float (&sb)[7], const float* raw,
                                              const float* cent, uint8_t* dst, bool live, u64& ee) {
    constexpr int STEP = QJL ? 1 : 2, NW = (STEP * 16 * BITS + 31) / 32;            // chunks of a step and its words
    const int nch = NCH ? NCH : nch_rt;
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += STEP) {
        uint32_t v[32], w[NW];
#pragma unroll
        for (int i = 0; i < NW; ++i) w[i] = 0;
        const int nc = min(STEP, nch - c0);                                         // a run may end on a half step
        if (!SPLITACC && !QJL) {
            tmem_ld32(t_row + col0 + c0 * 16, v);
            tmem_ld_wait();
        }
#pragma unroll
        for (int c = 0; c < STEP; ++c) {
            if (c < nc) {
                uint32_t g0, g1;
                uint32_t* vc = v + ((SPLITACC || QJL) ? 0 : 16 * c);
                if (QJL && !SPLITACC) {                                         // (they are replaced in place: sixteen columns at a time)
                    tmem_ld16(t_row + col0 + (c0 + c) * 16, *reinterpret_cast<uint32_t (*)[16]>(v));
                    tmem_ld_wait();
                }
                if (SPLITACC) {
                    uint32_t (&hi)[16] = *reinterpret_cast<uint32_t (*)[16]>(v);
                    uint32_t (&lo)[16] = *reinterpret_cast<uint32_t (*)[16]>(v + 16);
                    tmem_ld16(t_row + col0 + (c0 + c) * 16, hi);
                    tmem_ld16(t_row + lo_off + col0 + (c0 + c) * 16, lo);
                    if constexpr (TERMS == 3) {                                     // three bf16 terms of equal weight, smallest first
                        uint32_t t3[16];
                        tmem_ld16(t_row + 2 * lo_off + col0 + (c0 + c) * 16, t3);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __float_as_uint((__uint_as_float(t3[i]) + __uint_as_float(v[16 + i])) + __uint_as_float(v[i]));
                    } else {
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            float y0, y1;
                            upk(fma2(pk(__uint_as_float(v[16 + i]), __uint_as_float(v[17 + i])), pk(1.f / 2048.f, 1.f / 2048.f), pk(__uint_as_float(v[i]), __uint_as_float(v[i + 1]))), y0, y1);
                            v[i] = __float_as_uint(y0);
                            v[i + 1] = __float_as_uint(y1);
                        }
                    }
                }
                quantize16<BITS, QJL, SPLITACC>(vc, rc, sb, raw, g0, g1, cent, t_row + col0 + (c0 + c) * 16);
                put_group<BITS, NW>(w, 2 * c, g0);
                put_group<BITS, NW>(w, 2 * c + 1, g1);
                if constexpr (QJL) sketch16(vc, t_row + col0 + (c0 + c) * 16, ee);
            }
        }
        if (live) store_words<NW>(dst + c0 * 2 * BITS, w, nc * 2 * BITS);
    }
}

__device__ __forceinline__ uint32_t sbase_of(const EpiCtx& e) { return static_cast<uint32_t>(__cvta_generic_to_shared(e.smem)); }

// BH bits for coordinates [0, half), BL for [half, d) (BL == 0: BH for all of them, half = d).  Three shapes:
//   fp16 rows (SPLITACC): two accumulators per tile (high and low products: two independent chains of MMAs instead of
//     one twice as long) leave room for two stages, so all sixteen warps work on the same tile in step - thread <-> one
//     row and a quarter of its sixteen-coordinate chunks (of either width) - while the MMAs of the next tile run.
//   bf16 rows: one accumulator per tile, four stages; two groups of eight warps take alternate tiles (two stages each),
//     a thread owns one row and half of its chunks.
//   QJL sketch: as bf16 rows, three stages: a group hands its residuals to the MMA warp, waits for the tile's projections while
//     the other group works, and signs them; the MMAs of a third tile run meanwhile.
template <bool QJL, bool SPLITACC> struct EpiShape {
    static constexpr int GROUPS = SPLITACC ? 1 : 2;                                 // groups of warps that take tiles in turn
    static constexpr int WPG = EPI_WARPS / GROUPS;                                  // warps per group: 4 row quadrants x SPLIT shares of the columns
    static constexpr int SPLIT = WPG / 4;
    static constexpr int STAGES = SPLITACC ? 2 : QJL ? SK_STAGES : 4;               // accumulator stages
    static constexpr int STAGE_COLS = SPLITACC ? 2 * DMAX : DMAX;
};
// DC: head_dim when it is known at compile time (the chunk shares, row widths and store shapes then fold), 0 = read it
// from the parameters.
template <int BH, int BL, bool QJL, bool SPLITACC, int DC, int TERMS = 2>
__device__ __forceinline__ void epilogue_loop(const EpiCtx& e) {
    using Sh = EpiShape<QJL, SPLITACC>;
    const Params& p = e.p;
    const int group = e.warp / Sh::WPG, quad = e.warp & 3, part = (e.warp % Sh::WPG) >> 2, row_in_tile = quad * 32 + e.lane;
    const int d = DC == 256 ? SLICE : DC ? DC : p.d, half = BL ? d / 2 : d;
    const int nch_h = half / 16, nch_l = BL ? (d - half) / 16 : 0;                   // chunks of sixteen coordinates per bit width
    // this thread's chunks: [h0, h1) of the first width, [l0, l1) of the second
    // (share q of n chunks: [ceil(q n / SPLIT), ceil((q + 1) n / SPLIT)); the second width is dealt from the other end so
    // that the shares of a fractional row add up evenly)
    const int h0 = (part * nch_h + Sh::SPLIT - 1) / Sh::SPLIT, h1 = ((part + 1) * nch_h + Sh::SPLIT - 1) / Sh::SPLIT;
    const int l0 = part * nch_l / Sh::SPLIT, l1 = (part + 1) * nch_l / Sh::SPLIT;
    const float* raw_h = reinterpret_cast<const float*>(e.smem + OFF_BND);
    const float* raw_l = raw_h + 16;
    const float* cent_h = raw_h + 32;
    const float* cent_l = raw_h + 48;
    RowCtx rc;
    rc.bins = reinterpret_cast<const float2*>(e.smem + OFF_BINS) + (e.lane & (BIN_REP - 1));      // 4-bit side only
    float bnd_h[7], bnd_l[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) { bnd_h[i] = raw_h[(BH <= 3 && i < (1 << BH) - 1) ? i : 0]; bnd_l[i] = raw_l[(BL >= 1 && BL <= 3 && i < (1 << BL) - 1) ? i : 0]; }
    const uint32_t tpl = uint32_t(p.tiles_per_lane);
    const int a_stages = p.a_stages;
    const int nb_h = half * BH / 8, nb_l = BL ? (d - half) * BL / 8 : 0;            // bytes of a packed row (per width)
    int s = group % a_stages;                                                       // operand stage of iteration `it`
    // (cache lane, tile inside the lane) of the group's current tile, advanced by the group's tile stride: one division here
    constexpr uint32_t CPT = DC == 256 ? 4 : 1;                                     // CTAs per tile
    const uint32_t first_tile = (blockIdx.x + uint32_t(group) * gridDim.x) / CPT, stride_tiles = uint32_t(Sh::GROUPS) * gridDim.x / CPT;
    uint32_t lane_o = first_tile / tpl, tl = first_tile - lane_o * tpl;
    const uint32_t step_o = stride_tiles / tpl, step_t = stride_tiles - step_o * tpl;
    for (int64_t tile = first_tile, it = group; tile < p.n_tiles; tile += stride_tiles, it += Sh::GROUPS) {
        const int a = int(it % Sh::STAGES);
        if (!mbar_wait(e.bar_accfull + 8 * a, uint32_t(it / Sh::STAGES) & 1u, e.abort_flag, 3)) break;
        float nrm;
        if constexpr (DC == 256) {
            const int q = int(it % NSQ_SLOTS);
            if (!mbar_wait(sbase_of(e) + OFF_NRMBAR256 + 8 * q, uint32_t(it / NSQ_SLOTS) & 1u, e.abort_flag, 5)) break;
            tc_fence_after();
            // (the slot is written again eight tiles on, by which time this tile's accumulator has been freed and used again)
            nrm = sqrtf(reinterpret_cast<const float*>(e.smem + OFF_NSQ256)[q * TM + row_in_tile]);
        } else {
            if (!mbar_wait(e.bar_nrm + 8 * s, uint32_t(it / a_stages) & 1u, e.abort_flag, 5)) break;     // sums of squares written
            tc_fence_after();
            const float* nsq = reinterpret_cast<const float*>(e.smem + OFF_NSQ) + s * 2 * TM;
            nrm = sqrtf(nsq[row_in_tile] + nsq[TM + row_in_tile]);
            mbar_arrive(e.bar_afree + 8 * s);                       // norm slots of this stage are free again
            s = (s + Sh::GROUPS) % a_stages;
        }
        const float nden = fmaxf(nrm, 1e-10f);                  // cache.py:237-238 guards the zero vector the same way
        rc.rinv = 1.f / nden;
        rc.rbin = rc.rinv * 256.f;
        // register search: y / |x| > b is tested as y > b * |x| (one multiply per boundary and row instead of one per coordinate)
        float sb_h[7], sb_l[7];
#pragma unroll
        for (int i = 0; i < 7; ++i) { sb_h[i] = bnd_h[i] * nden; sb_l[i] = bnd_l[i] * nden; }
        const int64_t lane_r = int64_t(tl) * TM + row_in_tile;
        const bool live = lane_r < p.n_rows;                    // rows past the lane's end were zero-filled by the copy
        const int64_t orow = int64_t(lane_o) * p.out_lane_stride + lane_r;
        lane_o += step_o; tl += step_t;
        if (tl >= tpl) { tl -= tpl; ++lane_o; }
        const uint32_t t_row = e.tmem_base + (uint32_t(quad * 32) << 16) + a * Sh::STAGE_COLS;
        u64 ee2 = 0;                                            // squares of the residual: even and odd coordinates
        // with head_dim 128 and quarter shares every thread has two chunks of an integer width, or one of each fractional width
        constexpr int NCH_H = (DC == 128 && Sh::SPLIT == 4) ? (BL ? 1 : 2) : 0, NCH_L = (DC == 128 && Sh::SPLIT == 4) ? 1 : 0;
        if constexpr (DC == 256)
            quantize_part<BH, QJL, SPLITACC, 1, TERMS>(t_row, h0 * 16, 1, SLICE, rc, sb_h, raw_h, cent_h, e.dst + orow * e.nb + h0 * 2 * BH, live, ee2);
        else
        quantize_part<BH, QJL, SPLITACC, NCH_H>(t_row, h0 * 16, h1 - h0, d, rc, sb_h, raw_h, cent_h, p.p_hi + orow * nb_h + h0 * 2 * BH, live, ee2);
        if (BL) quantize_part<(BL ? BL : 1), QJL, SPLITACC, NCH_L>(t_row, half + l0 * 16, l1 - l0, d, rc, sb_l, raw_l, cent_l, p.p_lo + orow * nb_l + l0 * 2 * BL, live, ee2);
        if constexpr (QJL) {
            static_assert(Sh::SPLIT == 2, "two threads a row");
            float* ee_slot = reinterpret_cast<float*>(e.smem + OFF_EE) + a * TM + row_in_tile;
            float ee, ee_odd;
            upk(ee2, ee, ee_odd);
            ee += ee_odd;
            if (part == 1) *ee_slot = ee;
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(e.bar_res + 8 * a);                     // residuals and squares of this share are there
            const uint32_t ph = uint32_t(it / Sh::STAGES) & 1u;
            if (!mbar_wait(e.bar_res + 8 * a, ph, e.abort_flag, 4) || !mbar_wait(e.bar_proj + 8 * a, ph, e.abort_flag, 8)) break;
            tc_fence_after();
            uint32_t pr[16], zb = 0;                            // this thread's half of the row's projections
            tmem_ld16(e.tmem_base + (uint32_t(quad * 32) << 16) + SK_COL0 + a * QM + part * 16, pr);
            tmem_ld_wait();
            if (part == 0) ee += *ee_slot;
            tc_fence_before();
            mbar_arrive(e.bar_accfree + 8 * a);                 // the accumulator may be overwritten
#pragma unroll
            for (int i = 0; i < 16; ++i) zb |= __uint_as_float(pr[i]) >= 0.f ? 1u << i : 0u;
            if (live) {
                reinterpret_cast<uint16_t*>(p.qjl_bits + orow)[part] = uint16_t(nrm == 0.f ? 0xffffu : zb);     // zero row: the reference's residual is exactly 0, and 0 >= 0
                if (part == 0) {
                    p.norms[orow] = nrm;
                    p.qjl_gamma[orow] = nrm * sqrtf(ee) * (1.f / 256.f);   // |x - dequant(x)| = |x| |y_n - c| (the rotation is orthogonal); ee sums 2^16 times the squares
                }
            }
        } else {
            tc_fence_before();
            mbar_arrive(e.bar_accfree + 8 * a);                     // the accumulator may be overwritten
            if (live && part == 0 && (DC != 256 || e.write_norms)) p.norms[orow] = nrm;
        }
    }
}

// SPLITACC (fp16 rows without the sketch): high and low products in two accumulators, one MMA of N = 2 d per k-step
// against [R_hi ; R_lo].  Otherwise one accumulator: fp16 low products first and the scale-input-d trick, bf16 three terms.
template <bool QJL, bool SPLITACC, int DC>
__global__ void __launch_bounds__(n_threads(SPLITACC), 1) quantize_tc_kernel(Params p, const __grid_constant__ CUtensorMap tmap) {
    using Sh = EpiShape<QJL, SPLITACC>;
    constexpr int ACCS = Sh::STAGES, N_NORM = n_norm(SPLITACC), NT = n_threads(SPLITACC);
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // (warp: uniform)
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 4);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
    const int d = DC ? DC : p.d, a_stages = p.a_stages;
    const bool bf16 = p.bf16 != 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");        // (an independent job of the same call takes the SMs this one leaves idle)
    // barriers: full[3] (TMA -> MMA, norms), a_free[3] (MMA commit + norm warps + the epilogue's norm read -> TMA),
    //           nrm[3] (norm warps -> epilogue), acc_full[4] (MMA commit -> epilogue group), acc_free[4] (epilogue group -> MMA)
    const uint32_t bar_full = sbase + OFF_BAR, bar_afree = bar_full + 8 * A_STAGES_MAX, bar_nrm = bar_afree + 8 * A_STAGES_MAX;
    const uint32_t bar_accfull = bar_nrm + 8 * A_STAGES_MAX, bar_accfree = bar_accfull + 8 * ACC_STAGES;      // (ACCS of the 4 slots are used)
    const uint32_t bar_drain = bar_accfree + 8 * ACC_STAGES;              // products in flight when a wait ran out
    const uint32_t bar_res = bar_drain + 8, bar_proj = bar_res + 8 * SK_STAGES;       // QJL: residuals of a stage written (epilogue group -> MMA), its projections done (MMA commit -> group)

    if (sbase & 1023u) {                  // the swizzled operand tiles need 1024-byte alignment (uniform across the CTA)
        if (tid == 0) atomicCAS(&g_status, 0, 9);
        if (p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < A_STAGES_MAX; ++s) {
            // one arrival (the issuing thread, with the byte count) fills a stage; it is free again once the MMAs have
            // committed, the norm warps have read the rows and the tile's epilogue group has read the norms
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_afree + 8 * s, 1 + N_NORM + (DC == 256 ? 0 : N_EPI / Sh::GROUPS));
            mbar_init(bar_nrm + 8 * s, N_NORM);
        }
        if (DC == 256)
            for (int q = 0; q < NSQ_SLOTS; ++q) mbar_init(sbase + OFF_NRMBAR256 + 8 * q, N_NORM);
        mbar_init(bar_drain, 1);
        for (int a = 0; a < SK_STAGES; ++a) { mbar_init(bar_res + 8 * a, N_EPI / Sh::GROUPS); mbar_init(bar_proj + 8 * a, 1); }
        for (int a = 0; a < ACC_STAGES; ++a) { mbar_init(bar_accfull + 8 * a, 1); mbar_init(bar_accfree + 8 * a, N_EPI / Sh::GROUPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // head_dim 256: this CTA's slice of the columns, its width and its bytes of a packed row
    const int slice = DC == 256 ? int(blockIdx.x & 3u) : 0;
    const bool in_lo = DC == 256 && p.bits_lo != 0 && slice >= 2;
    const int slice_bits = in_lo ? p.bits_lo : p.bits_hi;
    const uint32_t tile0 = DC == 256 ? blockIdx.x >> 2 : blockIdx.x, tile_step = DC == 256 ? gridDim.x >> 2 : gridDim.x;
    if constexpr (DC == 256) {
        // operand rows: term t of slice row j at row 64 t + j, K-blocks of (64 TERMS) rows x 128 bytes
        const int terms = bf16 ? 3 : 2, kb_bytes = terms * SLICE * 128;
        unsigned char* rbase = smem + (bf16 ? OFF_R3 : OFF_R1);
        for (int idx = tid; idx < SLICE * 32; idx += NT) {
            const int j = idx >> 5, c = idx & 31, kblk = c >> 3, cc = c & 7;
            const float* src = p.rot + (slice * SLICE + j) * 256 + c * 8;
            const float4 f0 = __ldg(reinterpret_cast<const float4*>(src)), f1 = __ldg(reinterpret_cast<const float4*>(src + 4));
            float v[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
            for (int t = 0; t < terms; ++t) {
                __align__(16) uint16_t w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (bf16) {
                        const __nv_bfloat16 h = __float2bfloat16_rn(v[i]);
                        w[i] = __bfloat16_as_ushort(h);
                        v[i] -= __bfloat162float(h);                          // exact
                    } else {
                        const __half h = __float2half_rn(v[i]);
                        w[i] = __half_as_ushort(h);
                        v[i] = (v[i] - __half2float(h)) * 2048.f;
                    }
                }
                const int r = t * SLICE + j;
                *reinterpret_cast<uint4*>(rbase + kblk * kb_bytes + r * 128 + ((cc ^ (r & 7)) << 4)) = *reinterpret_cast<const uint4*>(w);
            }
        }
    } else
    // R -> operand tiles (swizzled K-major): B[n = j][k] = R[j][k], rows j < d, 16-byte chunks c < d / 8
    for (int idx = tid; idx < d * (d / 8); idx += NT) {
        const int j = idx / (d / 8), c = idx - j * (d / 8);      // row j, chunk c (8 elements) of the row
        const float4 f0 = __ldg(reinterpret_cast<const float4*>(p.rot + j * d + c * 8));
        const float4 f1 = __ldg(reinterpret_cast<const float4*>(p.rot + j * d + c * 8 + 4));
        const float v[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
        const int kblk = c >> 3, cc = c & 7;
        const int off = kblk * KBLK_BYTES + j * 128 + ((cc ^ (j & 7)) << 4);
        if (SPLITACC) {
            // one operand of 2 d rows per K-block: row j = R_hi[j], row d + j = 2^11 R_lo[j] (K-blocks 32 KB apart)
            __align__(16) __half hi[8], lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                hi[i] = __float2half_rn(v[i]);
                lo[i] = __float2half_rn((v[i] - __half2float(hi[i])) * 2048.f);
            }
            const int jl = d + j;
            *reinterpret_cast<uint4*>(smem + OFF_R1 + kblk * (2 * KBLK_BYTES) + j * 128 + ((cc ^ (j & 7)) << 4)) = *reinterpret_cast<const uint4*>(hi);
            *reinterpret_cast<uint4*>(smem + OFF_R1 + kblk * (2 * KBLK_BYTES) + jl * 128 + ((cc ^ (jl & 7)) << 4)) = *reinterpret_cast<const uint4*>(lo);
        } else if (!bf16) {
            __align__(16) __half hi[8], lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                hi[i] = __float2half_rn(v[i]);
                lo[i] = __float2half_rn((v[i] - __half2float(hi[i])) * 2048.f);
            }
            *reinterpret_cast<uint4*>(smem + OFF_R1 + off) = *reinterpret_cast<const uint4*>(hi);
            *reinterpret_cast<uint4*>(smem + OFF_R2 + off) = *reinterpret_cast<const uint4*>(lo);
        } else {
            __align__(16) __nv_bfloat16 t1[8], t2[8], t3[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                t1[i] = __float2bfloat16_rn(v[i]);
                const float r1 = v[i] - __bfloat162float(t1[i]);               // exact
                t2[i] = __float2bfloat16_rn(r1);
                t3[i] = __float2bfloat16_rn(r1 - __bfloat162float(t2[i]));     // exact remainder, 8 bits left at most
            }
            *reinterpret_cast<uint4*>(smem + OFF_R1 + off) = *reinterpret_cast<const uint4*>(t1);
            *reinterpret_cast<uint4*>(smem + OFF_R2 + off) = *reinterpret_cast<const uint4*>(t2);
            *reinterpret_cast<uint4*>(smem + OFF_R3 + off) = *reinterpret_cast<const uint4*>(t3);
        }
    }
    {
        float* raw = reinterpret_cast<float*>(smem + OFF_BND);
        if (tid < 64) {
            const int which = tid >> 4, i = tid & 15;                    // 0 / 1: boundaries hi / lo, 2 / 3: centroids hi / lo
            const int bits = DC == 256 ? slice_bits : (which & 1) ? p.bits_lo : p.bits_hi;
            float val = which < 2 ? INFINITY : 0.f;
            if (which < 2) {
                const float* src = (DC == 256 ? in_lo : which != 0) ? p.bnd_lo : p.bnd_hi;
                if (src != nullptr && bits > 0 && i < (1 << bits) - 1) val = src[i];
            } else if (QJL) {
                const float* src = (which & 1) ? p.cent_lo : p.cent_hi;
                if (src != nullptr && bits > 0 && i < (1 << bits)) val = src[i] * 256.f;     // (the sketch works on 2^8 times the residual)
            }
            raw[tid] = val;
        }
        if (QJL) {
            // (S R^T) is (32, d): row = projection, K-blocks of 64 coordinates, swizzled like R
            for (int idx = tid; idx < QM * (d / 8); idx += NT) {
                const int j = idx / (d / 8), c = idx - j * (d / 8);
                const float* srow = p.qjl_proj_rot + j * d + c * 8;
                __align__(16) __half hi[8], lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float x = __ldg(srow + i);
                    hi[i] = __float2half_rn(x);
                    lo[i] = __float2half_rn(x - __half2float(hi[i]));
                }
                unsigned char* dst = smem + OFF_PT + (c >> 3) * PT_KBLK + j * 128 + (((c & 7) ^ (j & 7)) << 4);
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(hi);
                *reinterpret_cast<uint4*>(dst + 2 * PT_KBLK) = *reinterpret_cast<const uint4*>(lo);
            }
        }
        __syncthreads();
        if ((DC == 256 ? slice_bits : p.bits_hi) == 4) build_bins(reinterpret_cast<float2*>(smem + OFF_BINS), raw, 15, tid, NT);
    }
    if (warp == EPI_WARPS) {              // one warp owns the TMEM allocation
        tmem_alloc(sbase + OFF_MISC, 512);
        tmem_relinquish();
    }
    fence_proxy_async();                  // the operand tiles written above are read by the tensor core
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t oper_bytes = d > 64 ? OPER_BYTES : KBLK_BYTES;        // bytes one tile's copies deliver

    if (warp < EPI_WARPS) {
        // ======================= epilogue: row = 32 * (warp % 4) + lane; groups and column halves as in EpiShape =======================
        EpiCtx e{p, smem, tmem_base, bar_accfull, bar_accfree, bar_afree, bar_nrm, bar_res, bar_proj, abort_flag, warp, lane, nullptr, 0, true};
        if constexpr (DC == 256) {
            const int coords = p.bits_lo ? 128 : 256;                      // of a packed row of this slice's width
            e.nb = coords * slice_bits / 8;
            e.dst = (in_lo ? p.p_lo : p.p_hi) + (slice * SLICE - (in_lo ? 128 : 0)) * slice_bits / 8;
            e.write_norms = slice == 0;
            if (bf16) {
                switch (slice_bits) {
                    case 4: epilogue_loop<4, 0, false, true, 256, 3>(e); break;
                    case 3: epilogue_loop<3, 0, false, true, 256, 3>(e); break;
                    case 2: epilogue_loop<2, 0, false, true, 256, 3>(e); break;
                    default: epilogue_loop<1, 0, false, true, 256, 3>(e); break;
                }
            } else {
                switch (slice_bits) {
                    case 4: epilogue_loop<4, 0, false, true, 256, 2>(e); break;
                    case 3: epilogue_loop<3, 0, false, true, 256, 2>(e); break;
                    case 2: epilogue_loop<2, 0, false, true, 256, 2>(e); break;
                    default: epilogue_loop<1, 0, false, true, 256, 2>(e); break;
                }
            }
        } else
        switch (p.bits_hi * 8 + p.bits_lo) {
            case 4 * 8 + 0: epilogue_loop<4, 0, QJL, SPLITACC, DC>(e); break;
            case 3 * 8 + 0: epilogue_loop<3, 0, QJL, SPLITACC, DC>(e); break;
            case 2 * 8 + 0: epilogue_loop<2, 0, QJL, SPLITACC, DC>(e); break;
            case 1 * 8 + 0: epilogue_loop<1, 0, QJL, SPLITACC, DC>(e); break;
            case 4 * 8 + 3: epilogue_loop<4, 3, QJL, SPLITACC, DC>(e); break;
            case 3 * 8 + 2: epilogue_loop<3, 2, QJL, SPLITACC, DC>(e); break;
            case 2 * 8 + 1: epilogue_loop<2, 1, QJL, SPLITACC, DC>(e); break;
            default: break;               // the host only launches the combinations above
        }
    } else if (warp == EPI_WARPS) {
        // ======================= MMA issue: the whole warp in uniform control flow, one elected lane issues =======================
        auto wait_all = [&](uint32_t bar, uint32_t parity, volatile int* flag, int code) { return bool(__all_sync(0xffffffffu, mbar_wait(bar, parity, flag, code))); };
        if (DC == 256) {
            {
                const int terms = bf16 ? 3 : 2, kb_bytes = terms * SLICE * 128;
                const uint32_t idesc = make_idesc(terms * SLICE, bf16), rb = sbase + (bf16 ? OFF_R3 : OFF_R1);
                int it = 0, hit = 0;
                bool ok = true;
                for (int64_t tile = tile0; ok && tile < p.n_tiles; tile += tile_step, ++it) {
                    const int a = it % ACCS;
                    if (it >= ACCS && !wait_all(bar_accfree + 8 * a, uint32_t((it / ACCS) - 1) & 1u, abort_flag, 2)) break;
                    for (int kh = 0; kh < 2; ++kh, ++hit) {
                        const int s = hit % a_stages;
                        ok = wait_all(bar_full + 8 * s, uint32_t(hit / a_stages) & 1u, abort_flag, 1);
                        if (!ok) break;
                        tc_fence_after();
                        for (int ks = 0; ks < 8; ++ks) {
                            const int kblk = kh * 2 + (ks >> 2);
                            umma_f16(tmem_base + a * Sh::STAGE_COLS, smem_desc(sbase + OFF_A + s * OPER_BYTES, ks >> 2, ks & 3), smem_desc(rb + kblk * kb_bytes, 0, ks & 3), idesc,
                                     (kh | ks) ? 1u : 0u);
                        }
                        umma_commit(bar_afree + 8 * s);
                    }
                    if (ok) umma_commit(bar_accfull + 8 * a);
                }
            }
        } else
        {
            const uint32_t idesc = make_idesc(SPLITACC ? 2 * d : d, bf16);
            const int ksteps = d / 16;
            // QJL: the projections of tile `n` of this CTA, in the order that leaves the next tiles' products in front of them
            const uint32_t idesc_p = make_idesc(QM, false);
            auto project = [&](int n) {
                const int a = n % ACCS;
                if (!wait_all(bar_res + 8 * a, uint32_t(n / ACCS) & 1u, abort_flag, 4)) return false;
                tc_fence_after();
                const uint32_t res = tmem_base + a * Sh::STAGE_COLS, acc = tmem_base + SK_COL0 + a * QM;
                for (int ks = 0; ks < ksteps; ++ks) {
                    const uint64_t hi = smem_desc(sbase + OFF_PT + (ks >> 2) * PT_KBLK, 0, ks & 3), lo = smem_desc(sbase + OFF_PT + (2 + (ks >> 2)) * PT_KBLK, 0, ks & 3);
                    umma_f16_ta(acc, res + 16 * ks, hi, idesc_p, ks ? 1u : 0u);
                    umma_f16_ta(acc, res + 16 * ks + 8, hi, idesc_p, 1u);
                    umma_f16_ta(acc, res + 16 * ks, lo, idesc_p, 1u);
                }
                umma_commit(bar_proj + 8 * a);
                return true;
            };
            int it = 0;
            for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++it) {
                const int a = it % ACCS, s = it % a_stages;
                if (it >= ACCS && !wait_all(bar_accfree + 8 * a, uint32_t((it / ACCS) - 1) & 1u, abort_flag, 2)) break;
                if (!wait_all(bar_full + 8 * s, uint32_t(it / a_stages) & 1u, abort_flag, 1)) break;
                tc_fence_after();
                const uint32_t a_tile = sbase + OFF_A + s * OPER_BYTES;
                const uint32_t d_acc = tmem_base + a * Sh::STAGE_COLS;
                if (SPLITACC) {
                    // columns [0, d): x.R_hi, columns [d, 2 d): 2^11 x.R_lo; the operand's K-blocks are 32 KB apart
                    for (int ks = 0; ks < ksteps; ++ks)
                        umma_f16(d_acc, smem_desc(a_tile, ks >> 2, ks & 3), smem_desc(sbase + OFF_R1 + (ks >> 2) * KBLK_BYTES, ks >> 2, ks & 3), idesc, ks ? 1u : 0u);
                } else if (!bf16) {
                    for (int ks = 0; ks < ksteps; ++ks)            // 2^11-scaled low products first
                        umma_f16(d_acc, smem_desc(a_tile, ks >> 2, ks & 3), smem_desc(sbase + OFF_R2, ks >> 2, ks & 3), idesc, ks ? 1u : 0u);
                    umma_f16_scaled11(d_acc, smem_desc(a_tile, 0, 0), smem_desc(sbase + OFF_R1, 0, 0), idesc);    // acc = x.R_hi + 2^-11 acc
                    for (int ks = 1; ks < ksteps; ++ks)
                        umma_f16(d_acc, smem_desc(a_tile, ks >> 2, ks & 3), smem_desc(sbase + OFF_R1, ks >> 2, ks & 3), idesc, 1u);
                } else {
                    const int r_off[3] = {OFF_R3, OFF_R2, OFF_R1};   // smallest term first
                    for (int term = 0; term < 3; ++term)
                        for (int ks = 0; ks < ksteps; ++ks)
                            umma_f16(d_acc, smem_desc(a_tile, ks >> 2, ks & 3), smem_desc(sbase + r_off[term], ks >> 2, ks & 3), idesc, (term | ks) ? 1u : 0u);
                }
                umma_commit(bar_afree + 8 * s);      // rows of this stage consumed
                umma_commit(bar_accfull + 8 * a);    // the accumulator is complete: its epilogue group may read it
                if (QJL && it >= ACCS - 1 && !project(it - (ACCS - 1))) break;
            }
            if (QJL)
                for (int n = max(0, it - (ACCS - 1)); n < it && !__any_sync(0xffffffffu, *abort_flag != 0); ++n)
                    if (!project(n)) break;
        }
        if (__any_sync(0xffffffffu, *abort_flag != 0)) { umma_commit(bar_drain); mbar_drain(bar_drain, 0); }
        __syncwarp();
    } else if (warp == EPI_WARPS + 1 + N_NORM / 32) {
        // ======================= TMA issue: one thread keeps the operand stages full =======================
        if (DC == 256) {
            if (lane == 0) {
                const uint32_t tpl = uint32_t(p.tiles_per_lane);
                int hit = 0;
                bool ok = true;
                for (int64_t tile = tile0; ok && tile < p.n_tiles; tile += tile_step) {
                    const uint32_t t32 = uint32_t(tile), o = t32 / tpl, tl = t32 - o * tpl;
                    for (int kh = 0; kh < 2 && ok; ++kh, ++hit) {
                        const int s = hit % a_stages;
                        if (hit >= a_stages) ok = mbar_wait(bar_afree + 8 * s, uint32_t((hit / a_stages) - 1) & 1u, abort_flag, 6);
                        if (!ok) break;
                        const uint32_t a_tile = sbase + OFF_A + s * OPER_BYTES;
                        mbar_expect_tx(bar_full + 8 * s, OPER_BYTES);
                        tma_load_3d(a_tile, &tmap, kh * 128, int(tl * TM), int(o), bar_full + 8 * s);
                        tma_load_3d(a_tile + KBLK_BYTES, &tmap, kh * 128 + 64, int(tl * TM), int(o), bar_full + 8 * s);
                    }
                }
                for (int h = hit > a_stages ? hit - a_stages : 0; h < hit; ++h) mbar_drain(bar_full + 8 * (h % a_stages), uint32_t(h / a_stages) & 1u);
            }
        } else
        if (lane == 0) {
            const uint32_t tpl = uint32_t(p.tiles_per_lane);
            int it = 0;
            for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++it) {
                const int s = it % a_stages;
                if (it >= a_stages && !mbar_wait(bar_afree + 8 * s, uint32_t((it / a_stages) - 1) & 1u, abort_flag, 6)) break;
                const uint32_t t32 = uint32_t(tile), o = t32 / tpl, tl = t32 - o * tpl;
                const uint32_t a_tile = sbase + OFF_A + s * OPER_BYTES;
                mbar_expect_tx(bar_full + 8 * s, oper_bytes);
                tma_load_3d(a_tile, &tmap, 0, int(tl * TM), int(o), bar_full + 8 * s);                              // columns 0..63
                if (d > 64) tma_load_3d(a_tile + KBLK_BYTES, &tmap, 64, int(tl * TM), int(o), bar_full + 8 * s);    // columns 64..127 (zeros past d)
            }
            for (int i = it > a_stages ? it - a_stages : 0; i < it; ++i) mbar_drain(bar_full + 8 * (i % a_stages), uint32_t(i / a_stages) & 1u);
        }
        __syncwarp();
    } else {
        // ======================= norm warps: sum of squares of every row, read back from the stage =======================
        // thread -> row 32 nw + lane (and the one 64 further), both 64-column blocks: eight consecutive rows hit eight different 16-byte columns
        // of the swizzled tile, so the 128-bit reads are free of bank conflicts
        const int nw = warp - (EPI_WARPS + 1), r = nw * 32 + lane;
        constexpr int KH = DC == 256 ? 2 : 1, RT = TM / N_NORM;
        int it = 0;                                                        // operand stages so far: KH per tile
        float a[RT], b[RT];
        for (int64_t tile = tile0; tile < p.n_tiles; tile += (KH == 1 || (it & 1)) ? tile_step : 0, ++it) {
            const int s = it % a_stages;
            if (!mbar_wait(bar_full + 8 * s, uint32_t(it / a_stages) & 1u, abort_flag, 7)) break;
            const unsigned char* rowp = smem + OFF_A + s * OPER_BYTES + r * 128;
            if (KH == 1 || !(it & 1)) {
#pragma unroll
                for (int h = 0; h < RT; ++h) a[h] = b[h] = 0.f;
            }
            const auto sum = [&](auto type) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
#pragma unroll
                    for (int h = 0; h < RT; ++h) {
                        const uint4 v = *reinterpret_cast<const uint4*>(rowp + h * 64 * 128 + ((c ^ (r & 7)) << 4));
                        const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) add_squares<decltype(type)::value>(a[h], vw[u]);
                        if (d > 64 + 8 * c) {
                            const uint4 w = *reinterpret_cast<const uint4*>(rowp + KBLK_BYTES + h * 64 * 128 + ((c ^ (r & 7)) << 4));
                            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int u = 0; u < 4; ++u) add_squares<decltype(type)::value>(b[h], ww[u]);
                        }
                    }
                }
            };
            if (bf16) sum(std::true_type{});
            else sum(std::false_type{});
            if constexpr (DC == 256) {
                if (it & 1) {
                    const int q = (it >> 1) % NSQ_SLOTS;
#pragma unroll
                    for (int h = 0; h < RT; ++h) reinterpret_cast<float*>(smem + OFF_NSQ256)[q * TM + r + 64 * h] = a[h] + b[h];
                    mbar_arrive(sbase + OFF_NRMBAR256 + 8 * q);
                }
            } else {
            float* nsq = reinterpret_cast<float*>(smem + OFF_NSQ) + s * 2 * TM;
#pragma unroll
            for (int h = 0; h < RT; ++h) { nsq[r + 64 * h] = a[h]; nsq[TM + r + 64 * h] = b[h]; }
            mbar_arrive(bar_nrm + 8 * s);        // release: the epilogue reads the sums after waiting on this barrier
            }
            mbar_arrive(bar_afree + 8 * s);      // this thread is done reading the stage
        }
    }
    // ---- teardown: every loop above is bounded, so every thread gets here ----
    tc_fence_before();
    __syncthreads();
    if (warp == EPI_WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace tc

}  // namespace tq

using namespace tq;

namespace tq {
static int quantize_sms() {
    static std::atomic<int> sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int n = sms[dev].load();
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        sms[dev].store(n);
    }
    return n;
}
}

// The jobs of one compression side by side: tiles per CTA with which all of them fit the SMs at once, or 0 where that would be above 8.
// A CTA pays 6 us of set-up (R as operand tiles) before its first tile and 1 to 1.5 us per tile: with a CTA per tile, up to the SMs, each
// job's set-up waited for the one before it.  us for keys and values of 8 lanes, one after the other / side by side:
//   tokens                          2048          4096          8192         16384
//   d = 128 fp16, 4 and 2 bits   15.7 / 12.4   18.6 / 16.5   24.7 / 22.6   36.3 / 36.7
//   d = 128 bf16, 4 and 2 bits   18.5 / 14.4   21.1 / 20.5   28.8 / 28.6   41.0 / 45.1
//   d = 128 fp16, 3.5 bits       17.9 / 13.6   20.6 / 16.6   26.7 / 22.6   39.0 / 34.9
//   d = 64 fp16, 4 bits          14.4 / 11.3   16.8 / 14.4   20.7 / 18.5   30.8 / 28.9
// The widths cost different times per tile: from 9 tiles on (between the last two columns) the cheaper job's CTAs end early.
int tq_quantize_tiles_each(const tq_quantize_args* q, int n) {
    int64_t total = 0, tiles[8];
    if (n > 8) return 0;
    for (int i = 0; i < n; ++i) total += tiles[i] = q[i].n_lanes * ((q[i].n_rows + tc::TM - 1) / tc::TM);
    const int64_t room = q[0].d == 256 ? quantize_sms() / 4 : quantize_sms();
    for (int64_t each = std::max<int64_t>(1, (total + room - 1) / room); each <= 8; ++each) {
        int64_t ctas = 0;
        for (int i = 0; i < n; ++i) ctas += (tiles[i] + each - 1) / each;
        if (ctas <= room) return int(each);
    }
    return 0;
}

// Takes the call when it fits the tensor-core kernel: fp16 / bf16 rows, d in {64, 96, 128} or 256 without a sketch, 16-byte aligned rows, no
// rotated-row output, a bit-width pair the epilogue is compiled for.  Otherwise reports "not handled" and the caller uses
// the general CUDA-core kernel.
int tq_quantize_pack_tc(const tq_quantize_args* q, cudaStream_t s, bool* handled, bool follows, int tiles_each) {
    *handled = false;
    const int d = q->d;
    if ((d != 64 && d != 96 && d != 128 && (d != 256 || q->qjl_bits)) || (q->x_dtype != TQ_F16 && q->x_dtype != TQ_BF16) || q->y_out) return TQ_OK;
    const bool frac = q->bits_lo != 0;
    if (frac && (q->bits_hi != q->bits_lo + 1)) return TQ_OK;                  // the reference's fractional widths only
    if (!aligned(q->x, 16) || q->x_row_stride % 8 || q->x_lane_stride % 8 || !aligned(q->rot, 16)) return TQ_OK;
    if ((q->n_rows > 1 && q->x_row_stride <= 0) || (q->n_lanes > 1 && q->x_lane_stride <= 0)) return TQ_OK;     // the same rows again and again: no tensor map
    if (q->n_rows >= (int64_t(1) << 31) || q->n_lanes >= (int64_t(1) << 31)) return TQ_OK;
    static int disabled = -1;
    if (disabled < 0) {
        const char* e = getenv("TQ_DISABLE_TC");
        disabled = (e && e[0] == '1') ? 1 : 0;
    }
    if (disabled) return TQ_OK;
    // (one row takes 8 us here and 38 in the row kernel at d = 128, 8 and 116 at d = 256: no size is too small)
    const bool qjl = q->qjl_bits != nullptr;
    static bool attr_set[16] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16) return TQ_OK;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(tc::quantize_tc_kernel<false, true, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tc::quantize_tc_kernel<false, true, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tc::quantize_tc_kernel<false, true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tc::quantize_tc_kernel<false, false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tc::quantize_tc_kernel<true, false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES);
        if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_quantize_pack: shared memory %d B: %s", tc::SMEM_BYTES, cudaGetErrorString(e));
        attr_set[dev] = true;
    }
    static PFN_cuTensorMapEncodeTiled encode = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
        looked_up = true;
    }
    if (!encode) return TQ_OK;
    // Tensor map over the rows as (column, row, lane): boxes of 64 columns x 128 rows x 1 lane land in shared memory in
    // the 128-byte-swizzled layout the MMA descriptors describe; rows past a lane's end and columns past d read as zeros.
    CUtensorMap tmap{};
    const cuuint64_t dims[3] = {cuuint64_t(d), cuuint64_t(q->n_rows), cuuint64_t(q->n_lanes)};
    // bytes, multiples of 16 (a single row or lane: any stride will do)
    const int64_t row_stride = q->n_rows > 1 ? q->x_row_stride : d, lane_stride = q->n_lanes > 1 ? q->x_lane_stride : row_stride * q->n_rows;
    const cuuint64_t strides[2] = {cuuint64_t(row_stride) * 2, cuuint64_t(lane_stride) * 2};
    const cuuint32_t box[3] = {64, cuuint32_t(tc::TM), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(&tmap, q->x_dtype == TQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(q->x),
                              dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return TQ_OK;

    tc::Params p{};
    p.follows = follows ? 1 : 0;
    p.d = d; p.bf16 = q->x_dtype == TQ_BF16 ? 1 : 0; p.a_stages = p.bf16 ? 2 : 3;
    p.n_rows = q->n_rows;
    p.tiles_per_lane = (q->n_rows + tc::TM - 1) / tc::TM;
    p.n_tiles = q->n_lanes * p.tiles_per_lane;
    if (p.n_tiles >= (int64_t(1) << 31)) return TQ_OK;
    p.rot = q->rot; p.bnd_hi = q->bnd_hi; p.bnd_lo = q->bnd_lo; p.bits_hi = q->bits_hi; p.bits_lo = q->bits_lo;
    p.p_hi = q->packed_hi; p.p_lo = q->packed_lo; p.norms = q->norms; p.out_lane_stride = q->out_lane_stride;
    p.qjl_proj_rot = q->qjl_proj_rot; p.cent_hi = q->cent_hi; p.cent_lo = q->cent_lo; p.qjl_bits = q->qjl_bits; p.qjl_gamma = q->qjl_gamma;
    const int64_t room = d == 256 ? quantize_sms() / 4 : quantize_sms(), ctas = std::min(room, tiles_each > 0 ? (p.n_tiles + tiles_each - 1) / tiles_each : p.n_tiles);
    const unsigned grid = unsigned(d == 256 ? 4 * ctas : ctas);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(unsigned(tc::n_threads(d == 256 || (!qjl && !p.bf16))));
    cfg.dynamicSmemBytes = tc::SMEM_BYTES;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = follows ? 1 : 0;
    if (d == 256) cudaLaunchKernelEx(&cfg, tc::quantize_tc_kernel<false, true, 256>, p, tmap);
    else if (qjl) cudaLaunchKernelEx(&cfg, tc::quantize_tc_kernel<true, false, 0>, p, tmap);
    else if (p.bf16) cudaLaunchKernelEx(&cfg, tc::quantize_tc_kernel<false, false, 0>, p, tmap);
    else if (d == 128) cudaLaunchKernelEx(&cfg, tc::quantize_tc_kernel<false, true, 128>, p, tmap);
    else cudaLaunchKernelEx(&cfg, tc::quantize_tc_kernel<false, true, 0>, p, tmap);
    *handled = true;
    return check_launch("tq_quantize_pack (tensor core)");
}

namespace tq { int decode_status_host(); int decode_status_clear(); }   // decode_direct.cu

// 0 if no kernel on the current device has reported a timed-out wait, else the code of the first one.
// Synchronises the device.
extern "C" int tq_device_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, tc::g_status, sizeof(int)) != cudaSuccess) return -1;
    return v ? v : decode_status_host();
}

extern "C" int tq_device_status_clear(void) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(tc::g_status, &zero, sizeof(int)) != cudaSuccess) return -1;
    return decode_status_clear();
}
