// Causal attention for several query tokens per sequence over the compressed cache, in two steps: the cache's tokens are
// expanded ONCE per call into fp16 rows in workspace memory, then a flash-attention kernel on the fifth-generation tensor
// cores reads those rows through TMA for every block of queries.
// Same contract and arithmetic as prefill_tc.cu / prefill.cu (what the reference does as dense reassembly, cache.py:674-706,
// followed by the consumer's masked attention).
//
// Why a pre-pass: with the unpacking inside the attention kernel every block of 128 query rows turned the same codes into
// the same operands again, and the table lookups shared the shared-memory pipe with the softmax (3 us per 128 x 128 tile
// against 0.77 us of tensor-core time; 15 us at widths without whole-byte tables).  A row costs 2 d bytes of writes once and
// is then read from L2 by every block.
//
// An expanded packed row is the token's CENTROIDS in fp16 (the values' under their table's scale): rotated space, not c @ R.
// Rotated-back rows would have to be rounded to fp16 once more; results were then 1.4 times as far from 64-bit attention as the
// other kernels' (2.1e-4 against 3.0e-4 relative at d = 64, 128, 256; now 2.1e-4).  So the packed tokens are met by the rotated
// queries, their weighted sum is rotated back once, in float32 accuracy, and the uncompressed tokens (rows as they are, float32 /
// bfloat16 ones under a power-of-two scale) follow with the queries as they are.  Norms stay float32 beside the rows, so no
// magnitude is lost: scores take the key norm as a multiply-add, the softmax weights take the value norm before they become fp16.
//
//   fa_query_kernel    queries times scale * log2(e) as fp16, raw and rotated; R as operand tiles.  28 us for 65,536 rows at d = 128,
//                      beside the expansion
//   fa_expand_kernel   the rows and norms.  32 lanes x 16,384 tokens at d = 128, 4 / 2 bits: 81 us, bound by writing 268 MB
//                      (118 us as unit rows c @ R through the dequantize kernel)
//   fa_kernel          below
//   fa_merge_kernel    when there are too few query blocks for the device, the key tiles of a block are split over several CTAs,
//                      which leave float32 partials
//
// fa_kernel: a CTA owns NQ (2; 1 at d = 256) tiles of 128 rows = 128 / GP query tokens x the GP query heads of a GQA group, and a
// range of key tiles (TN tokens each), packed tokens first:
//   * 8 NQ softmax warps, two rows' shares per thread: tcgen05.ld of the scores as mma.sync fragments, one multiply-add each (packed in
//     pairs), ex2, P (fp16) back into tensor memory over the scores it came from; a row's reference maximum is looked at through its sum;
//   * one warp issues S = Q K^T (both operands in shared memory) and O += P V (P from tensor memory), the tiles of the two
//     query blocks alternating so that one block's softmax runs under the other's products;
//   * one thread each keeps four key tiles (and eight tiles' norms) and four value tiles in flight (tiled TMA, bulk copies); scores
//     are two key tiles ahead of the softmax;
//   * between the two regions the softmax warps leave O as high and low fp16 parts where the scores were, the MMA warp multiplies
//     them with R's parts in place (three products, the small ones first) and the raw queries replace the rotated ones.
//   512 queries x 32 lanes over 16,384 tokens at d = 128: 580 us = 930 TFLOP/s (350 with the unpacking inside the kernel).
//
// Every mbarrier wait is bounded; a wait that runs out leaves status 111 (tq_device_status) and raises a flag that ends
// every other wait; copies and products in flight are waited for (bounded), tensor memory is freed on every path.
#include <algorithm>
#include <atomic>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "decode_dev.cuh"
#include "dequantize_tc.cuh"

namespace tq {

int* decode_status_ptr();

namespace fa {

constexpr uint32_t WAIT_LIMIT = 4u << 20;
constexpr int ERR_WAIT = 111;
constexpr int TM = 128, NSC = 8;                       // rows per query tile, tiles' norms in flight
constexpr int MAX_RANGES = 16;                         // key ranges of a row block

template <int D> struct Plan {
    static constexpr int NQ = D == 256 ? 1 : 2;        // query tiles per CTA
    static constexpr int TN = 64;                      // tokens per key tile
    static constexpr int SB = 2;                       // score buffers per query tile
    static constexpr int ST = D == 256 ? 2 : 4;        // key tiles (and value tiles) in flight
    static constexpr int NBLK = (D + 63) / 64;         // 64-column blocks of a row
    static constexpr int DP = NBLK * 64;               // columns of O (d = 96: the last 32 are zeros)
    static constexpr int SW = NQ * 8, NT = SW * 32 + 96;      // softmax warps; MMA warp, a TMA warp for keys and norms, one for values
    static constexpr uint32_t QBLK = TM * 128u, KBLK = TN * 128u;            // bytes of a 64-column block
    static constexpr uint32_t Q_TILE = NBLK * QBLK, K_TILE = NBLK * KBLK;
    static constexpr uint32_t OFF_Q = 0, OFF_K = NQ * Q_TILE, OFF_V = OFF_K + ST * K_TILE;
    static constexpr uint32_t OFF_SC = OFF_V + ST * K_TILE;                  // float [NSC][2][TN]: key norms, value norms
    static constexpr uint32_t OFF_R = D == 64 ? OFF_SC + NSC * 2 * TN * 4 : OFF_K;      // R (see below): through the key ring where it has no room of its own
    static constexpr uint32_t OFF_BAR = OFF_SC + NSC * 2 * TN * 4 + (D == 64 ? 2 * 64 * 128 : 0);
    static constexpr uint32_t OFF_SLOT = OFF_BAR + 464;                      // [0] tensor-memory base, [1] abort
    static constexpr size_t NEED = OFF_SLOT + 16 + 1024, SMEM = NEED > 116 * 1024 ? NEED : 116 * 1024;      // one CTA per SM: it takes all of the tensor memory
    static constexpr uint32_t COL_O = NQ * SB * TN;                          // scores first, then the accumulators
    // rotation of the packed tokens' sums: they sit in tensor memory as A operands (high parts and low parts, two per column) where
    // scores were (d = 256: the low parts behind the accumulator), R as RC columns at a time, high, then low parts, passes taking turns
    // in the key ring and the value ring
    static constexpr int RC = D == 256 ? 64 : DP, PASSES = DP / RC;
    static constexpr uint32_t COL_A = SB * TN, COL_LO = D == 256 ? COL_O + DP : DP / 2;      // columns per query tile; low parts from the high ones
    static constexpr uint32_t RBLK = D * 128u, R_HALF = RC / 64 * RBLK;                      // a block of 64 columns of R; bytes of a pass's high parts
    static_assert(COL_O + NQ * DP <= 512 && (D == 256 ? COL_LO + DP / 2 <= 512 : DP <= COL_A), "tensor memory");
    static constexpr bool R_RING = OFF_R == OFF_K;
    static_assert((R_RING ? 2 * R_HALF <= ST * K_TILE && (PASSES == 1 || PASSES % 2 == 0) : 2 * R_HALF == 2 * 64 * 128 && PASSES == 1) && RBLK % 1024 == 0 && OFF_R % 1024 == 0, "R's place");
    static_assert(SMEM <= 227 * 1024, "shared memory");
};
enum Bars { K_FULL = 0, K_FREE = 4, V_FULL = 8, V_FREE = 12, SC_FULL = 16, SC_FREE = 24, S_FULL = 32, P_FULL = 36, O_DONE = 40, ALL_DONE = 42, DRAIN = 44, ROT_IN = 45, ROT_A = 47, ROT_OUT = 49, R_FULL = 51, R_DONE = 53, Q_FULL = 55 };       // (57 of 8 bytes)

struct Params {
    void* out; int out_dtype;
    int Hq, Hkv, G, HG, GP, QT, Tq;                    // QT: query tokens per query tile
    int lane0, n_lanes;                                // cache lanes of this launch
    int q_pos0, sink_len, c_len, n_dense, c64;         // position of query token 0; tokens of the regions, c_len rounded up to 64
    const float *kn, *vn; int ts;                      // norms (lane, ts), ts a multiple of 128
    int n_blk, n_splits;                               // row blocks, key ranges
    float* part;                                       // (lane x head group, row block, range, NQ * 128 rows, D + 4)
    const unsigned char* r_img;                        // R as B operands: per pass high parts, low parts
    float v_inv_hi, v_inv_lo;                          // one over the value tables' scales
    int* status;
};

// ---- PTX wrappers -----------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// The tensor core's instructions take their operands from uniform registers.  A whole warp in uniform control flow computes
// them there and one elected lane issues; with a single thread in a divergent branch every operand is moved over one by one (the
// issuing thread, not the products, was what the softmax warps waited for; quantize of bfloat16 rows went from 154 to 121 us).
// D = A.B (+ D when accumulate != 0), both operands through shared-memory descriptors
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with A in tensor memory (two fp16 per 32-bit column)
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// D = A.B + 2^-11 D
__device__ __forceinline__ void umma_ts_scaled11(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 11;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(1u) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// Sixteen rows as mma.sync accumulator fragments: of eight columns, lane 4 g + t holds columns 2 t, + 1 of row g (r[0], r[1]) and of row g + 8
// (r[2], r[3]).  64 columns; 32 of them; and, stored, 64 fp16 values: columns 2 t, + 1 of each row packed into r[0], r[1].
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_frag32(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_half64(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// two float32 at once
using u64 = unsigned long long;
__device__ __forceinline__ u64 pk(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(u64 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// two values as fp16 high parts and 2^11 times what those leave
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& l) {
    const __half2 hh = __floats2half2_rn(a, b);
    const float2 hf = __half22float2(hh);
    h = *reinterpret_cast<const uint32_t*>(&hh);
    l = pack_h2((a - hf.x) * 2048.f, (b - hf.y) * 2048.f);
}
// Shared-memory descriptors of tiles made of 64-column blocks `blk` bytes apart, rows of 128 B, 128-byte swizzle.
// K-major (rows = M or N index): the 16-column slab ks; MN-major (rows = K index): the 16-row slab ks.
__device__ __forceinline__ uint64_t desc_k(uint32_t tile, uint32_t blk, int ks) {
    const uint32_t addr = tile + uint32_t(ks >> 2) * blk + uint32_t(ks & 3) * 32u;
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t tile, uint32_t blk, int ks) {
    const uint32_t addr = tile + uint32_t(ks) * 2048u;
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(blk >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// kind::f16: fp32 accumulate, fp16 operands, A K-major, M = 128
__host__ __device__ constexpr uint32_t idesc_of(int n, bool b_mn) { return (1u << 4) | (b_mn ? 1u << 16 : 0u) | (uint32_t(n >> 3) << 17) | (uint32_t(TM >> 4) << 24); }

template <int D>
__global__ void __launch_bounds__(Plan<D>::NT, 1) fa_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                                                         const __grid_constant__ CUtensorMap qmap_rot, const __grid_constant__ CUtensorMap qmap_raw) {
    using P = Plan<D>;
    constexpr int NQ = P::NQ, TN = P::TN, DP = P::DP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t raw_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    const uint32_t sbase = (raw_addr + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (sbase - raw_addr);
    volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(smem + P::OFF_SLOT);
    auto bar = [&](int which) -> uint32_t { return sbase + P::OFF_BAR + 8u * uint32_t(which); };
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // (uniform)

    // CTA = (lane x head group, row block, key range); the latest query rows (the longest runs of tiles) first
    const int y = blockIdx.x / (p.n_blk * p.n_splits), x_of = blockIdx.x - y * p.n_blk * p.n_splits;
    const int blk = p.n_blk - 1 - x_of / p.n_splits, split = x_of % p.n_splits;
    const int lane_c = y / p.HG, hg = y - lane_c * p.HG, gl = p.lane0 + lane_c;
    const int b = gl / p.Hkv, hkv = gl - b * p.Hkv;
    const int heads_here = min(HPG, p.G - hg * HPG);
    const int tq0 = blk * NQ * p.QT, gp_bits = 31 - __clz(p.GP);       // (GP is a power of two: no divisions, of cold code, behind the loop)
    auto row_head = [&](int m) { return m & (p.GP - 1); };
    auto row_token = [&](int m) { return tq0 + (m >> 7) * p.QT + ((m & 127) >> gp_bits); };
    auto row_valid = [&](int m) { return row_head(m) < heads_here && row_token(m) < p.Tq; };
    auto row_q_index = [&](int m) -> int64_t {
        const int h = hkv * p.G + hg * HPG + row_head(m);
        return ((int64_t(b) * p.Hq + h) * p.Tq + row_token(m)) * D;
    };
    // the last packed token, and the last of the others (sink and recent tokens one after the other), that position `pos` sees, or less than 0
    auto limit_p = [&](int pos) { return min(pos - p.sink_len, p.c_len - 1); };
    auto limit_d = [&](int pos) { return pos < p.sink_len ? pos : max(p.sink_len - 1, pos - p.c_len); };
    // key tiles of this CTA: its share of those that some row of it sees, packed ones first
    const int last_pos = p.q_pos0 + min(tq0 + NQ * p.QT, p.Tq) - 1;
    const int all_p = (max(limit_p(last_pos) + 1, 0) + TN - 1) / TN, n_all = all_p + (max(limit_d(last_pos) + 1, 0) + TN - 1) / TN;
    const int per = (n_all + p.n_splits - 1) / p.n_splits, t_lo = split * per, n = max(0, min(t_lo + per, n_all) - t_lo);
    const int n_p = min(max(all_p - t_lo, 0), n);              // packed ones among them
    auto tile_row = [&](int j) { return j < n_p ? (t_lo + j) * TN : p.c64 + (t_lo + j - all_p) * TN; };      // first row of key tile j in the expanded arrays

    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(bar(K_FULL + i), 1); mbar_init(bar(K_FREE + i), 1); mbar_init(bar(V_FULL + i), 1); mbar_init(bar(V_FREE + i), 1);
            mbar_init(bar(S_FULL + i), 1); mbar_init(bar(P_FULL + i), 256);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(bar(O_DONE + i), 1); mbar_init(bar(ALL_DONE + i), 1); }
        mbar_init(bar(DRAIN), 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(ROT_IN + i), 1); mbar_init(bar(ROT_A + i), 256); mbar_init(bar(ROT_OUT + i), 1); mbar_init(bar(Q_FULL + i), 1);
            mbar_init(bar(R_FULL + i), 1); mbar_init(bar(R_DONE + i), 1);
        }
        for (int i = 0; i < NSC; ++i) { mbar_init(bar(SC_FULL + i), 1); mbar_init(bar(SC_FREE + i), NQ * 256); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        slot[1] = 0u;
    }
    if (warp == P::SW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + P::OFF_SLOT), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    const uint32_t tmem = __shfl_sync(0xffffffffu, slot[0], 0);

    auto wait_bar = [&](int which, int phase) -> bool {
        const uint32_t addr = bar(which);
        for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
            if (mbar_try(addr, uint32_t(phase & 1))) return true;
            if ((i & 1023u) == 1023u && slot[1]) return false;
        }
        slot[1] = 1u;
        atomicCAS(p.status, 0, ERR_WAIT);
        return false;
    };
    // copies and products end (bounded) before their memory is given up, also after a wait that ran out
    auto drain = [&](int which, int phase) {
        for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try(bar(which), uint32_t(phase & 1)); ++i) {}
    };
    // score buffer of (query tile q, key tile j) and the phase of its barriers
    constexpr int SB = P::SB, ST = P::ST;
    auto sbuf = [](int q, int j) { return q * SB + j % SB; };
    auto sph = [](int j) { return j / SB; };
    auto first_row = [&]() { return (warp >> 3) * TM + (warp & 3) * 32 + (warp & 4) * 4 + (lane >> 2); };      // a softmax thread has this row and the eighth one after it

    if (warp == P::SW + 1) {
        // ======================= keys and norms: one thread (a key tile is free as soon as its scores are computed, long before =====
        // ======================= the value tile: each of the two rings is kept full by a thread of its own) =======================
        if (lane == 0) {
            const float* kn = p.kn + int64_t(lane_c) * p.ts;
            const float* vn = p.vn + int64_t(lane_c) * p.ts;
            int nk = 0, nsc = 0, nr = 0, nq = 0;                   // copies asked for so far
            // the query tiles as A operands, rotated for the packed tokens, as they are for the others: rows (token, head of the group)
            auto load_q = [&](const CUtensorMap* map) {
                for (int q = 0; q < NQ; ++q) {
                    mbar_expect_tx(bar(Q_FULL + q), P::Q_TILE);
                    for (int x = 0; x < P::NBLK; ++x)
                        tma_load_3d(sbase + P::OFF_Q + q * P::Q_TILE + x * P::QBLK, map, x * 64, lane_c * p.G + hg * HPG, tq0 + q * p.QT, bar(Q_FULL + q));
                }
                ++nq;
            };
            auto load_r = [&](int x) {                             // (even passes)
                mbar_expect_tx(bar(R_FULL), 2 * P::R_HALF);
                bulk_g2s(sbase + P::OFF_R, p.r_img + x * 2 * P::R_HALF, 2 * P::R_HALF, bar(R_FULL));
                ++nr;
            };
            // between the packed tiles and the others, as soon as the scores that used them are computed: R through the key ring, the other queries
            auto turn = [&]() -> bool {
                for (int j = max(0, n_p - ST); j < n_p; ++j)
                    if (!wait_bar(K_FREE + j % ST, j / ST)) return false;
                if (P::R_RING) load_r(0);
                if (n > n_p) load_q(&qmap_raw);
                for (int x = 2; x < P::PASSES; x += 2) {
                    if (!wait_bar(R_DONE, x / 2 - 1)) return false;
                    load_r(x);
                }
                return !P::R_RING || wait_bar(R_DONE, (P::PASSES - 1) / 2);
            };
            if (n > 0) load_q(n_p > 0 ? &qmap_rot : &qmap_raw);
            if (!P::R_RING && n_p > 0) load_r(0);
            for (int j = 0; j < n; ++j) {
                const int row = tile_row(j), s = j % NSC, st = j % ST;
                if (j == n_p && n_p > 0 && !turn()) break;
                if (j >= ST && !wait_bar(K_FREE + st, j / ST - 1)) break;
                nk = j + 1;
                mbar_expect_tx(bar(K_FULL + st), P::K_TILE);
                for (int x = 0; x < P::NBLK; ++x) tma_load_3d(sbase + P::OFF_K + st * P::K_TILE + x * P::KBLK, &kmap, x * 64, row, lane_c, bar(K_FULL + st));
                if (j >= NSC && !wait_bar(SC_FREE + s, j / NSC - 1)) break;
                const uint32_t sc = sbase + P::OFF_SC + s * 2 * TN * 4;
                nsc = j + 1;
                mbar_expect_tx(bar(SC_FULL + s), 2 * TN * 4);
                bulk_g2s(sc, kn + row, TN * 4, bar(SC_FULL + s));
                bulk_g2s(sc + TN * 4, vn + row, TN * 4, bar(SC_FULL + s));
            }
            if (n_p == n && n > 0 && nsc == n) turn();
            if (nr > 0) drain(R_FULL, nr - 1);
            for (int q = 0; q < NQ && nq > 0; ++q) drain(Q_FULL + q, nq - 1);
            for (int j = max(0, nk - ST); j < nk; ++j) drain(K_FULL + j % ST, j / ST);
            for (int j = max(0, nsc - NSC); j < nsc; ++j) drain(SC_FULL + j % NSC, j / NSC);
        }
        __syncwarp();
    } else if (warp == P::SW + 2) {
        // ======================= values: one thread =======================
        if (lane == 0) {
            int nv = 0, nr = 0;
            auto turn = [&]() -> bool {                            // odd passes of R through the value ring
                for (int j = max(0, n_p - ST); j < n_p; ++j)
                    if (!wait_bar(V_FREE + j % ST, j / ST)) return false;
                for (int x = 1; x < P::PASSES; x += 2) {
                    if (x > 1 && !wait_bar(R_DONE + 1, x / 2 - 1)) return false;
                    mbar_expect_tx(bar(R_FULL + 1), 2 * P::R_HALF);
                    bulk_g2s(sbase + P::OFF_V, p.r_img + x * 2 * P::R_HALF, 2 * P::R_HALF, bar(R_FULL + 1));
                    ++nr;
                }
                return wait_bar(R_DONE + 1, P::PASSES / 2 - 1);
            };
            for (int j = 0; j < n; ++j) {
                const int row = tile_row(j), st = j % ST;
                if (P::PASSES > 1 && j == n_p && n_p > 0 && !turn()) break;
                if (j >= ST && !wait_bar(V_FREE + st, j / ST - 1)) break;
                nv = j + 1;
                mbar_expect_tx(bar(V_FULL + st), P::K_TILE);
                for (int x = 0; x < P::NBLK; ++x) tma_load_3d(sbase + P::OFF_V + st * P::K_TILE + x * P::KBLK, &vmap, x * 64, row, lane_c, bar(V_FULL + st));
            }
            if (P::PASSES > 1 && n_p == n && n > 0 && nv == n) turn();
            if (nr > 0) drain(R_FULL + 1, nr - 1);
            for (int j = max(0, nv - ST); j < nv; ++j) drain(V_FULL + j % ST, j / ST);
        }
        __syncwarp();
    } else if (warp == P::SW) {
        // ======================= MMA issue: one warp, uniform =======================
        if (n > 0) {
            auto issue_qk = [&](int q, int j) {                    // S = Q K^T of key tile j
                const uint32_t s = tmem + sbuf(q, j) * TN;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ss(s, desc_k(sbase + P::OFF_Q + q * P::Q_TILE, P::QBLK, ks), desc_k(sbase + P::OFF_K + (j % ST) * P::K_TILE, P::KBLK, ks),
                            idesc_of(TN, false), ks > 0 ? 1u : 0u);
                umma_commit(bar(S_FULL + sbuf(q, j)));
            };
            auto issue_pv = [&](int q, int j) {                    // O += P V
                const uint32_t a = tmem + sbuf(q, j) * TN;
#pragma unroll
                for (int ks = 0; ks < TN / 16; ++ks)
                    umma_ts(tmem + P::COL_O + q * DP, a + ks * 8, desc_mn(sbase + P::OFF_V + (j % ST) * P::K_TILE, P::KBLK, ks), idesc_of(DP, true),
                            (j > 0 || ks > 0) ? 1u : 0u);
                umma_commit(bar(O_DONE + q));
                if (j == n_p - 1) umma_commit(bar(ROT_IN + q));
                if (j == n - 1) umma_commit(bar(ALL_DONE + q));    // (a barrier of its own: a parity wait on O_DONE could be two phases early or one late)
            };
            auto wait_all = [&](int which, int phase) -> bool { return __all_sync(0xffffffffu, wait_bar(which, phase)); };
            bool ok = true;
            // key tiles [j0, j1): scores SB tiles ahead of the products
            auto tiles = [&](int j0, int j1, int q_phase) {
                for (int q = 0; q < NQ && ok && j0 < j1; ++q) ok = wait_all(Q_FULL + q, q_phase);
                for (int j = j0; j < min(j1, j0 + SB) && ok; ++j) {
                    ok = wait_all(K_FULL + j % ST, j / ST);
                    if (!ok) break;
                    tc_fence_after();
                    for (int q = 0; q < NQ; ++q) issue_qk(q, j);
                    umma_commit(bar(K_FREE + j % ST));
                }
                for (int j = j0; j < j1 && ok; ++j) {
                    ok = wait_all(V_FULL + j % ST, j / ST);
                    const int jn = j + SB;                         // the key tile whose scores go where P of tile j sits now
                    for (int q = 0; q < NQ && ok; ++q) {
                        ok = wait_all(P_FULL + sbuf(q, j), sph(j));
                        if (!ok) break;
                        tc_fence_after();
                        issue_pv(q, j);
                        if (q == NQ - 1) umma_commit(bar(V_FREE + j % ST));
                        if (jn < j1) {                             // (the tensor core takes one thread's products in order)
                            if (q == 0) ok = wait_all(K_FULL + jn % ST, jn / ST);
                            if (!ok) break;
                            issue_qk(q, jn);
                            if (q == NQ - 1) umma_commit(bar(K_FREE + jn % ST));
                        }
                    }
                }
            };
#pragma unroll 1
            for (int region = 0; region < 2 && ok; ++region) {     // (one copy of the loop)
                tiles(region ? n_p : 0, region ? n : n_p, region && n_p > 0 ? 1 : 0);
                if (region || n_p == 0 || !ok) continue;
                // the packed tokens' sums times R, in place: 2^11 (high . low + low . high) first, then that times 2^-11 plus high . high
                for (int x = 0; x < P::PASSES && ok; ++x) {
                    ok = wait_all(R_FULL + (x & 1), x >> 1);
                    for (int q = 0; q < NQ && ok; ++q) {
                        if (x == 0) ok = wait_all(ROT_A + q, 0);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t o = tmem + P::COL_O + q * DP + x * P::RC, hi = tmem + q * P::COL_A, lo = hi + P::COL_LO;
                        const uint32_t r_hi = sbase + (x & 1 ? P::OFF_V : P::OFF_R), r_lo = r_hi + P::R_HALF;
                        constexpr uint32_t id = idesc_of(P::RC, true);
                        for (int ks = 0; ks < D / 16; ++ks) umma_ts(o, hi + ks * 8, desc_mn(r_lo, P::RBLK, ks), id, ks > 0 ? 1u : 0u);
                        for (int ks = 0; ks < D / 16; ++ks) umma_ts(o, lo + ks * 8, desc_mn(r_hi, P::RBLK, ks), id, 1u);
                        umma_ts_scaled11(o, hi, desc_mn(r_hi, P::RBLK, 0), id);
                        for (int ks = 1; ks < D / 16; ++ks) umma_ts(o, hi + ks * 8, desc_mn(r_hi, P::RBLK, ks), id, 1u);
                        if (x == P::PASSES - 1) umma_commit(bar(ROT_OUT + q));
                    }
                    if (ok) umma_commit(bar(R_DONE + (x & 1)));
                }
            }
            if (!ok) { umma_commit(bar(DRAIN)); drain(DRAIN, 0); }
        }
        __syncwarp();
    } else if (__any_sync(0xffffffffu, row_valid(first_row()) || row_valid(first_row() + 8))) {
        // ======================= softmax: two rows per thread, sixteen columns of each =======================
        // Scores are read as mma.sync fragments: lane 4 g + t of a warp holds columns 8 r + 2 t, + 1 of rows g and g + 8 of its sixteen, so that it
        // needs the norms of 16 tokens a side, not of all 64.  Two warps share the 32 lanes of a quarter of tensor memory: four per scheduler
        // hide one another's latencies.  (A row per thread in half as many warps read every norm in every thread: 760 shared-memory wavefronts
        // per key tile beside 1035 of operands and 256 of copies; with those the shared-memory pipe was 90 % busy: 667 -> 610 us for 512 queries x 32
        // lanes over 16,384 tokens at d = 128, of 1280 cycles of products per key tile and 1700 in all.  Scores of two key tiles in one product of
        // 128 columns, 1024 cycles, take a query tile's two score buffers at once: 660 us.)  A warp owns its sixteen rows from the scores to the
        // result: the accumulator is read, split for the product with R and written out as fragments too.  (With a row per thread there, two
        // warps shared every row, looked at all of its columns each for the scale and told one another its sum: 3200 cycles of a call's 33,500.)
        //   us per call of 8 heads, 4 / 2 bits, d = 128: 8 queries over 500 tokens 26.2 -> 21.7 (with the warps without a row, below), 64 over 500,
        //   four sequences, 36.4 -> 33.4; 512 over 16,384, four sequences, 775 -> 761 with their compression.
        const int q = warp >> 3, hh = (warp >> 2) & 1, g = lane >> 2, t2 = 2 * (lane & 3);       // query tile; half of the 32 lanes
        const uint32_t t_frag = tmem + (uint32_t((warp & 3) * 32 + 16 * hh) << 16);
        const int mf = first_row();
        const int pos0 = p.q_pos0 + tq0 + q * p.QT;
        int last[2];                                               // the last token of the region (packed tokens first) that each row sees
#pragma unroll
        for (int k = 0; k < 2; ++k) last[k] = row_valid(mf + 8 * k) ? limit_p(p.q_pos0 + row_token(mf + 8 * k)) : -1;
        int full_upto = limit_p(pos0);                             // tokens every row of the query tile sees
        // A row that has seen no token yet keeps m_ref = -1e30, has lvsc for a bias and asks for a reference at its first one.
        float vsc = 1.f, vthr = 0.f, lvsc = 0.f;                   // (vthr 0: the first tile with a non-zero value norm picks the scale); log2(vsc)
        float m_ref[2] = {-1e30f, -1e30f};
        u64 l2[2] = {pk(0.f, 0.f), pk(0.f, 0.f)};                  // this thread's share of the rows' sums
        auto bias_of = [&](int k) { return m_ref[k] > -1e30f ? lvsc - m_ref[k] : lvsc; };
        bool ok = true;
        for (int j = 0; j <= n; ++j) {
            if (j == n_p) {
                if (n_p > 0) {
                    // ---- behind the last packed tile: the rows' sums as high and low fp16 parts (under a power-of-two scale) for the
                    // ---- product with R; then the scale is taken back
                    ok = __all_sync(0xffffffffu, wait_bar(ROT_IN + q, 0));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t o_frag = t_frag + P::COL_O + q * DP, a_frag = t_frag + q * P::COL_A;
                    auto inv_of = [&](int c) { return c < D / 2 ? p.v_inv_hi : p.v_inv_lo; };      // (eight columns from a multiple of 8: one scale)
                    float mx[2] = {0.f, 0.f}, sc[2];
#pragma unroll 1
                    for (int c0 = 0; c0 < DP; c0 += 32) {
                        uint32_t o[16];
                        tmem_ld_frag32(o_frag + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i += 2)
                            mx[(i >> 1) & 1] = fmaxf(mx[(i >> 1) & 1], fmaxf(fabsf(__uint_as_float(o[i])), fabsf(__uint_as_float(o[i + 1]))) * inv_of(c0 + 2 * (i & 12)));
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
#pragma unroll
                        for (int off = 1; off < 4; off <<= 1) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], off));
                        sc[k] = stage_scale(__float_as_uint(mx[k]));
                    }
#pragma unroll 1
                    for (int c0 = 0; c0 < DP; c0 += 64) {
                        uint32_t o[32], hi[16], lo[16];
                        tmem_ld_frag64(o_frag + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float u = sc[(i >> 1) & 1] * inv_of(c0 + 2 * (i & 28));
                            split2(__uint_as_float(o[i]) * u, __uint_as_float(o[i + 1]) * u, hi[i / 2], lo[i / 2]);
                        }
                        tmem_st_half64(a_frag + c0 / 2, hi);
                        tmem_st_half64(a_frag + P::COL_LO + c0 / 2, lo);
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    mbar_arrive(bar(ROT_A + q));
                    ok = __all_sync(0xffffffffu, wait_bar(ROT_OUT + q, 0));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < 2; ++k) sc[k] = __int_as_float(0x7f000000 - __float_as_int(sc[k]));      // 1 / sc, a power of two in [2^-118, 2^118]
#pragma unroll 1
                    for (int c0 = 0; c0 < DP; c0 += 32) {
                        uint32_t o[16];
                        tmem_ld_frag32(o_frag + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * sc[(i >> 1) & 1]);
                        tmem_st_frag32(o_frag + c0, o);
                    }
                    tmem_st_wait();
                }
                if (j == n) break;
#pragma unroll
                for (int k = 0; k < 2; ++k) last[k] = row_valid(mf + 8 * k) ? limit_d(p.q_pos0 + row_token(mf + 8 * k)) : -1;
                full_upto = limit_d(pos0);
            }
            if (j == n) break;
            const int s = j % NSC, base = j < n_p ? (t_lo + j) * TN : (t_lo + j - all_p) * TN;
            ok = wait_bar(SC_FULL + s, j / NSC) && wait_bar(S_FULL + sbuf(q, j), sph(j));
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
            const float* kn = reinterpret_cast<const float*>(smem + P::OFF_SC) + s * 2 * TN + t2;
            const float* vn = kn + TN;
            const uint32_t s_col = t_frag + sbuf(q, j) * TN;
            constexpr int NR = TN / 8;
            uint32_t v[4 * NR];                                    // of eight columns: two of row g, two of row g + 8
            tmem_ld_frag64(s_col, v);
            u64 nv[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) nv[r] = *reinterpret_cast<const u64*>(kn + 8 * r);
            tmem_ld_wait();
            // t = score * key norm - reference + log2(value scale)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t* x = v + 2 * k;
                const float bias = bias_of(k);
                const u64 b2 = pk(bias, bias);
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    float x0, x1;
                    upk(fma2(pk(__uint_as_float(x[4 * r]), __uint_as_float(x[4 * r + 1])), nv[r], b2), x0, x1);
                    x[4 * r] = __float_as_uint(x0); x[4 * r + 1] = __float_as_uint(x1);
                }
            }
            if (base + TN > full_upto + 1) {                       // some token of the tile is hidden from some row, or past the end
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint32_t* x = v + 2 * k;
                    const int lim = last[k] - base - t2;
#pragma unroll
                    for (int r = 0; r < NR; ++r) { x[4 * r] = 8 * r <= lim ? x[4 * r] : 0xff800000u; x[4 * r + 1] = 8 * r + 1 <= lim ? x[4 * r + 1] : 0xff800000u; }
                }
            }
            // Weights, their sums, P = weight * value norm (both carry the value scale) as fp16.  A row needs another reference when a weight
            // exceeds 2^MAX_SLACK, which its sum then does too: the sums are looked at behind the exponentials and no maximum is taken in the
            // common case.  The lanes share the check of the tile's norms, eight tokens' pairs each.
            const float2 v2 = *reinterpret_cast<const float2*>(vn + 8 * g);
            float vmax = fmaxf(v2.x, v2.y);
#pragma unroll
            for (int r = 0; r < NR; ++r) nv[r] = *reinterpret_cast<const u64*>(vn + 8 * r);
            uint32_t w[2 * NR];
            u64 ls[2];
#pragma unroll 1
            for (int pass = 0;; ++pass) {
                ls[0] = ls[1] = pk(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < NR; ++r)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const u64 x = pk(ex2(__uint_as_float(v[4 * r + 2 * k])), ex2(__uint_as_float(v[4 * r + 2 * k + 1])));
                        ls[k] = add2(ls[k], x);
                        float x0, x1;
                        upk(mul2(x, nv[r]), x0, x1);
                        w[2 * r + k] = pack_h2(x0, x1);
                    }
                bool again = vmax > vthr;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    float x0, x1;
                    upk(ls[k], x0, x1);
                    again = again || x0 + x1 > (m_ref[k] > -1e30f ? float(1 << int(MAX_SLACK)) * vsc : last[k] >= base ? -1.f : INFINITY);      // (a row's first token: always)
                }
                if (pass > 0 || !__any_sync(0xffffffffu, again)) break;
                // Reference maximum / value scale: refreshed for the whole warp when any row needs it (rare after the first tile):
                // the rows' sums and their O in tensor memory are rescaled.
                float a[2], bias[2] = {bias_of(0), bias_of(1)}, mx[2] = {-INFINITY, -INFINITY}, ratio = 1.f;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
#pragma unroll
                    for (int r = 0; r < NR; ++r) mx[k] = fmaxf(fmaxf(mx[k], __uint_as_float(v[4 * r + 2 * k])), __uint_as_float(v[4 * r + 2 * k + 1]));
#pragma unroll
                    for (int off = 1; off < 4; off <<= 1) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], off));
                }
#pragma unroll
                for (int off = 16; off; off >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
                if (vmax > vthr) {
                    int eb = (__float_as_int(vmax) >> 23) & 0xff;
                    eb = min(max(eb, 16), 240);
                    const float nsc = __int_as_float((261 - eb) << 23);    // the largest value norm lands in [128, 256)
                    ratio = nsc / vsc;
                    vsc = nsc;
                    vthr = VSC_CAP / nsc;
                    lvsc = float(134 - eb);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float mn = fmaxf(fmaxf(m_ref[k], mx[k] - bias[k]), -1e30f);
                    a[k] = ex2(m_ref[k] - mn) * ratio;
                    m_ref[k] = mn;
                    const float delta = bias_of(k) - bias[k];
                    l2[k] = mul2(l2[k], pk(a[k], a[k]));
                    uint32_t* x = v + 2 * k;
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        x[4 * r] = __float_as_uint(__uint_as_float(x[4 * r]) + delta);
                        x[4 * r + 1] = __float_as_uint(__uint_as_float(x[4 * r + 1]) + delta);
                    }
                }
                if (j > 0) {
                    ok = wait_bar(O_DONE + q, j - 1);
                    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c0 = 0; c0 < DP; c0 += 32) {
                        uint32_t o[16];
                        tmem_ld_frag32(t_frag + P::COL_O + q * DP + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * a[(i >> 1) & 1]);
                        tmem_st_frag32(t_frag + P::COL_O + q * DP + c0, o);
                    }
                    tmem_st_wait();
                }
            }
            if (!ok) break;
            l2[0] = add2(l2[0], ls[0]);
            l2[1] = add2(l2[1], ls[1]);
            tmem_st_half64(s_col, w);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar(P_FULL + sbuf(q, j)));
            mbar_arrive(bar(SC_FREE + s));
        }
        // ---- the rows' results, still as fragments: 32 bytes of a row from four lanes.  (A row per thread wrote 16 of every 32 bytes at a time, and
        // the two warps of its 32 lanes had to tell one another the rows' sums.) ----
        float l_sum[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float l1;
            upk(l2[k], l_sum[k], l1);
            l_sum[k] += l1;
#pragma unroll
            for (int off = 1; off < 4; off <<= 1) l_sum[k] += __shfl_xor_sync(0xffffffffu, l_sum[k], off);
        }
        if (ok && n > n_p) ok = wait_bar(ALL_DONE + q, 0);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        const bool done = n > 0 && ok, parts = p.n_splits > 1;
        float* const part = parts ? p.part + (((int64_t(y) * p.n_blk + blk) * p.n_splits + split) * (NQ * TM) + mf) * (D + 4) : nullptr;
        if (parts && t2 == 0) {
#pragma unroll
            for (int k = 0; k < 2; ++k) *reinterpret_cast<float2*>(part + k * 8 * (D + 4) + D) = done ? make_float2(m_ref[k] - lvsc, l_sum[k]) : make_float2(-INFINITY, 0.f);
        }
        if (done) {
            const bool words = !parts && p.out_dtype != TQ_F32, f16 = p.out_dtype == TQ_F16, odd = (t2 & 2) != 0;
            float il[2];
            bool store[2];
            char* dst[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                il[k] = parts ? 1.f : 1.f / l_sum[k];
                store[k] = parts || row_valid(mf + 8 * k);
                const int64_t at = row_q_index(mf + 8 * k) + (words ? (t2 & 4) + (odd ? 8 : 0) : t2);
                dst[k] = parts ? reinterpret_cast<char*>(part + k * 8 * (D + 4) + t2) : static_cast<char*>(p.out) + at * (words ? 2 : 4);
            }
            if (__any_sync(0xffffffffu, store[0] || store[1])) {
                auto rows = [&](int c0, uint32_t (&o)[16]) {           // of eight columns: two of row g, two of row g + 8
                    tmem_ld_frag32(t_frag + P::COL_O + q * DP + c0, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * il[(i >> 1) & 1]);
                };
                if (!words) {
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += 32) {
                        uint32_t o[16];
                        rows(c0, o);
#pragma unroll
                        for (int i = 0; i < 16; i += 2)
                            if (store[(i >> 1) & 1]) *reinterpret_cast<uint2*>(dst[(i >> 1) & 1] + 4 * c0 + 8 * (i & 12)) = make_uint2(o[i], o[i + 1]);
                    }
                } else {
                    // two neighbouring lanes trade words: four columns each, the even one of eight columns, the odd one of the next eight
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += 32) {
                        uint32_t o[16];
                        rows(c0, o);
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            const float x = __uint_as_float(o[i]), z = __uint_as_float(o[i + 1]);
                            o[i] = f16 ? pack_h2(x, z) : pack_bf2(x, z);
                        }
#pragma unroll
                        for (int i = 0; i < 16; i += (i & 2) ? 6 : 2) {
                            const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? o[i] : o[i + 4], 1);
                            if (store[(i >> 1) & 1]) *reinterpret_cast<uint2*>(dst[(i >> 1) & 1] + 2 * c0 + 4 * (i & 12)) = odd ? make_uint2(other, o[i + 4]) : make_uint2(o[i], other);
                        }
                    }
                }
            }
        }
    } else {
        // ======================= softmax warps without a row: the others' exponentials have the pipe to themselves =======================
        // (8 queries x 4 heads over 2000 tokens, four sequences: 43.4 -> 37.0 us, d = 64 34.4 -> 28.9)
        // (What they leave in tensor memory meets rows that nobody reads.  A score buffer is full again only behind the products that every warp of
        // the query tile has arrived for, so that no arrival is a phase early.)
        const int q = warp >> 3;
        for (int j = 0; j <= n; ++j) {
            if (j == n_p && n_p > 0) mbar_arrive(bar(ROT_A + q));
            if (j == n || !__all_sync(0xffffffffu, wait_bar(S_FULL + sbuf(q, j), sph(j)))) break;
            mbar_arrive(bar(P_FULL + sbuf(q, j)));
            mbar_arrive(bar(SC_FREE + j % NSC));
        }
    }
    // ---------------- teardown: every loop above is bounded, so every thread gets here ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == P::SW) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- the queries ----------------------------------------------------------------------------------------------------------
// The queries of a round's lanes times f = scale * log2(e) as fp16: as they are, for the uncompressed tokens, and rotated (q @ R^T,
// rotation.py:81-110) in float32 accuracy - the roundings that the kernels which unpack as they go give their queries.  And R as the
// B operand of the rotation back: per pass, high then low parts; rows k of 128 bytes, blocks of 64 columns, 128-byte swizzle.
//
// 16 rows per warp on mma.sync.  A 16-bit query under the power of two that takes its row's largest element to [2^7, 2^8) is an fp16
// number up to 2^-33 of that element; the matrix is split into fp16 high and 2^-11 low parts and sits in shared memory as B
// fragments {high, low}, NC of its columns; a lane reads 16 bytes of it for two products.  A CTA with few rows of its own takes few
// columns: the table's set-up is what such a call waits for.
template <int D, int NC> __host__ __device__ constexpr uint32_t rot_bytes() { return (D / 16) * (NC / 8) * 512u; }
constexpr int Q_T = 512;
template <int D, int NC>
__global__ void __launch_bounds__(Q_T, 1) fa_query_kernel(const void* q, int q_dtype, float f, const float* rot, int64_t n_rows, __half* raw, __half* rotated, unsigned char* r_img) {
    using P = Plan<D>;
    constexpr int KS = D / 16, NTL = NC / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint4* tab = reinterpret_cast<uint4*>(smem_raw);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, col0 = blockIdx.y * NC;
    if (rotated) {         // (constants only: before the wait)
        // B[k][n] = R[col0 + n][k]; fragment of (k step, eight columns): lane 4 (n % 8) + (k % 8) / 2 holds the pairs (k, k + 1) and
        // (k + 8, k + 9).  Rows of R are read in whole sectors, the pairs put where they belong.
#pragma unroll 8
        for (int i = threadIdx.x; i < NC * (D / 4); i += Q_T) {
            const int n = i / (D / 4), k = (i - n * (D / 4)) * 4;
            const float4 x = __ldg(reinterpret_cast<const float4*>(rot + (col0 + n) * D + k));
            uint32_t h0, l0, h1, l1;
            split2(x.x, x.y, h0, l0);
            split2(x.z, x.w, h1, l1);
            uint32_t* w = reinterpret_cast<uint32_t*>(tab + ((k >> 4) * NTL + (n >> 3)) * 32 + (n & 7) * 4 + ((k & 7) >> 1)) + ((k >> 3) & 1);
            w[0] = h0; w[2] = l0; w[4] = h1; w[6] = l1;
        }
    }
    pdl_wait();
    pdl_trigger();         // (the expansion runs beside this: what came before has ended)
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * Q_T + threadIdx.x; rotated && i < D * (P::DP / 8); i += gridDim.x * gridDim.y * Q_T) {
        const int k = i / (P::DP / 8), c = i - k * (P::DP / 8), x = c * 8 / P::RC, cc = c - x * (P::RC / 8);       // row, chunk of eight columns, pass, chunk in it
        uint32_t h[4] = {0u, 0u, 0u, 0u}, l[4] = {0u, 0u, 0u, 0u};
        if (c * 8 < D) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(rot + k * D + c * 8)), b = __ldg(reinterpret_cast<const float4*>(rot + k * D + c * 8 + 4));
            split2(a.x, a.y, h[0], l[0]); split2(a.z, a.w, h[1], l[1]);
            split2(b.x, b.y, h[2], l[2]); split2(b.z, b.w, h[3], l[3]);
        }
        unsigned char* dst = r_img + x * 2 * P::R_HALF + (cc >> 3) * P::RBLK + k * 128 + (((cc & 7) ^ (k & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(dst + P::R_HALF) = make_uint4(l[0], l[1], l[2], l[3]);
    }
    __syncthreads();
    auto two = [&](uint32_t w) { return q_dtype == TQ_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w)) : make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); };
    for (int64_t r0 = (int64_t(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 16; r0 < n_rows; r0 += int64_t(gridDim.x) * (Q_T / 2)) {
        // a[ks][r]: columns 16 ks + 2 t, + 1 of rows g (r = 0) and g + 8 (1), then the same + 8 (2, 3)
        uint32_t a[KS][4];
        float m[2] = {0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int64_t row = r0 + g + (r & 1) * 8;
                a[ks][r] = row < n_rows ? __ldg(reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(q) + row * D + ks * 16 + 2 * t + (r >> 1) * 8)) : 0u;
            }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int64_t row = r0 + g + (r & 1) * 8;
                const float2 v = two(a[ks][r]);
                m[r & 1] = fmaxf(m[r & 1], fmaxf(fabsf(v.x), fabsf(v.y)));
                if (blockIdx.y == 0 && row < n_rows) *reinterpret_cast<uint32_t*>(raw + row * D + ks * 16 + 2 * t + (r >> 1) * 8) = pack_h2(v.x * f, v.y * f);
            }
        if (!rotated) continue;
        float sc[2], back[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int off = 1; off < 4; off <<= 1) m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], off));
            sc[r] = stage_scale(__float_as_uint(m[r]));
            back[r] = f / sc[r];
        }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int r = 0; r < 4; ++r) { const float2 v = two(a[ks][r]); a[ks][r] = pack_h2(v.x * sc[r & 1], v.y * sc[r & 1]); }
#pragma unroll 2
        for (int nt = 0; nt < NTL; ++nt) {             // columns 8 nt + 2 t, + 1 of the rows
            float h[4] = {0.f, 0.f, 0.f, 0.f}, l[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const uint4 w = tab[(ks * NTL + nt) * 32 + lane];
                mma16816(h, a[ks][0], a[ks][1], a[ks][2], a[ks][3], w.x, w.y);
                mma16816(l, a[ks][0], a[ks][1], a[ks][2], a[ks][3], w.z, w.w);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int64_t row = r0 + g + 8 * r;
                if (row < n_rows)
                    *reinterpret_cast<uint32_t*>(rotated + row * D + col0 + nt * 8 + 2 * t) =
                        pack_h2(fmaf(l[2 * r], 1.f / 2048.f, h[2 * r]) * back[r], fmaf(l[2 * r + 1], 1.f / 2048.f, h[2 * r + 1]) * back[r]);
            }
        }
    }
}

// Partials of a row block's key ranges -> result: a warp per row.
template <int D>
__global__ void __launch_bounds__(256) fa_merge_kernel(Params p, int64_t n_rows) {
    constexpr int ROWS = Plan<D>::NQ * TM;
    const int lane = threadIdx.x & 31;
    const int64_t i = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);               // row of the launch: (lane x head group, row block, row)
    if (i >= n_rows) return;
    const int m = int(i % ROWS), blk = int(i / ROWS % p.n_blk), y = int(i / ROWS / p.n_blk);
    const int lane_c = y / p.HG, hg = y - lane_c * p.HG, gl = p.lane0 + lane_c, b = gl / p.Hkv, hkv = gl - b * p.Hkv;
    const int tok = blk * Plan<D>::NQ * p.QT + (m >> 7) * p.QT + (m & 127) / p.GP, hh = (m & 127) % p.GP;
    if (hh >= min(HPG, p.G - hg * HPG) || tok >= p.Tq) return;
    const float* part = p.part + ((int64_t(y) * p.n_blk + blk) * p.n_splits * ROWS + m) * (D + 4);
    const int64_t stride = int64_t(ROWS) * (D + 4);
    float mm = -INFINITY, ll = 0.f;
    if (lane < p.n_splits) { mm = part[lane * stride + D]; ll = part[lane * stride + D + 1]; }
    float M = mm;
#pragma unroll
    for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    // (a range without a visible token has sum 0 and left no sums; one whose sum is not a number makes the row that)
    const float w = ll != 0.f ? ex2(mm - M) : 0.f;
    float sum = ll != 0.f ? w * ll : 0.f;
#pragma unroll
    for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    float acc[D / 32];
#pragma unroll
    for (int u = 0; u < D / 32; ++u) acc[u] = 0.f;
    for (int s = 0; s < p.n_splits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s);
        if (ws == 0.f) continue;
#pragma unroll
        for (int u = 0; u < D / 32; ++u) acc[u] = fmaf(ws, part[s * stride + u * 32 + lane], acc[u]);
    }
    const int64_t o = ((int64_t(b) * p.Hq + hkv * p.G + hg * HPG + hh) * p.Tq + tok) * D;
    const float il = 1.f / sum;
#pragma unroll
    for (int u = 0; u < D / 32; ++u) store_from_f32(p.out, p.out_dtype, o + u * 32 + lane, acc[u] * il);
}

// ---- expansion: codes -> fp16 centroids, uncompressed tokens -> fp16 rows, norms --------------------------------------------
struct ExpandParams {
    DecodeParams c; int lane0, n_lanes, c64, ts, blocks_per_lane, steps;      // blocks of packed rows per lane and side, steps of a block
    __half *k, *v; float *kn, *vn;
};
constexpr int EX_T = 256, EX_U = 4;                    // a block: `steps` times EX_U x EX_T chunks of eight coordinates of one side of a lane
template <int D, int BH, int BL>
__device__ __forceinline__ void expand_block(const ExpandParams& e, int lane_c, int side, int blk) {
    constexpr int CPR = D / 8, HALF = BL ? D / 2 : D, WH = HALF * BH / 8, WL = BL ? HALF * BL / 8 : 0;
    const DecodeParams& c = e.c;
    __shared__ uint32_t ctab[32];
    const int64_t lane = e.lane0 + lane_c;
    const uint8_t* src_h = (side ? c.v_hi : c.k_hi) + lane * c.c_ls * WH;
    const uint8_t* src_l = BL ? (side ? c.v_lo : c.k_lo) + lane * c.c_ls * WL : nullptr;
    const float* norms = (side ? c.v_norms : c.k_norms) + lane * c.c_ls;
    float* nn = (side ? e.vn : e.kn) + int64_t(lane_c) * e.ts;
    __half* dst = (side ? e.v : e.k) + int64_t(lane_c) * e.ts * D;
    const uint32_t n = uint32_t(e.c64) * CPR;
    const uint32_t i0 = uint32_t(blk * e.steps) * (EX_U * EX_T) + threadIdx.x;
    uint32_t w[EX_U];
    auto load = [&](uint32_t i) -> uint32_t {
        const uint32_t row = i / CPR, ch = i - row * CPR;
        if (row >= uint32_t(c.c_len)) return 0u;
        if (ch == 0) nn[row] = norms[row];
        if (BL && ch >= CPR / 2) return dqtc::load_codes<(BL ? BL : 1)>(src_l + int64_t(row) * WL + (ch - CPR / 2) * BL);
        return dqtc::load_codes<BH>(src_h + int64_t(row) * WH + ch * BH);
    };
#pragma unroll
    for (int u = 0; u < EX_U; ++u) w[u] = load(i0 + u * EX_T);
    if (threadIdx.x < 32) {                            // fp16 centroids, the values' under their table's scale
        const int lo = threadIdx.x >> 4, k = threadIdx.x & 15;
        const float* src = lo ? (side ? c.vc_lo : c.kc_lo) : (side ? c.vc_hi : c.kc_hi);
        const bool in = k < (1 << (lo ? BL : BH)) && (!lo || BL);
        ctab[threadIdx.x] = in ? uint32_t(__half_as_ushort(__float2half_rn(src[k] * (side ? (lo ? c.v_scale_lo : c.v_scale_hi) : 1.f)))) : 0u;
    }
    __syncthreads();
    dqtc::Planes<BH> th;
    dqtc::Planes<BL> tl;
    th.load(ctab);
    tl.load(ctab + 16);
#pragma unroll 1
    for (int it = 0; it < e.steps; ++it) {
        const uint32_t i1 = i0 + it * (EX_U * EX_T);
#pragma unroll
        for (int u = 0; u < EX_U; ++u) {
            const uint32_t i = i1 + u * EX_T, row = i / CPR, ch = i - row * CPR;
            if (i >= n) return;                        // (i only grows)
            uint4 x = make_uint4(0u, 0u, 0u, 0u);      // (rows between the last packed token and the next multiple of 64: weight 0 times these)
            if (row < uint32_t(c.c_len)) {
                if (BL && ch >= CPR / 2) { if constexpr (BL != 0) x = tl.template lookup<0>(dqtc::Planes<BL>::nibbles(w[u])); }
                else x = th.template lookup<0>(dqtc::Planes<BH>::nibbles(w[u]));
            } else if (ch == 0) nn[row] = 0.f;
            if (it + 1 < e.steps) w[u] = load(i + EX_U * EX_T);       // this slot's next codes are on their way under the other slots' stores
            *reinterpret_cast<uint4*>(dst + int64_t(i) * 8) = x;
        }
    }
}
// Packed rows as unit vectors in rotated space (what the kernels that unpack as they go multiply with); uncompressed tokens a warp
// per (lane, side, token): float16 rows as they are, float32 / bfloat16 rows under a power-of-two scale (largest magnitude into
// [2^7, 2^8)) whose inverse takes the norm's place; zero norms behind the last token.
template <int D>
__global__ void __launch_bounds__(EX_T) fa_expand_kernel(const __grid_constant__ ExpandParams e) {
    const DecodeParams& c = e.c;
    const int n_packed = e.n_lanes * 2 * e.blocks_per_lane;
    if (int(blockIdx.x) < n_packed) {
        const int ls = blockIdx.x / e.blocks_per_lane, blk = blockIdx.x - ls * e.blocks_per_lane, side = ls & 1, lane_c = ls >> 1;
        switch (side ? c.vb_hi * 8 + c.vb_lo : c.kb_hi * 8 + c.kb_lo) {
            case 8: expand_block<D, 1, 0>(e, lane_c, side, blk); break;
            case 16: expand_block<D, 2, 0>(e, lane_c, side, blk); break;
            case 24: expand_block<D, 3, 0>(e, lane_c, side, blk); break;
            case 32: expand_block<D, 4, 0>(e, lane_c, side, blk); break;
            case 17: expand_block<D, 2, 1>(e, lane_c, side, blk); break;
            case 26: expand_block<D, 3, 2>(e, lane_c, side, blk); break;
            default: expand_block<D, 4, 3>(e, lane_c, side, blk); break;      // (the host admits no other)
        }
    } else {
        const int lane = threadIdx.x & 31, n_dense = int(c.sink_len + c.res_len), n_items = e.ts - e.c64;
        const int64_t i = int64_t(blockIdx.x - n_packed) * (EX_T / 32) + (threadIdx.x >> 5);
        if (i < int64_t(e.n_lanes) * 2 * n_items) {
            const int item = int(i % n_items), side = int(i / n_items) & 1, lc = int(i / n_items / 2);
            float* nn = (side ? e.vn : e.kn) + int64_t(lc) * e.ts + e.c64 + item;
            if (item >= n_dense) {
                if (lane == 0) *nn = 0.f;
            } else {
                const bool in_sink = item < c.sink_len;
                const int64_t src = (in_sink ? (e.lane0 + lc) * c.sink_ls + item : (e.lane0 + lc) * c.res_ls + (item - c.sink_len)) * D;
                const void* base = in_sink ? (side ? c.sink_v : c.sink_k) : (side ? c.res_v : c.res_k);
                __half* dst = (side ? e.v : e.k) + (int64_t(lc) * e.ts + e.c64 + item) * D;
                float x[D / 32], mx = 0.f;
#pragma unroll
                for (int u = 0; u < D / 32; ++u) { x[u] = load_as_f32(base, c.dense_dtype, src + u * 32 + lane); mx = fmaxf(mx, fabsf(x[u])); }
                float sc = 1.f;
                if (c.dense_dtype != TQ_F16) {
#pragma unroll
                    for (int off = 16; off; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
                    sc = stage_scale(__float_as_uint(mx));
                }
#pragma unroll
                for (int u = 0; u < D / 32; ++u) dst[u * 32 + lane] = __float2half_rn(x[u] * sc);
                if (lane == 0) *nn = 1.f / sc;
            }
        }
    }
    pdl_wait();            // (this grid's end stands for the query kernel's too)
}

static PFN_cuTensorMapEncodeTiled encoder() {
    static PFN_cuTensorMapEncodeTiled fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(f);
    }();
    return fn;
}

static int sm_count() {
    static std::atomic<int> n[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int v = n[dev].load();
    if (!v) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        n[dev].store(v);
    }
    return v;
}

static size_t up(size_t v) { return (v + 255) / 256 * 256; }

// Key ranges per row block: as many as shorten the whole launch, a CTA costing its tiles and some twelve more for set-up, first
// scores and the partials (with four, 512 queries x 32 lanes over 16,384 tokens were split for a merge of 34 us and no gain).
static int ranges(int64_t tiles, int64_t ctas, int64_t most) {
    const int64_t sms = sm_count();
    double best = 0.0;
    int n = 1;
    for (int s = 1; s <= std::min<int64_t>(most, MAX_RANGES) && (s == 1 || tiles >= 2 * s); ++s) {
        const double t = double((ctas * s + sms - 1) / sms) * (double((tiles + s - 1) / s) + 12.0) + (s > 1 ? 8.0 : 0.0);
        if (s == 1 || t < best) { best = t; n = s; }
    }
    return n;
}

// How a call is laid out in the workspace, once for all of its rounds: `chunk` cache lanes are expanded and attended to at a time (the
// last round may have fewer).  Everything fits ws_bytes, whatever the sizes, from least<D>() bytes on: where the partials do not, there
// are fewer key ranges.
struct Layout {
    int GP, QT, n_blocks, chunk, n_splits, c64, ts;
    size_t v, kn, vn, q, r, part, bytes;               // (the key rows come first)
};
static int groups_of(int G) { return (G + HPG - 1) / HPG; }
template <int D> static size_t block_bytes(int G) { return size_t(groups_of(G)) * Plan<D>::NQ * TM * (D + 4) * 4; }      // a lane's partials of a row block and range
template <int D> static void row_shape(Layout& l, int G, int t_q) {
    const int g = std::min(G, HPG);
    l.GP = g <= 1 ? 1 : g <= 2 ? 2 : g <= 4 ? 4 : 8;
    l.QT = TM / l.GP;
    l.n_blocks = (t_q + Plan<D>::NQ * l.QT - 1) / (Plan<D>::NQ * l.QT);
}
// rows, norms, queries (as they are, rotated) of n lanes; R
template <int D> static void row_areas(Layout& l, int n, int G, int t_q) {
    const size_t rows = size_t(n) * l.ts;
    l.v = up(rows * D * 2);
    l.kn = l.v + up(rows * D * 2);
    l.vn = l.kn + up(rows * 4);
    l.q = l.vn + up(rows * 4);
    l.r = l.q + 2 * up(size_t(n) * G * t_q * D * 2);
    l.part = l.r + up(size_t(Plan<D>::PASSES) * 2 * Plan<D>::R_HALF);
}
template <int D> static Layout layout(int lanes, int G, int64_t c_len, int64_t n_dense, int t_q, size_t ws_bytes) {
    Layout l{};
    row_shape<D>(l, G, t_q);
    l.c64 = int((c_len + 63) / 64 * 64);
    l.ts = int((l.c64 + n_dense + 127) / 128 * 128);
    for (l.chunk = lanes;; l.chunk = (l.chunk + 1) / 2) {
        row_areas<D>(l, l.chunk, G, t_q);
        if (l.chunk == 1 || l.part <= ws_bytes) break;
    }
    const size_t parts = block_bytes<D>(G) * l.chunk * l.n_blocks;                  // the partials of one range
    l.n_splits = ranges(l.c64 / 64 + (n_dense + 63) / 64, int64_t(l.n_blocks) * l.chunk * groups_of(G), ws_bytes > l.part ? int64_t((ws_bytes - l.part) / parts) : 0);
    l.bytes = l.part + (l.n_splits == 1 ? 0 : parts * l.n_splits);
    return l;
}

// The workspace a call asks for: all lanes' rows, PART_CAP for partials at most, WS_CAP in all unless a single lane needs more.  Only the number of tokens is known here, not their regions: up to 63 rows more.
constexpr size_t WS_CAP = size_t(1) << 29, PART_CAP = size_t(1) << 27;
template <int D> static Layout rows_of(int lanes, int G, int64_t total, int t_q) {
    Layout l{};
    row_shape<D>(l, G, t_q);
    l.ts = int((total + 63 + 127) / 128 * 128);
    row_areas<D>(l, lanes, G, t_q);
    return l;
}
template <int D> static size_t least(int G, int64_t total, int t_q) { return rows_of<D>(1, G, total, t_q).part; }
template <int D> static size_t workspace(int lanes, int G, int64_t total, int t_q) {
    const Layout l = rows_of<D>(lanes, G, total, t_q);
    const size_t one = block_bytes<D>(G) * lanes * l.n_blocks;
    const int n = ranges((total + 126) / 64, int64_t(l.n_blocks) * lanes * groups_of(G), MAX_RANGES);
    const size_t parts = n == 1 ? 0 : std::min(one * std::min(n + 1, MAX_RANGES), PART_CAP);
    return std::max(std::min(l.part + parts, WS_CAP), least<D>(G, total, t_q) + parts);
}

template <int D> static int run(const DecodeParams& c, const void* q, int q_dtype, void* out, int out_dtype, int t_q, int64_t q_pos0, unsigned char* ws,
                                size_t ws_bytes, cudaStream_t s) {
    using P = Plan<D>;
    constexpr int NC = D > 128 ? 128 : D, NC_FEW = 32;
    const int64_t n_dense = c.sink_len + c.res_len;
    const int lanes = c.B * c.Hkv;
    const Layout l = layout<D>(lanes, c.G, c.c_len, n_dense, t_q, ws_bytes);
    if (l.bytes > ws_bytes) return fail(TQ_ERR_INVALID, "tq_prefill_attn: workspace %zu B < %zu B", ws_bytes, l.bytes);
    static std::atomic<bool> set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !set[dev].load()) {
        cudaError_t e = cudaFuncSetAttribute(fa_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(P::SMEM));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fa_query_kernel<D, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(rot_bytes<D, NC>()));
        if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: shared memory %zu B: %s", P::SMEM, cudaGetErrorString(e));
        set[dev].store(true);
    }
    Params p{};
    p.out = out; p.out_dtype = out_dtype;
    p.Hq = c.Hq; p.Hkv = c.Hkv; p.G = c.G; p.HG = c.HG; p.GP = l.GP; p.QT = l.QT; p.Tq = t_q;
    p.q_pos0 = int(q_pos0); p.sink_len = int(c.sink_len); p.c_len = int(c.c_len); p.n_dense = int(n_dense); p.c64 = l.c64;
    p.kn = reinterpret_cast<const float*>(ws + l.kn); p.vn = reinterpret_cast<const float*>(ws + l.vn); p.ts = l.ts;
    p.n_blk = l.n_blocks; p.n_splits = l.n_splits;
    p.part = reinterpret_cast<float*>(ws + l.part);
    p.r_img = ws + l.r;
    p.v_inv_hi = 1.f / c.v_scale_hi; p.v_inv_lo = c.vb_lo ? 1.f / c.v_scale_lo : p.v_inv_hi;
    if (!(p.status = decode_status_ptr())) return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: cannot locate the status word");
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    const int sms = sm_count();
    for (int lane0 = 0; lane0 < lanes; lane0 += l.chunk) {
        const int n = std::min(l.chunk, lanes - lane0);
        const bool rotate = c.c_len > 0;
        const int64_t rows = int64_t(n) * c.G * t_q;
        __half* q_raw = reinterpret_cast<__half*>(ws + l.q);
        __half* q_rot = q_raw + up(size_t(l.chunk) * c.G * t_q * D * 2) / 2;
        cudaLaunchConfig_t cfg{};
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const bool few = rows <= 16 * 2 * int64_t(sms);         // two groups of sixteen rows per SM
        cfg.gridDim = few ? dim3(unsigned((rows + 63) / 64), D / NC_FEW) : dim3(unsigned(std::min<int64_t>((rows + 15) / 16, sms)), D / NC);
        cfg.blockDim = dim3(Q_T);
        cfg.dynamicSmemBytes = few ? rot_bytes<D, NC_FEW>() : rot_bytes<D, NC>();
        cudaLaunchKernelEx(&cfg, few ? fa_query_kernel<D, NC_FEW> : fa_query_kernel<D, NC>, static_cast<const void*>(static_cast<const uint16_t*>(q) + int64_t(lane0) * c.G * t_q * D), q_dtype,
                           float(c.scale * LOG2E), c.rot, rows, q_raw, rotate ? q_rot : nullptr, ws + l.r);
        if (int rc = check_launch("tq_prefill_attn")) return rc;
        ExpandParams e{};
        e.c = c; e.lane0 = lane0; e.n_lanes = n; e.c64 = l.c64; e.ts = l.ts;
        // (blocks of eight steps pay for their set-up - centroids, tables in registers - best; with few tokens it takes as many blocks as fit the SMs)
        const int64_t steps = (int64_t(l.c64) * (D / 8) + EX_T * EX_U - 1) / (EX_T * EX_U);
        e.steps = int(std::max<int64_t>(1, std::min<int64_t>(8, steps * n * 2 / (8 * sms))));
        e.blocks_per_lane = int((steps + e.steps - 1) / e.steps);
        e.k = reinterpret_cast<__half*>(ws); e.v = reinterpret_cast<__half*>(ws + l.v);
        e.kn = reinterpret_cast<float*>(ws + l.kn); e.vn = reinterpret_cast<float*>(ws + l.vn);
        cfg.gridDim = dim3(unsigned(int64_t(n) * 2 * e.blocks_per_lane + (int64_t(n) * 2 * (l.ts - l.c64) + EX_T / 32 - 1) / (EX_T / 32)));
        cfg.blockDim = dim3(EX_T);
        cfg.dynamicSmemBytes = 0;
        cudaLaunchKernelEx(&cfg, fa_expand_kernel<D>, e);
        if (int rc = check_launch("tq_prefill_attn")) return rc;
        // keys, values (rows past the last token read as zeros) as (column, row, lane); queries as (column, head, token): a box is a query
        // tile's columns, rows (token, head) in the order that the tiles have
        CUtensorMap maps[4];
        for (int i = 0; i < 4; ++i) {
            const bool kv = i < 2;
            const cuuint64_t row = cuuint64_t(D) * 2;
            const cuuint64_t dims[3] = {cuuint64_t(D), kv ? cuuint64_t(l.c64 + n_dense) : cuuint64_t(n) * c.G, kv ? cuuint64_t(n) : cuuint64_t(t_q)};
            const cuuint64_t strides[2] = {kv ? row : row * t_q, kv ? row * l.ts : row};
            const cuuint32_t box[3] = {64, kv ? cuuint32_t(P::TN) : cuuint32_t(l.GP), kv ? 1u : cuuint32_t(l.QT)}, es[3] = {1, 1, 1};
            if (encoder()(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, i == 0 ? e.k : i == 1 ? e.v : i == 2 && rotate ? q_rot : q_raw, dims, strides, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: cannot describe the expanded rows to the tensor memory accelerator");
        }
        p.lane0 = lane0; p.n_lanes = n;
        cfg.gridDim = dim3(unsigned(int64_t(n) * c.HG * l.n_blocks * l.n_splits));
        cfg.blockDim = dim3(P::NT);
        cfg.dynamicSmemBytes = P::SMEM;
        cudaLaunchKernelEx(&cfg, fa_kernel<D>, p, maps[0], maps[1], maps[2], maps[3]);
        if (int rc = check_launch("tq_prefill_attn")) return rc;
        if (l.n_splits > 1) {
            const int64_t rows = int64_t(n) * c.HG * l.n_blocks * P::NQ * TM;
            fa_merge_kernel<D><<<unsigned((rows + 7) / 8), 256, 0, s>>>(p, rows);
            if (int rc = check_launch("tq_prefill_attn")) return rc;
        }
    }
    return TQ_OK;
}

}  // namespace fa

size_t prefill_fa_workspace(int batch, int n_q_heads, int n_kv_heads, int d, int64_t total, int t_q) {
    if (batch <= 0 || n_kv_heads <= 0 || n_q_heads <= 0 || n_q_heads % n_kv_heads || t_q <= 0 || total < t_q) return 0;
    const int lanes = batch * n_kv_heads, g = n_q_heads / n_kv_heads;
    if (d == 64) return fa::workspace<64>(lanes, g, total, t_q);
    if (d == 96) return fa::workspace<96>(lanes, g, total, t_q);
    if (d == 128) return fa::workspace<128>(lanes, g, total, t_q);
    return d == 256 ? fa::workspace<256>(lanes, g, total, t_q) : 0;
}
static size_t prefill_fa_least(int g, int d, int64_t total, int t_q) {
    return d == 64 ? fa::least<64>(g, total, t_q) : d == 96 ? fa::least<96>(g, total, t_q) : d == 128 ? fa::least<128>(g, total, t_q) : fa::least<256>(g, total, t_q);
}

// Whether this kernel takes the call with this workspace; the caller has validated the arguments.
bool prefill_fa_applicable(const tq_decode_args* a, int t_q) {
    const int64_t total = a->c_len + a->sink_len + a->res_len;
    if (a->q_dtype == TQ_F32) return false;                    // (its callers hand over no workspace)
    if (!a->workspace || !aligned(a->workspace, 256) || total >= (int64_t(1) << 30) || !fa::encoder()) return false;
    if (a->c_len > 0) {
        if ((a->k_bits_lo && a->k_bits_lo != a->k_bits_hi - 1) || (a->v_bits_lo && a->v_bits_lo != a->v_bits_hi - 1)) return false;
        // eight codes of 4 bits are read as a word, of 2 bits as half of one
        if (!aligned(a->k_hi, 4) || !aligned(a->v_hi, 4) || (a->k_bits_lo && !aligned(a->k_lo, 4)) || (a->v_bits_lo && !aligned(a->v_lo, 4))) return false;
    }
    if (!aligned(a->q, 4) || !aligned(a->out, 16) || !aligned(a->rot, 16)) return false;
    return a->workspace_bytes >= prefill_fa_least(a->n_q_heads / a->n_kv_heads, a->d, total, t_q);
}

// Whether prefill_tc.cu, which unpacks as it goes, is the faster one of two that take the call: with a single block of 128 query rows
// per lane nothing is unpacked twice there, and the expansion here costs as much as the attention.  Its time goes by waves of CTAs, a
// lane each, this one's by lanes x tokens; us on 148 SMs, fa / tc, 32 queries of 4 heads, 4-bit keys and 2-bit values at d = 128 (other widths:
// always fa): 64 lanes x 8192 175 / 294, 112 x 8192 285 / 332, 128 x 8192 348 / 336, 112 x 16384 541 / 526, 128 x 4000 171 / 199, 160 x 8192 443 /
// 644, 224 x 8192 568 / 666, 256 x 8192 695 / 676.  (A sweep of 236 calls of 16 to 296 lanes: the rule's choice is never more than 3 % slower than the other.)
bool prefill_tc_faster(const tq_decode_args* a, int t_q) {
    const int g = a->n_q_heads / a->n_kv_heads, gp = g <= 1 ? 1 : g <= 2 ? 2 : g <= 4 ? 4 : 8;
    if (a->d != 128 || a->k_bits_hi != 4 || a->k_bits_lo || a->v_bits_hi != 2 || a->v_bits_lo || t_q > fa::TM / gp) return false;
    const int64_t lanes = int64_t(a->batch) * a->n_kv_heads * fa::groups_of(g), total = a->c_len + a->sink_len + a->res_len, sms = fa::sm_count();
    const double fa_us = 20.0 + 3.2e-4 * double(lanes) * double(total), tc_us = double((lanes + sms - 1) / sms) * (100.0 + 0.0265 * double(total));
    return tc_us < fa_us;
}

int launch_prefill_fa(const DecodeParams& c, const void* q, int q_dtype, void* out, int out_dtype, int t_q, int64_t q_pos0, void* ws, size_t ws_bytes,
                      cudaStream_t s) {
    unsigned char* w = static_cast<unsigned char*>(ws);
    if (c.D == 64) return fa::run<64>(c, q, q_dtype, out, out_dtype, t_q, q_pos0, w, ws_bytes, s);
    if (c.D == 96) return fa::run<96>(c, q, q_dtype, out, out_dtype, t_q, q_pos0, w, ws_bytes, s);
    if (c.D == 128) return fa::run<128>(c, q, q_dtype, out, out_dtype, t_q, q_pos0, w, ws_bytes, s);
    return fa::run<256>(c, q, q_dtype, out, out_dtype, t_q, q_pos0, w, ws_bytes, s);
}

}  // namespace tq

extern "C" size_t tq_prefill_workspace_bytes(int batch, int n_q_heads, int n_kv_heads, int d, int64_t total_len, int t_q) {
    return tq::prefill_fa_workspace(batch, n_q_heads, n_kv_heads, d, total_len, t_q);
}

extern "C" size_t tq_prefill_workspace_used(int batch, int n_q_heads, int n_kv_heads, int d, int64_t c_len, int64_t dense_len, int t_q, size_t workspace_bytes) {
    using namespace tq;
    const int64_t total = c_len + dense_len;
    if (prefill_fa_workspace(batch, n_q_heads, n_kv_heads, d, total, t_q) == 0 || workspace_bytes < prefill_fa_least(n_q_heads / n_kv_heads, d, total, t_q)) return 0;
    const int lanes = batch * n_kv_heads, g = n_q_heads / n_kv_heads;
    if (d == 64) return fa::layout<64>(lanes, g, c_len, dense_len, t_q, workspace_bytes).bytes;
    if (d == 96) return fa::layout<96>(lanes, g, c_len, dense_len, t_q, workspace_bytes).bytes;
    if (d == 128) return fa::layout<128>(lanes, g, c_len, dense_len, t_q, workspace_bytes).bytes;
    return fa::layout<256>(lanes, g, c_len, dense_len, t_q, workspace_bytes).bytes;
}
