// Dequantize on the fifth-generation tensor cores: unpack -> centroid -> inverse rotation -> scale (+ QJL correction)
// (TurboQuantMSE.dequantize / cache._dequantize_kv(_fractional) / metal_dequantize: quantizer.py:87-109,
// cache.py:276-343, 396-427, kernels.py:313-360) for head_dim 64 / 96 / 128 / 256, any bit width 1-4 and the fractional
// splits, one or two jobs (keys and values) per launch; unaligned outputs stay with the CUDA-core row kernel (rowops.cu).
//
//   out[t][j] = norm[t] * sum_k c[code(t, k)] R[k][j]          (y @ R, rotation.py:68-78)
//
// is a dense 128 x d x d contraction per 128 rows.  To stay float32-faithful on fp16 operands both factors are split,
// c = c_hi + 2^-11 c_lo and R = R_hi + 2^-11 R_lo, and three products are kept: c_hi R_hi in one accumulator,
// c_hi R_lo + c_lo R_hi in a second one that the epilogue adds with weight 2^-11 (the fourth product is below float32
// resolution).
//
// Persistent CTAs (one per SM) walk the 128-row tiles, 17 warps:
//   * warps 8-15 turn a tile's codes into fp16 A tiles (high parts, then low parts;
//     K-major, 128-byte swizzle) in a ring of buffers and stage the rows' norms, offsets, sign words;
//   * warp 16 (in uniform control flow, one elected lane) issues the tcgen05.mma: c_hi [R_hi | R_lo] as one product per K step, then c_lo R_hi, into
//     accumulator pair t & 1 - R sits in shared memory as MN-major B tiles built once per CTA (d = 256: a CTA owns 128 of
//     the output columns);
//   * warps 0-7 (two groups of four, alternating tiles) read both accumulators, a row per thread, combine, scale and stage
//     64 bytes of 32 rows at a time for a tiled bulk store.  With the sketch correction (c/d) gamma (signs @ S) they read
//     the accumulators in the register layout of mma.sync fragments instead, which compute the correction on +-1 operands.
// Every mbarrier wait is bounded (status 105); tensor memory is freed on every path.
//
// No pipe is full: at d = 128 (4 bits, float32 results) memory runs at 68 % of a copy, issue slots are 51 % busy, the tensor pipe
// 45 %, shared memory 30 %; what is left is the hand-over between the three roles of a tile.  Eight producer warps: with four, one per scheduler,
// the chains of a chunk do not overlap (166 us).  Measured at 134 million coordinates, float32 / fp16 results, against the
// four-warp table-lookup kernel before (d = 256 and sketches: the row kernel):
//   d = 128: 4 bits 132 / 118 us (163 / 150), 3.5 bits 138 / 122 (326 / 314), 3 bits 145 / 136 (165 / 156), 2 bits 128 / 108 (162 / 140)
//   d = 64: 4 bits 177 / 173 (228 / 215), 3.5 bits 185 / 178 (524 / 523);  d = 256: 4 bits 300 / 289 (3804 / 3793)
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace tq {

int* decode_status_ptr();

namespace dqtc {

constexpr int TM = 128, EPI_T = 128;
constexpr int PW = 8, RW = TM / PW, PROD_T = PW * 32;                         // producer warps, their rows of a tile
constexpr int MMA_W = 8 + PW, NT = (MMA_W + 1) * 32;
constexpr float QJL_C = 1.2533141373155003f;                                // sqrt(pi / 2), qjl.py:91-92
constexpr uint32_t WAIT_LIMIT = 4u << 20;
constexpr int ERR_WAIT = 105;
constexpr int PF_AHEAD = 4;                                                 // a tile's packed rows are asked for in L2 this many tiles early
constexpr int SLOTS = 6;                                                    // tiles whose rows' norms, offsets, sign words are kept
constexpr uint32_t TMEM_COLS = 512;                                         // accumulator pair b: columns 256 b (high), + NC (mixed products)

template <int D> struct Plan {
    static constexpr int NC = D == 64 ? 64 : 128;                           // output columns of a CTA (d = 96: the last 32 are zeros)
    static constexpr int KB = (D + 63) / 64;                                // 64-column blocks of an A tile
    static constexpr int NB = D == 256 ? 1 : 3;                             // A tiles in the ring
    static constexpr uint32_t ABLK = TM * 128u, A_TILE = KB * ABLK;         // K-major: 128 rows x 128 B per block
    static constexpr int RROWS = D == 96 ? 96 : D;
    static constexpr uint32_t RBLK = RROWS * 128u, R_TILE = (NC / 64) * RBLK;     // MN-major: d rows x 128 B per block of 64 columns
    static constexpr uint32_t OFF_R = 0;                                    // R_hi, then R_lo
    static constexpr uint32_t OFF_A = 2 * R_TILE;
    static constexpr uint32_t STG = D == 256 ? 2048 : 4096;                 // staging of an epilogue warp: one or two buffers of 32 rows x 64 B
    static constexpr uint32_t OFF_S = OFF_A + NB * A_TILE;                  // the eight warps' staging; QJL: S as mma B fragments instead,
                                                                            // [2 k-steps][NC / 8][hi | lo][32 lanes] x 8 B
    static constexpr uint32_t OFF_ROWS = OFF_S + 8 * STG;                     // uint4 [SLOTS][128]: norm, output offset / 8 elements (~0: no such row); cache lane and row in it (QJL: sign word, (c/d) residual norm)
    static constexpr uint32_t OFF_CTAB = OFF_ROWS + SLOTS * TM * 16;        // uint32 [2][16] centroids as {hi, lo} fp16 pairs
    static constexpr uint32_t OFF_BAR = OFF_CTAB + 128;
    static constexpr uint32_t OFF_SLOT = OFF_BAR + 128;                     // [0] tensor-memory base, [1] abort
    static constexpr size_t SMEM = OFF_SLOT + 16 + 1024;
    static_assert(SMEM <= 227 * 1024 && OFF_S % 1024 == 0 && 2 * (NC / 8) * 2 * 32 * 8 <= 8 * STG, "shared-memory plan");
    static_assert(RBLK % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
};
enum Bars { A_FULL = 0, A_FREE = 4, ACC_FULL = 8, ACC_FREE = 10, DRAIN = 12 };

struct Params {
    const uint8_t* packed_hi; const uint8_t* packed_lo; const float* norms;
    uint32_t n_rows, total; int64_t in_lane_stride;           // rows per lane, lanes x rows, lane stride (rows)
    int half, bits_hi, bits_lo, w_hi, w_lo;                   // half: coordinates in packed_hi; w: bytes per packed row
    const float* cent_hi; const float* cent_lo; const float* rot;
    const float* qjl_proj; const uint32_t* qjl_bits; const float* qjl_gamma;     // null: no correction
    void* out; int out_dtype; int64_t out_lane_stride, out_row_stride;
    int n_tiles;
    int follows;                                              // the second of a pair: it may run beside the first and ends after it
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
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// (issued by one elected lane of a warp in uniform control flow: the operands then come straight from uniform registers, where a
// single thread in a divergent branch moves each of them over one by one)
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
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
// 16 lanes x 64 columns: register 4 i + 2 h + e of thread (g, t) = row g + 8 h, column 8 i + 2 t + e
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* ptr) { asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr)); }
__device__ __forceinline__ uint32_t h2_bits(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t sign_pair16(uint32_t x) { return (x & 0x80008000u) ^ 0xBC00BC00u; }
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
// Operand tiles are blocks of 64 columns, rows of 128 B, 16-byte chunk c of row r at chunk position c ^ (r & 7) (128-byte swizzle).
__device__ __forceinline__ uint32_t chunk_off(uint32_t blk, int r, int c16) {
    return uint32_t(c16 >> 3) * blk + uint32_t(r) * 128u + (uint32_t((c16 & 7) ^ (r & 7)) << 4);
}
// K-major descriptor (rows = M index, 64-column blocks along K): the 16-column slab `ks` of the tile
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, uint32_t blk, int ks) {
    const uint32_t addr = tile + uint32_t(ks >> 2) * blk + uint32_t(ks & 3) * 32u;
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// MN-major descriptor (rows = K index, blocks of 64 columns along N): the 16-row slab `ks`
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile, uint32_t blk, int ks) {
    const uint32_t addr = tile + uint32_t(ks) * 2048u;
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(blk >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// kind::f16: fp32 accumulate, fp16 A (K-major) and B (MN-major), M = 128
__host__ __device__ constexpr uint32_t idesc_of(int n) { return (1u << 4) | (1u << 16) | (uint32_t(n >> 3) << 17) | (uint32_t(TM >> 4) << 24); }

// Eight codes of BITS bits each: BITS bytes of a packed row (4 bits: one aligned word; 2 bits: an aligned half-word).
template <int BITS> __device__ __forceinline__ uint32_t load_codes(const uint8_t* src) {
    if (BITS == 4) return __ldg(reinterpret_cast<const uint32_t*>(src));
    if (BITS == 2) return __ldg(reinterpret_cast<const uint16_t*>(src));
    if (BITS == 1) return __ldg(src);
    return uint32_t(__ldg(src)) | (uint32_t(__ldg(src + 1)) << 8) | (uint32_t(__ldg(src + 2)) << 16);
}

// Compile-time loop: f(Ic<0>{}), f(Ic<1>{}), ...
template <int I> struct Ic { static constexpr int v = I; };
template <int N, int I = 0, typename F> __device__ __forceinline__ void each(F&& f) {
    if constexpr (I < N) {
        f(Ic<I>{});
        each<N, I + 1>(f);
    }
}

// Bounded wait on a barrier of the CTA; a wait that runs out ends every other one.
struct Waiter {
    uint32_t bars; volatile uint32_t* slot; int* status;
    __device__ __forceinline__ bool operator()(int which, int phase) const {
        const uint32_t addr = bars + 8u * uint32_t(which);
        for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
            if (mbar_try(addr, uint32_t(phase & 1))) return true;
            if ((i & 1023u) == 1023u && slot[1]) return false;
        }
        slot[1] = 1u;
        atomicCAS(status, 0, ERR_WAIT);
        return false;
    }
};

// byte permute with PTX's selectors: their top bit asks for the byte's sign, eight times
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// The centroids of one width as byte planes in registers: byte k of plane p = byte p of {fp16 high part, fp16 low part} of
// centroid k.  One byte-permute then looks four codes up at once (their selectors are nibbles), two more put the bytes of a
// pair of codes together: no shared-memory lookup, and the shared-memory pipe is what bounds this kernel (an operand tile
// is 512 wavefronts of stores, a tile of results another 512; table lookups by code pairs cost 1000 more: 3.6 us per tile).
template <int BITS> struct Planes {
    static constexpr int NR = BITS == 4 ? 4 : BITS == 3 ? 2 : 1;              // registers per plane
    uint32_t t[4][NR];
    __device__ __forceinline__ void load(const uint32_t* ctab) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t a = ctab[4 * r], b = ctab[4 * r + 1], c = ctab[4 * r + 2], d = ctab[4 * r + 3];
#pragma unroll
            for (int p = 0; p < 4; ++p) t[p][r] = ((a >> (8 * p)) & 255u) | (((b >> (8 * p)) & 255u) << 8) | (((c >> (8 * p)) & 255u) << 16) | (((d >> (8 * p)) & 255u) << 24);
        }
    }
    // eight codes -> one nibble each (three bits: nothing above bit 23 is looked at)
    static __device__ __forceinline__ uint32_t nibbles(uint32_t x) {
        if (BITS == 3) {
            x = (x & 0xFFFu) | ((x << 4) & 0x0FFF0000u);
            x = (x & 0x003F003Fu) | ((x << 2) & 0x3F003F00u);
            x = (x & 0x07070707u) | ((x << 1) & 0x70707070u);
        } else if (BITS == 2) {
            x = (x | (x << 8)) & 0x00FF00FFu;
            x = (x | (x << 4)) & 0x0F0F0F0Fu;
            x = (x | (x << 2)) & 0x33333333u;
        } else if (BITS == 1) {
            x = (x | (x << 12)) & 0x000F000Fu;
            x = (x | (x << 6)) & 0x03030303u;
            x = (x | (x << 3)) & 0x11111111u;
        }
        return x;
    }
    // eight codes (x: nibbles) -> fp16 parts: planes P, P + 1
    template <int P> __device__ __forceinline__ uint4 lookup(uint32_t x) const {
        uint32_t o[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t v[2];
            const uint32_t sel = BITS == 4 ? (h ? x >> 16 : x) & 0x7777u : (h ? x >> 16 : x);
            if constexpr (BITS == 4) {
                const uint32_t m = prmt(x, x << 4, h ? 0xBFAE : 0x9D8C);          // bytes of ones where a code's top bit is set
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t a = prmt(t[P + u][0], t[P + u][NR > 1 ? 1 : 0], sel), b = prmt(t[P + u][NR > 2 ? 2 : 0], t[P + u][NR > 3 ? 3 : 0], sel);
                    v[u] = (a & ~m) | (b & m);
                }
            } else {
#pragma unroll
                for (int u = 0; u < 2; ++u) v[u] = prmt(t[P + u][0], t[P + u][NR > 1 ? 1 : 0], sel);
            }
            o[2 * h] = prmt(v[0], v[1], 0x5140);
            o[2 * h + 1] = prmt(v[0], v[1], 0x7362);
        }
        return make_uint4(o[0], o[1], o[2], o[3]);
    }
};
template <> struct Planes<0> {
    __device__ __forceinline__ void load(const uint32_t*) {}
};

// The producers.  BH / BL: bits of the first / second half of the coordinates (BL = 0: one width); warp pw takes sixteen
// rows of a tile in NK steps: a step is RP rows of one half (of the whole row), lane -> row lane / HC, chunk
// lane mod HC of eight coordinates.  Rows that sit in one cache lane are one contiguous run of bytes: a chunk's word is
// replaced by the next tile's as soon as it has been converted, so loads are in flight under the conversion.  Three-bit
// chunks (three bytes) arrive as the aligned words of the run, one per lane, and are put together with two shuffles and a
// funnel shift.  Rows that straddle cache lanes (or the end) are looked up one by one.
template <int D, int BH, int BL, bool QJL>
__device__ __forceinline__ void produce(const Params& job, unsigned char* smem, uint32_t sbase, int first, int stride, int pw, int lane, const Waiter& wait_bar) {
    using P = Plan<D>;
    constexpr int HALVES = BL ? 2 : 1, HC = D / 8 / HALVES;    // chunks of a row (of a half)
    constexpr int RP = D == 96 ? (BL ? 4 : 2) : 32 / HC, LPK = RP * HC, NK = RW / RP * HALVES;
    bool ok = true;
    uint4* s_rows = reinterpret_cast<uint4*>(smem + P::OFF_ROWS);
    const uint32_t* ctab = reinterpret_cast<const uint32_t*>(smem + P::OFF_CTAB);
    Planes<BH> tab_h;
    Planes<BL> tab_l;
    tab_h.load(ctab);
    tab_l.load(ctab + 16);
    const int n_mine = job.n_tiles > first ? (job.n_tiles - first + stride - 1) / stride : 0;
    const bool active = LPK == 32 || lane < LPK;
    const int rl0 = lane / HC, c8 = lane % HC;                 // row of the step, chunk of the half
    uint32_t w[NK], wn[NK];
    uint4 row;                                                 // norm, offset / 8, sign word, (c/d) residual norm of this lane's row
    int in_row = -1;
    bool run = false;
    const uint8_t* src[HALVES];                                // this lane's first word of either half
    uint32_t mis[HALVES];                                      // bytes between the word boundary and the run's start (three bits)
    auto setup = [&](int i) {
        const uint32_t gr = lane < RW ? uint32_t(first + i * stride) * TM + pw * RW + lane : ~0u;
        row = make_uint4(0u, ~0u, 0u, 0u);
        in_row = -1;
        if (gr < job.total) {
            const uint32_t ln = gr / job.n_rows, rw = gr - ln * job.n_rows;
            const int64_t ir = int64_t(ln) * job.in_lane_stride + rw;
            in_row = int(ir);
            row.y = uint32_t((int64_t(ln) * job.out_lane_stride + int64_t(rw) * job.out_row_stride) >> 3);
            row.x = __float_as_uint(__ldg(job.norms + ir));
            if (QJL) { row.z = __ldg(job.qjl_bits + ir); row.w = __float_as_uint(__ldg(job.qjl_gamma + ir) * (QJL_C / D)); }
            else { row.z = ln; row.w = rw; }
        }
        const int r0 = __shfl_sync(0xffffffffu, in_row, 0);
        run = __all_sync(0xffffffffu, (in_row == r0 + lane && r0 >= 0) || lane >= RW);
        if (run) {
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
                constexpr int B[2] = {BH, BL ? BL : BH};
                const uint8_t* base = h ? job.packed_lo + int64_t(r0) * job.w_lo : job.packed_hi + int64_t(r0) * job.w_hi;
                if (B[h] == 3) {
                    mis[h] = uint32_t(reinterpret_cast<uintptr_t>(base)) & 3u;
                    src[h] = base - mis[h] + (4u * lane < 3u * LPK + mis[h] ? 4 * lane : 0);       // (lanes beyond the last word repeat the first)
                } else {
                    src[h] = base + lane * B[h];
                }
            }
        }
        {   // the same rows of the tile PF_AHEAD of the CTA's tiles further on: asked for in L2 now
            const uint32_t gp = gr + uint32_t(PF_AHEAD * stride) * TM;
            if (lane < RW && gp < job.total && gp > gr) {
                const uint32_t pl = gp / job.n_rows, pr = gp - pl * job.n_rows;
                const int64_t ir = int64_t(pl) * job.in_lane_stride + pr;
                prefetch_l2(job.packed_hi + ir * job.w_hi);
                if (BL != 0) prefetch_l2(job.packed_lo + ir * job.w_lo);
                if (lane == 0 || pr == 0) prefetch_l2(job.norms + ir);
            }
        }
    };
    // step k: half k mod HALVES, rows (k / HALVES) RP ...; a step's rows of w bytes follow one another
    auto load_run = [&](auto kc) -> uint32_t {
        constexpr int k = decltype(kc)::v, h = HALVES == 2 ? k & 1 : 0, B = h ? BL : BH;
        const uint8_t* x = src[h] + (k / HALVES) * (LPK * B);
        if constexpr (B == 3) return __ldg(reinterpret_cast<const uint32_t*>(x));
        else return load_codes<B>(x);
    };
    auto load_row = [&](auto kc, int ir) -> uint32_t {         // (rows of several cache lanes; ir: this lane's row, or -1)
        constexpr int k = decltype(kc)::v, h = HALVES == 2 ? k & 1 : 0, B = h ? BL : BH;
        const int r = __shfl_sync(0xffffffffu, ir, min(rl0 + (k / HALVES) * RP, RW - 1));
        if (r < 0 || !active) return 0u;
        return load_codes<B>((h ? job.packed_lo + int64_t(r) * job.w_lo : job.packed_hi + int64_t(r) * job.w_hi) + c8 * B);
    };
    if (n_mine > 0) {
        setup(0);
        if (run && active) each<NK>([&](auto kc) { w[decltype(kc)::v] = load_run(kc); });
    }
    for (int it = 0; it < n_mine; ++it) {
        const int sub = it * 2;
        const uint4 row_cur = row;
        const int row_in = in_row;
        const bool run_cur = run, more = it + 1 < n_mine;
        uint32_t mis_cur[HALVES];
#pragma unroll
        for (int h = 0; h < HALVES; ++h) mis_cur[h] = mis[h];
        if (more) setup(it + 1);
        if (more && run && active) each<NK>([&](auto kc) { wn[decltype(kc)::v] = load_run(kc); });
        // one pass writes the high and the low parts when the ring has room for both, else a pass each
        constexpr bool ONE_PASS = P::NB > 1;
        for (int part = 0; part < 2; part += ONE_PASS ? 2 : 1) {
            const int n0 = sub + part, bf = n0 % P::NB, bf2 = (n0 + 1) % P::NB;
            if (n0 / P::NB > 0) ok = wait_bar(A_FREE + bf, n0 / P::NB - 1);        // the products that read the buffer's previous tile have completed
            if (ok && ONE_PASS && (n0 + 1) / P::NB > 0) ok = wait_bar(A_FREE + bf2, (n0 + 1) / P::NB - 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            // (the products of tile it - 4 or a later one have completed; they could start only after the rows of tile it - 6 had been
            // written out, so the slot's previous tenant has left)
            if (part == 0 && lane < RW) s_rows[(it % SLOTS) * TM + pw * RW + lane] = row_cur;
            int row_o = pw * RW + rl0;                         // (opaque: offsets kept across tiles would not fit the registers)
            asm volatile("" : "+r"(row_o));
            unsigned char* a = smem + P::OFF_A + bf * P::A_TILE + row_o * 128;
            const int a2 = (bf2 - bf) * int(P::A_TILE);
            each<NK>([&](auto kc) {
                constexpr int k = decltype(kc)::v, h = HALVES == 2 ? k & 1 : 0, B = h ? BL : BH, R = (k / HALVES) * RP;
                uint32_t x = w[k];
                if (!run_cur) x = load_row(kc, row_in);
                else if constexpr (B == 3) {
                    const uint32_t off = 3u * lane + mis_cur[h];
                    const uint32_t lo = __shfl_sync(0xffffffffu, w[k], off >> 2), hi = __shfl_sync(0xffffffffu, w[k], min((off >> 2) + 1u, 31u));
                    x = __funnelshift_r(lo, hi, (off & 3u) * 8u);
                }
                x = Planes<B>::nibbles(x);
                const int j8 = h * HC + c8;
                unsigned char* d = a + (j8 >> 3) * P::ABLK + R * 128 + (uint32_t((j8 & 7) ^ ((row_o + R) & 7)) << 4);
                auto put = [&](const auto& tab) {
                    if (ONE_PASS || part == 0) {
                        const uint4 hi = tab.template lookup<0>(x);
                        if (active) *reinterpret_cast<uint4*>(d) = hi;
                    }
                    if (ONE_PASS || part == 1) {
                        const uint4 lo = tab.template lookup<2>(x);
                        if (active) *reinterpret_cast<uint4*>(ONE_PASS ? d + a2 : d) = lo;
                    }
                };
                if constexpr (h == 1) put(tab_l);
                else put(tab_h);
            });
            fence_proxy_async();
            mbar_arrive(sbase + P::OFF_BAR + 8u * (A_FULL + bf));
            if (ONE_PASS) mbar_arrive(sbase + P::OFF_BAR + 8u * (A_FULL + bf2));
        }
#pragma unroll
        for (int k = 0; k < NK; ++k) w[k] = wn[k];
    }
}

template <int D, int BH, int BL, bool QJL>
__global__ void __launch_bounds__(NT, 1) dequantize_tc_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap omap) {
    using P = Plan<D>;
    constexpr int NC = P::NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t raw_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    const uint32_t sbase = (raw_addr + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (sbase - raw_addr);
    volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(smem + P::OFF_SLOT);
    auto bar = [&](int which) -> uint32_t { return sbase + P::OFF_BAR + 8u * uint32_t(which); };
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // (warp: uniform)
    // d = 256: CTAs with an even number own output columns 0 .. 127, the others 128 .. 255 of the same tiles
    constexpr int SPLIT = D == 256 ? 2 : 1;
    const int first = blockIdx.x / SPLIT, stride = gridDim.x / SPLIT, col_base = (blockIdx.x % SPLIT) * NC;
    if (p.follows) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---------------- set-up: barriers, tensor memory, centroid tables, R as two fp16 B tiles, S ------------------------
    if (tid == 0) {
        for (int i = 0; i < P::NB; ++i) { mbar_init(bar(A_FULL + i), PROD_T); mbar_init(bar(A_FREE + i), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(bar(ACC_FULL + i), 1); mbar_init(bar(ACC_FREE + i), EPI_T); }
        mbar_init(bar(DRAIN), 1);
        fence_barrier_init();
        slot[1] = 0u;
    }
    if (warp == MMA_W) {
        tmem_alloc(sbase + P::OFF_SLOT, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid < 32) {
        const int which = (tid >> 4) & 1, k = tid & 15;
        const float* src = which ? p.cent_lo : p.cent_hi;
        const int bits = which ? p.bits_lo : p.bits_hi;
        float c = 0.f;
        if (src != nullptr && bits > 0 && k < (1 << bits)) c = src[k];
        const __half hi = __float2half_rn(c);
        const __half lo = __float2half_rn((c - __half2float(hi)) * 2048.f);
        reinterpret_cast<uint32_t*>(smem + P::OFF_CTAB)[tid] = uint32_t(__half_as_ushort(hi)) | (uint32_t(__half_as_ushort(lo)) << 16);
    }
    for (int i = tid; i < D * (NC / 8); i += NT) {                           // chunk (row k, columns 8 c .. 8 c + 7) of this CTA's columns of R
        const int k = i / (NC / 8), c = i - k * (NC / 8);
        uint32_t hi[4] = {0u, 0u, 0u, 0u}, lo[4] = {0u, 0u, 0u, 0u};
        if (col_base + c * 8 < D) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(p.rot + k * D + col_base + c * 8));
            const float4 b = __ldg(reinterpret_cast<const float4*>(p.rot + k * D + col_base + c * 8 + 4));
            const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const __half2 h = __floats2half2_rn(x[2 * u], x[2 * u + 1]);
                const float2 hf = __half22float2(h);
                hi[u] = *reinterpret_cast<const uint32_t*>(&h);
                lo[u] = h2_bits((x[2 * u] - hf.x) * 2048.f, (x[2 * u + 1] - hf.y) * 2048.f);
            }
        }
        *reinterpret_cast<uint4*>(smem + P::OFF_R + chunk_off(P::RBLK, k, c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(smem + P::OFF_R + P::R_TILE + chunk_off(P::RBLK, k, c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    if constexpr (QJL) {
        // k slot (ks, register h, half e) of thread t stands for sketch row 4 t + 2 ks + h + 16 e: the halves of an operand
        // register are then bits 16 apart in a token's sign word
        uint2* sf = reinterpret_cast<uint2*>(smem + P::OFF_S);
        for (int i = tid; i < 2 * (NC / 8) * 32; i += NT) {
            const int ks = i / ((NC / 8) * 32), nt = i / 32 % (NC / 8), ln = i & 31, col = col_base + nt * 8 + (ln >> 2);
            uint32_t hw[2] = {0u, 0u}, lw[2] = {0u, 0u};
            if (col < D) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = 4 * (ln & 3) + 2 * ks + h;
                    const float x0 = __ldg(p.qjl_proj + r * D + col), x1 = __ldg(p.qjl_proj + (r + 16) * D + col);
                    const __half2 hh = __floats2half2_rn(x0, x1);
                    const float2 hf = __half22float2(hh);
                    hw[h] = *reinterpret_cast<const uint32_t*>(&hh);
                    lw[h] = h2_bits(x0 - hf.x, x1 - hf.y);
                }
            }
            sf[((ks * (NC / 8) + nt) * 2 + 0) * 32 + ln] = make_uint2(hw[0], hw[1]);
            sf[((ks * (NC / 8) + nt) * 2 + 1) * 32 + ln] = make_uint2(lw[0], lw[1]);
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!p.follows) {          // the set-up read constants only; the second job may start once everything before this one has ended
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, slot[0], 0);

    const Waiter wait_bar{sbase + P::OFF_BAR, slot, p.status};
    const int n_mine = p.n_tiles > first ? (p.n_tiles - first + stride - 1) / stride : 0;

    if (warp == MMA_W) {
        // ======================= MMA issue: one warp, uniform =======================
        {
            auto wait_all = [&](int which, int phase) { return bool(__all_sync(0xffffffffu, wait_bar(which, phase))); };
            bool ok = true;
            for (int it = 0; it < n_mine && ok; ++it) {
                const int st = it & 1;
                const uint32_t acc = tmem_base + uint32_t(st) * 256u;
                if (it >= 2) ok = wait_all(ACC_FREE + st, (it >> 1) - 1);
                for (int part = 0; part < 2 && ok; ++part) {
                    const int s = it * 2 + part, bf = s % P::NB;
                    ok = wait_all(A_FULL + bf, s / P::NB);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = sbase + P::OFF_A + bf * P::A_TILE;
                    // high parts: [R_hi | R_lo] as one operand of 2 NC columns; low parts join the second accumulator
                    for (int ks = 0; ks < D / 16; ++ks) {
                        if (part == 0) umma_f16(acc, desc_kmajor(a, P::ABLK, ks), desc_mnmajor(sbase + P::OFF_R, P::RBLK, ks), idesc_of(2 * NC), ks > 0 ? 1u : 0u);
                        else umma_f16(acc + NC, desc_kmajor(a, P::ABLK, ks), desc_mnmajor(sbase + P::OFF_R, P::RBLK, ks), idesc_of(NC), 1u);
                    }
                    umma_commit(bar(A_FREE + bf));
                }
                if (ok) umma_commit(bar(ACC_FULL + st));
            }
            if (!ok) {             // a wait ran out: the products in flight end (bounded) before their memory is given up
                umma_commit(bar(DRAIN));
                for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try(bar(DRAIN), 0); ++i) {}
            }
        }
        __syncwarp();
    } else if (warp >= 8) {
        produce<D, BH, BL, QJL>(p, smem, sbase, first, stride, warp - 8, lane, wait_bar);
    } else if constexpr (QJL) {
        // ======================= epilogue with the sketch correction: registers in mma.sync fragment layout =======================
        const int grp = warp >> 2, g = lane >> 2, t = lane & 3;
        const uint4* s_rows = reinterpret_cast<const uint4*>(smem + P::OFF_ROWS);
        const uint2* sf = reinterpret_cast<const uint2*>(smem + P::OFF_S) + lane;
        const int es = p.out_dtype == TQ_F32 ? 4 : 2;
        for (int it = grp; it < n_mine; it += 2) {
            const int st = it & 1;
            if (!__all_sync(0xffffffffu, wait_bar(ACC_FULL + st, it >> 1))) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + (uint32_t((warp & 3) * 32) << 16) + uint32_t(st) * 256u;
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {                      // sixteen rows at a time: rows g and g + 8 of them
                const int r = (it % SLOTS) * TM + (warp & 3) * 32 + 16 * h + g;
                const uint4 ra = s_rows[r], rb = s_rows[r + 8];
                const float na = __uint_as_float(ra.x), nb = __uint_as_float(rb.x);
                const float ga = __uint_as_float(ra.w), gb = __uint_as_float(rb.w);
                unsigned char* oa = static_cast<unsigned char*>(p.out) + (int64_t(ra.y) * 8 + col_base + 2 * t) * es;
                unsigned char* ob = static_cast<unsigned char*>(p.out) + (int64_t(rb.y) * 8 + col_base + 2 * t) * es;
                uint32_t az[2][4];
                if (QJL) {
                    const uint32_t za = ra.z << (12 - 4 * t), zb = rb.z << (12 - 4 * t);
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
                        az[ks][0] = sign_pair16(za << (3 - 2 * ks)); az[ks][1] = sign_pair16(zb << (3 - 2 * ks));
                        az[ks][2] = sign_pair16(za << (2 - 2 * ks)); az[ks][3] = sign_pair16(zb << (2 - 2 * ks));
                    }
                }
#pragma unroll 1
                for (int c0 = 0; c0 < NC; c0 += 64) {
                    uint32_t hi[32], lo[32];
                    tmem_ld_frag64(acc + (uint32_t(16 * h) << 16) + c0, hi);
                    tmem_ld_frag64(acc + (uint32_t(16 * h) << 16) + NC + c0, lo);
                    tmem_ld_wait();
#pragma unroll
                    for (int b = 0; b < 8; ++b) {              // eight columns: this lane has two of them in either row
                        const int col = c0 + 8 * b;
                        if (D == 96 && col >= 96) break;
                        float v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            v[u] = fmaf(__uint_as_float(lo[4 * b + u]), 1.f / 2048.f, __uint_as_float(hi[4 * b + u])) * (u < 2 ? na : nb);
                        if (QJL) {
                            float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                            for (int ks = 0; ks < 2; ++ks) {
                                const uint2* f = sf + (ks * (NC / 8) + (c0 / 8 + b)) * 64;
                                mma16816(z, az[ks], f[0]);
                                mma16816(z, az[ks], f[32]);
                            }
                            v[0] = fmaf(ga, z[0], v[0]); v[1] = fmaf(ga, z[1], v[1]);
                            v[2] = fmaf(gb, z[2], v[2]); v[3] = fmaf(gb, z[3], v[3]);
                        }
                        if (es == 4) {
                            if (ra.y != ~0u) *reinterpret_cast<float2*>(oa + col * 4) = make_float2(v[0], v[1]);
                            if (rb.y != ~0u) *reinterpret_cast<float2*>(ob + col * 4) = make_float2(v[2], v[3]);
                        } else {
                            uint32_t wa, wb;
                            if (p.out_dtype == TQ_F16) { wa = h2_bits(v[0], v[1]); wb = h2_bits(v[2], v[3]); }
                            else {
                                const __nv_bfloat162 x = __floats2bfloat162_rn(v[0], v[1]), y = __floats2bfloat162_rn(v[2], v[3]);
                                wa = *reinterpret_cast<const uint32_t*>(&x); wb = *reinterpret_cast<const uint32_t*>(&y);
                            }
                            if (ra.y != ~0u) *reinterpret_cast<uint32_t*>(oa + col * 2) = wa;
                            if (rb.y != ~0u) *reinterpret_cast<uint32_t*>(ob + col * 2) = wb;
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(bar(ACC_FREE + st));
        }
    } else {
        // ======================= epilogue: a row per thread; combine, scale, stage, store =======================
        // Sixteen float32 (32 sixteen-bit) columns at a time go to the warp's staging buffer (32 rows of 64 bytes, 64-byte
        // swizzle) and leave with one tiled bulk store; rows of several cache lanes are stored directly.
        const int grp = warp >> 2;
        const uint4* s_rows = reinterpret_cast<const uint4*>(smem + P::OFF_ROWS);
        const bool f32 = p.out_dtype == TQ_F32;
        const int es = f32 ? 4 : 2;
        constexpr int NBUF = P::STG / 2048;
        int n_st = 0;                                          // bulk stores of this warp so far
        for (int it = grp; it < n_mine; it += 2) {
            const int st = it & 1;
            if (!__all_sync(0xffffffffu, wait_bar(ACC_FULL + st, it >> 1))) break;
            tc_fence_after();
            const uint4 row = s_rows[(it % SLOTS) * TM + (warp & 3) * 32 + lane];
            const float nrm = __uint_as_float(row.x);
            const uint32_t ln0 = __shfl_sync(0xffffffffu, row.z, 0), rw0 = __shfl_sync(0xffffffffu, row.w, 0);
            // one box of the tensor map: the valid rows follow one another in one cache lane (rows past the lane's end are clipped)
            const bool box = __all_sync(0xffffffffu, row.y == ~0u ? lane > 0 : (row.z == ln0 && row.w == rw0 + lane));
            const uint32_t acc = tmem_base + (uint32_t((warp & 3) * 32) << 16) + uint32_t(st) * 256u;
            unsigned char* out = static_cast<unsigned char*>(p.out) + (int64_t(row.y) * 8 + col_base) * es;
            constexpr int NCOLS = D == 96 ? 96 : NC;
            auto leave = [&](int c0, const uint4 (&q)[4]) {    // 64 bytes of this thread's row, from column c0 on
                if (box) {
                    const uint32_t buf = sbase + P::OFF_S + warp * P::STG + uint32_t(n_st % NBUF) * 2048u;
                    if (lane == 0) {
                        if (NBUF == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(smem + (buf - sbase) + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = q[c];
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
                                     ::"l"(reinterpret_cast<uint64_t>(&omap)), "r"(col_base + c0), "r"(int(rw0)), "r"(int(ln0)), "r"(buf) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    ++n_st;
                } else if (row.y != ~0u) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(out + c0 * es + 16 * c) = q[c];
                }
            };
            if (f32) {
#pragma unroll 1
                for (int c0 = 0; c0 < NCOLS; c0 += 16) {
                    uint32_t hi[16], lo[16];
                    tmem_ld16(acc + c0, hi);
                    tmem_ld16(acc + NC + c0, lo);
                    tmem_ld_wait();
                    uint4 q[4];
#pragma unroll
                    for (int i = 0; i < 16; ++i) hi[i] = __float_as_uint(fmaf(__uint_as_float(lo[i]), 1.f / 2048.f, __uint_as_float(hi[i])) * nrm);
#pragma unroll
                    for (int c = 0; c < 4; ++c) q[c] = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                    leave(c0, q);
                }
            } else {
                const bool f16 = p.out_dtype == TQ_F16;
#pragma unroll 1
                for (int c0 = 0; c0 < NCOLS; c0 += 32) {
                    uint32_t hi[32], lo[32];
                    tmem_ld32(acc + c0, hi);
                    tmem_ld32(acc + NC + c0, lo);
                    tmem_ld_wait();
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float x = fmaf(__uint_as_float(lo[2 * i]), 1.f / 2048.f, __uint_as_float(hi[2 * i])) * nrm;
                        const float y = fmaf(__uint_as_float(lo[2 * i + 1]), 1.f / 2048.f, __uint_as_float(hi[2 * i + 1])) * nrm;
                        if (f16) w[i] = h2_bits(x, y);
                        else {
                            const __nv_bfloat162 bb = __floats2bfloat162_rn(x, y);
                            w[i] = *reinterpret_cast<const uint32_t*>(&bb);
                        }
                    }
                    uint4 q[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) q[c] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
                    leave(c0, q);
                }
            }
            tc_fence_before();
            mbar_arrive(bar(ACC_FREE + st));
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // nothing may read this CTA's memory after it has gone
    }
    // ---------------- teardown: every loop above is bounded, so every thread gets here ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_W) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (p.follows) asm volatile("griddepcontrol.wait;" ::: "memory");
}

using Kernel = void (*)(Params, CUtensorMap);
// The kernel for a pair of widths (bits_lo 0: one width), or null.  One translation unit per head_dim.
template <int D> Kernel kernel_of(int bits_hi, int bits_lo, bool qjl);
#define TQ_DEQUANTIZE_KERNELS(D) \
    namespace tq { namespace dqtc { \
    template <> Kernel kernel_of<D>(int bits_hi, int bits_lo, bool qjl) { \
        switch (bits_hi * 8 + bits_lo) { \
            case 8: return qjl ? dequantize_tc_kernel<D, 1, 0, true> : dequantize_tc_kernel<D, 1, 0, false>; \
            case 16: return qjl ? dequantize_tc_kernel<D, 2, 0, true> : dequantize_tc_kernel<D, 2, 0, false>; \
            case 24: return qjl ? dequantize_tc_kernel<D, 3, 0, true> : dequantize_tc_kernel<D, 3, 0, false>; \
            case 32: return qjl ? dequantize_tc_kernel<D, 4, 0, true> : dequantize_tc_kernel<D, 4, 0, false>; \
            case 17: return qjl ? dequantize_tc_kernel<D, 2, 1, true> : dequantize_tc_kernel<D, 2, 1, false>; \
            case 26: return qjl ? dequantize_tc_kernel<D, 3, 2, true> : dequantize_tc_kernel<D, 3, 2, false>; \
            case 35: return qjl ? dequantize_tc_kernel<D, 4, 3, true> : dequantize_tc_kernel<D, 4, 3, false>; \
            default: return nullptr; \
        } \
    } \
    } }

}  // namespace dqtc
}  // namespace tq
