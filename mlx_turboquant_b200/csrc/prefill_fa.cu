// Causal attention for several query tokens per sequence over the compressed cache, in two steps: the cache's tokens are
// expanded ONCE per call into fp16 rows in workspace memory (positions in order: sink, packed, recent), then a plain
// flash-attention kernel on the fifth-generation tensor cores reads those rows through TMA for every block of queries.
// Same contract and arithmetic as prefill_tc.cu / prefill.cu (what the reference does as dense reassembly, cache.py:674-706,
// followed by the consumer's masked attention).
//
// Why a pre-pass: with the unpacking inside the attention kernel every block of 128 query rows turned the same codes into
// the same operands again, and the table lookups shared the shared-memory pipe with the softmax (3 us per 128 x 128 tile
// against 0.77 us of tensor-core time; 15 us at widths without whole-byte tables).  A row costs 2 d bytes of writes once and
// is then read from L2 by every block.
//
// An expanded row is the UNIT vector c @ R of the token in fp16 and its norm stays float32 beside it (uncompressed tokens:
// the row itself under a power-of-two scale), so no magnitude is lost: scores take the key norm as a multiply-add, the
// softmax weights take the value norm before they become fp16, as in the other kernels.
//
// fa_kernel: a CTA owns NQ (2; 1 at d = 256) tiles of 128 rows = 128 / GP query tokens x the GP query heads of a GQA group, and a
// range of key tiles (TN tokens each):
//   * 4 NQ softmax warps, a row per thread: tcgen05.ld of the row's TN scores into registers, one multiply-add each
//     (packed in pairs), maximum, ex2, P (fp16) back into tensor memory over the scores it came from;
//   * one warp issues S = Q K^T (both operands in shared memory) and O += P V (P from tensor memory), the tiles of the two
//     query blocks alternating so that one block's softmax runs under the other's products;
//   * one thread each keeps four key tiles (and eight tiles' norms) and four value tiles in flight (tiled TMA, bulk copies); scores
//     are two key tiles ahead of the softmax.
//   512 queries x 32 lanes over 16,384 tokens at d = 128: 675 us = 800 TFLOP/s (350 with the unpacking inside the kernel); the tensor
//   pipe is 51 % busy, the rest is the softmax's latency and shared memory (operand reads of the products, norms).
// When there are too few query blocks for the device, the key tiles of a block are split over several CTAs, which leave
// float32 partials that fa_merge_kernel combines.
//
// Every mbarrier wait is bounded; a wait that runs out leaves status 111 (tq_device_status) and raises a flag that ends
// every other wait; tensor memory is freed on every path.
#include <algorithm>
#include <atomic>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "decode_dev.cuh"

namespace tq {

int* decode_status_ptr();

namespace fa {

constexpr uint32_t WAIT_LIMIT = 4u << 20;
constexpr int ERR_WAIT = 111;
constexpr int TM = 128, NSC = 8;                       // rows per query tile, tiles' norms in flight

template <int D> struct Plan {
    static constexpr int NQ = D == 256 ? 1 : 2;        // query tiles per CTA
    static constexpr int TN = 64;                      // tokens per key tile
    static constexpr int SB = 2;                       // score buffers per query tile
    static constexpr int ST = D == 256 ? 2 : 4;        // key tiles (and value tiles) in flight
    static constexpr int NBLK = (D + 63) / 64;         // 64-column blocks of a row
    static constexpr int DP = NBLK * 64;               // columns of O (d = 96: the last 32 are zeros)
    static constexpr int NT = NQ * 128 + 96;           // softmax warps, MMA warp, a TMA warp for keys and norms, one for values
    static constexpr uint32_t QBLK = TM * 128u, KBLK = TN * 128u;            // bytes of a 64-column block
    static constexpr uint32_t Q_TILE = NBLK * QBLK, K_TILE = NBLK * KBLK;
    static constexpr uint32_t OFF_Q = 0, OFF_K = NQ * Q_TILE, OFF_V = OFF_K + ST * K_TILE;
    static constexpr uint32_t OFF_SC = OFF_V + ST * K_TILE;                  // float [NSC][2][TN]: key norms, value norms
    static constexpr uint32_t OFF_BAR = OFF_SC + NSC * 2 * TN * 4;
    static constexpr uint32_t OFF_SLOT = OFF_BAR + 368;                      // [0] tensor-memory base, [1] abort
    static constexpr size_t NEED = OFF_SLOT + 16 + 1024, SMEM = NEED > 116 * 1024 ? NEED : 116 * 1024;      // one CTA per SM: it takes all of the tensor memory
    static constexpr uint32_t COL_O = NQ * SB * TN;                          // scores first, then the accumulators
    static_assert(COL_O + NQ * DP <= 512, "tensor memory");
    static_assert(SMEM <= 227 * 1024, "shared memory");
};
enum Bars { K_FULL = 0, K_FREE = 4, V_FULL = 8, V_FREE = 12, SC_FULL = 16, SC_FREE = 24, S_FULL = 32, P_FULL = 36, O_DONE = 40, ALL_DONE = 42, DRAIN = 44 };       // (45 of 8 bytes)

struct Params {
    const void* q; int q_dtype; float f;               // scale * log2(e)
    void* out; int out_dtype;
    int Hq, Hkv, G, HG, GP, QT, Tq;                    // QT: query tokens per query tile
    int lane0;                                         // first cache lane of this launch
    int q_pos0, total;                                 // position of query token 0, tokens per lane
    const float *kn, *vn; int ts;                      // norms (lane, ts), ts a multiple of 128
    int n_splits;
    float* part;                                       // (row block, split, NQ * 128 rows, D + 4)
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
// them there and one elected lane issues; with a single thread in a divergent branch every operand is moved over one by one
// (70 cycles per instruction: the issuing thread, not the products, was what the softmax warps waited for).
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
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
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
__global__ void __launch_bounds__(Plan<D>::NT, 1) fa_kernel(Params p, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
    using P = Plan<D>;
    constexpr int NQ = P::NQ, TN = P::TN, DP = P::DP, NT = P::NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t raw_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    const uint32_t sbase = (raw_addr + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (sbase - raw_addr);
    volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(smem + P::OFF_SLOT);
    auto bar = [&](int which) -> uint32_t { return sbase + P::OFF_BAR + 8u * uint32_t(which); };
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // (uniform)

    // blockIdx.x = row block x split, the latest query rows (the longest runs of tiles) first
    const int n_blocks = gridDim.x / p.n_splits, split = blockIdx.x % p.n_splits, blk = n_blocks - 1 - int(blockIdx.x) / p.n_splits;
    const int lane_c = blockIdx.y / p.HG, hg = blockIdx.y - lane_c * p.HG, gl = p.lane0 + lane_c;
    const int b = gl / p.Hkv, hkv = gl - b * p.Hkv;
    const int heads_here = min(HPG, p.G - hg * HPG);
    const int tq0 = blk * NQ * p.QT, GP = p.GP;
    auto row_token = [&](int m) { return tq0 + (m >> 7) * p.QT + (m & 127) / GP; };
    auto row_valid = [&](int m) { return (m & 127) % GP < heads_here && row_token(m) < p.Tq; };
    auto row_q_index = [&](int m) -> int64_t {
        const int h = hkv * p.G + hg * HPG + (m & 127) % GP;
        return ((int64_t(b) * p.Hq + h) * p.Tq + row_token(m)) * D;
    };
    // key tiles of this CTA: its share of those that some row of it sees
    const int vis = p.q_pos0 + min(tq0 + NQ * p.QT, p.Tq);
    const int n_all = (vis + TN - 1) / TN, per = (n_all + p.n_splits - 1) / p.n_splits;
    const int t_lo = split * per, n = max(0, min(t_lo + per, n_all) - t_lo);

    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(bar(K_FULL + i), 1); mbar_init(bar(K_FREE + i), 1); mbar_init(bar(V_FULL + i), 1); mbar_init(bar(V_FREE + i), 1);
            mbar_init(bar(S_FULL + i), 1); mbar_init(bar(P_FULL + i), 128);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(bar(O_DONE + i), 1); mbar_init(bar(ALL_DONE + i), 1); }
        mbar_init(bar(DRAIN), 1);
        for (int i = 0; i < NSC; ++i) { mbar_init(bar(SC_FULL + i), 1); mbar_init(bar(SC_FREE + i), NQ * 128); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        slot[1] = 0u;
    }
    if (warp == NQ * 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + P::OFF_SLOT), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the query tiles, scaled, as fp16 A operands
    for (int i = tid; i < NQ * TM * (P::NBLK * 8); i += NT) {
        const int m = i / (P::NBLK * 8), c = i - m * (P::NBLK * 8);          // 16-byte chunk c of row m
        uint32_t h[4] = {0u, 0u, 0u, 0u};
        if (c * 8 < D && row_valid(m)) {
            const int64_t e = row_q_index(m) + c * 8;
#pragma unroll
            for (int u = 0; u < 4; ++u) h[u] = pack_h2(load_as_f32(p.q, p.q_dtype, e + 2 * u) * p.f, load_as_f32(p.q, p.q_dtype, e + 2 * u + 1) * p.f);
        }
        const int r = m & 127;
        *reinterpret_cast<uint4*>(smem + P::OFF_Q + (m >> 7) * P::Q_TILE + (c >> 3) * P::QBLK + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
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

    if (warp == NQ * 4 + 1) {
        // ======================= keys and norms: one thread (a key tile is free as soon as its scores are computed, long before =====
        // ======================= the value tile: each of the two rings is kept full by a thread of its own) =======================
        if (lane == 0) {
            const float* kn = p.kn + int64_t(lane_c) * p.ts;
            const float* vn = p.vn + int64_t(lane_c) * p.ts;
            int nk = 0, nsc = 0;                                   // copies asked for so far
            for (int j = 0; j < n; ++j) {
                const int row = (t_lo + j) * TN, s = j % NSC, st = j % ST;
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
            for (int j = max(0, nk - ST); j < nk; ++j) drain(K_FULL + j % ST, j / ST);
            for (int j = max(0, nsc - NSC); j < nsc; ++j) drain(SC_FULL + j % NSC, j / NSC);
        }
        __syncwarp();
    } else if (warp == NQ * 4 + 2) {
        // ======================= values: one thread =======================
        if (lane == 0) {
            int nv = 0;
            for (int j = 0; j < n; ++j) {
                const int row = (t_lo + j) * TN, st = j % ST;
                if (j >= ST && !wait_bar(V_FREE + st, j / ST - 1)) break;
                nv = j + 1;
                mbar_expect_tx(bar(V_FULL + st), P::K_TILE);
                for (int x = 0; x < P::NBLK; ++x) tma_load_3d(sbase + P::OFF_V + st * P::K_TILE + x * P::KBLK, &vmap, x * 64, row, lane_c, bar(V_FULL + st));
            }
            for (int j = max(0, nv - ST); j < nv; ++j) drain(V_FULL + j % ST, j / ST);
        }
        __syncwarp();
    } else if (warp == NQ * 4) {
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
                if (j == n - 1) umma_commit(bar(ALL_DONE + q));    // (a barrier of its own: a parity wait on O_DONE could be two phases early or one late)
            };
            auto wait_all = [&](int which, int phase) -> bool { return __all_sync(0xffffffffu, wait_bar(which, phase)); };
            bool ok = true;
            for (int j = 0; j < min(n, SB) && ok; ++j) {
                ok = wait_all(K_FULL + j % ST, 0);
                if (!ok) break;
                tc_fence_after();
                for (int q = 0; q < NQ; ++q) issue_qk(q, j);
                umma_commit(bar(K_FREE + j % ST));
            }
            for (int j = 0; j < n && ok; ++j) {
                ok = wait_all(V_FULL + j % ST, j / ST);
                const int jn = j + SB;                             // the key tile whose scores go where P of tile j sits now
                for (int q = 0; q < NQ && ok; ++q) {
                    ok = wait_all(P_FULL + sbuf(q, j), sph(j));
                    if (!ok) break;
                    tc_fence_after();
                    issue_pv(q, j);
                    if (q == NQ - 1) umma_commit(bar(V_FREE + j % ST));
                    if (jn < n) {                                  // (the tensor core takes one thread's products in order)
                        if (q == 0) ok = wait_all(K_FULL + jn % ST, jn / ST);
                        if (!ok) break;
                        issue_qk(q, jn);
                        if (q == NQ - 1) umma_commit(bar(K_FREE + jn % ST));
                    }
                }
            }
            if (!ok) { umma_commit(bar(DRAIN)); drain(DRAIN, 0); }
        }
        __syncwarp();
    } else {
        // ======================= softmax: a row per thread =======================
        const int q = warp >> 2, m = tid;                          // (rows of query tile q: threads 128 q ... )
        const uint32_t t_row = tmem + (uint32_t((warp & 3) * 32) << 16);
        const bool valid = row_valid(m);
        const int q_pos = valid ? p.q_pos0 + row_token(m) : -1;    // the latest position this row sees
        const int full_upto = p.q_pos0 + tq0 + q * p.QT;           // positions every row of the query tile sees
        float m_ref = -1e30f, vsc = 1.f, vthr = 0.f;               // (vthr 0: the first tile with a non-zero value norm picks the scale)
        float lvsc = 0.f, bias = 0.f, t_thr = -INFINITY;           // log2(vsc); lvsc - m_ref (0 before the first tile); MAX_SLACK + lvsc
        u64 l2a = pk(0.f, 0.f), l2b = l2a;
        bool ok = true;
        for (int j = 0; j < n; ++j) {
            const int s = j % NSC, base = (t_lo + j) * TN;
            ok = wait_bar(SC_FULL + s, j / NSC) && wait_bar(S_FULL + sbuf(q, j), sph(j));
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
            const float* kn = reinterpret_cast<const float*>(smem + P::OFF_SC) + s * 2 * TN;
            const float* vn = kn + TN;
            const uint32_t s_col = t_row + sbuf(q, j) * TN;
            uint32_t v[TN];
#pragma unroll
            for (int i = 0; i < TN / 32; ++i) tmem_ld32(s_col + 32 * i, v + 32 * i);
            float vmax = 0.f;
#pragma unroll
            for (int i = 0; i < TN / 32; ++i) vmax = fmaxf(vmax, vn[lane + 32 * i]);
#pragma unroll
            for (int off = 16; off; off >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
            tmem_ld_wait();
            // t = score * key norm - reference + log2(value scale)
            const u64 bias2 = pk(bias, bias);
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < TN; i += 4) {
                const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(kn + i);
                const u64 a = fma2(pk(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), k4.x, bias2);
                const u64 c = fma2(pk(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), k4.y, bias2);
                float x0, x1, x2, x3;
                upk(a, x0, x1); upk(c, x2, x3);
                v[i] = __float_as_uint(x0); v[i + 1] = __float_as_uint(x1); v[i + 2] = __float_as_uint(x2); v[i + 3] = __float_as_uint(x3);
            }
            if (base + TN > full_upto + 1) {                       // some token of the tile is hidden from some row, or past the end
                const int lim = q_pos - base;
#pragma unroll
                for (int i = 0; i < TN; ++i) v[i] = i <= lim ? v[i] : 0xff800000u;
            }
#pragma unroll
            for (int i = 0; i < TN; i += 2) mx = fmaxf(fmaxf(mx, __uint_as_float(v[i])), __uint_as_float(v[i + 1]));
            // Reference maximum / value scale: refreshed for the whole warp when any row needs it (rare after the first tile):
            // the row's sums and its O in tensor memory are rescaled.
            if (__any_sync(0xffffffffu, mx > t_thr || vmax > vthr)) {
                const float mn = fmaxf(fmaxf(m_ref, mx - bias), -1e30f);
                float a = ex2(m_ref - mn);
                m_ref = mn;
                if (vmax > vthr) {
                    int eb = (__float_as_int(vmax) >> 23) & 0xff;
                    eb = min(max(eb, 16), 240);
                    const float nsc = __int_as_float((261 - eb) << 23);    // the largest value norm lands in [128, 256)
                    a *= nsc / vsc;
                    vsc = nsc;
                    vthr = VSC_CAP / nsc;
                    lvsc = float(134 - eb);
                }
                const float nb = lvsc - m_ref, delta = nb - bias;
                bias = nb;
                t_thr = MAX_SLACK + lvsc;
                const u64 a2 = pk(a, a);
                l2a = mul2(l2a, a2); l2b = mul2(l2b, a2);
#pragma unroll
                for (int i = 0; i < TN; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + delta);
                if (j > 0) {
                    ok = wait_bar(O_DONE + q, j - 1);
                    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c0 = 0; c0 < DP; c0 += 32) {
                        uint32_t o[32];
                        tmem_ld32(t_row + P::COL_O + q * DP + c0, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * a);
                        tmem_st32(t_row + P::COL_O + q * DP + c0, o);
                    }
                    tmem_st_wait();
                }
            }
            // weights, their sum, P = weight * value norm (both carry the value scale) as fp16 over the scores
#pragma unroll
            for (int h = 0; h < TN / 64; ++h) {
                uint32_t w[32];
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    const int e = 64 * h + i;
                    const ulonglong2 n4 = *reinterpret_cast<const ulonglong2*>(vn + e);
                    const u64 x = pk(ex2(__uint_as_float(v[e])), ex2(__uint_as_float(v[e + 1]))), y = pk(ex2(__uint_as_float(v[e + 2])), ex2(__uint_as_float(v[e + 3])));
                    l2a = add2(l2a, x); l2b = add2(l2b, y);
                    float x0, x1, y0, y1;
                    upk(mul2(x, n4.x), x0, x1); upk(mul2(y, n4.y), y0, y1);
                    w[i / 2] = pack_h2(x0, x1); w[i / 2 + 1] = pack_h2(y0, y1);
                }
                tmem_st32(s_col + 32 * h, w);
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar(P_FULL + sbuf(q, j)));
            mbar_arrive(bar(SC_FREE + s));
        }
        // ---- the row's result ----
        float l0, l1, l_sum;
        upk(add2(l2a, l2b), l0, l1);
        l_sum = l0 + l1;
        if (ok && n > 0) ok = wait_bar(ALL_DONE + q, 0);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        float* part = nullptr;
        if (p.n_splits > 1) {
            part = p.part + (((int64_t(blockIdx.y) * n_blocks + blk) * p.n_splits + split) * (NQ * TM) + m) * (D + 4);
            part[D] = n > 0 && ok ? m_ref - lvsc : -INFINITY;
            part[D + 1] = n > 0 && ok ? l_sum : 0.f;
        }
        if (n > 0 && ok) {
            const float il = 1.f / l_sum;
            const int64_t o0 = valid ? row_q_index(m) : 0;
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t o[32];
                tmem_ld32(t_row + P::COL_O + q * DP + c0, o);
                tmem_ld_wait();
                if (part) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<uint4*>(part + c0 + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                } else if (valid) {
                    if (p.out_dtype == TQ_F32) {
                        float* dst = static_cast<float*>(p.out) + o0 + c0;
#pragma unroll
                        for (int i = 0; i < 32; i += 4)
                            *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(o[i]) * il, __uint_as_float(o[i + 1]) * il, __uint_as_float(o[i + 2]) * il, __uint_as_float(o[i + 3]) * il);
                    } else {
                        uint32_t w[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float x = __uint_as_float(o[2 * i]) * il, y = __uint_as_float(o[2 * i + 1]) * il;
                            if (p.out_dtype == TQ_F16) w[i] = pack_h2(x, y);
                            else {
                                const __nv_bfloat162 bb = __floats2bfloat162_rn(x, y);
                                w[i] = *reinterpret_cast<const uint32_t*>(&bb);
                            }
                        }
                        uint4* dst = reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + o0 + c0);
#pragma unroll
                        for (int i = 0; i < 4; ++i) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
                    }
                }
            }
        }
    }
    // ---------------- teardown: every loop above is bounded, so every thread gets here ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == NQ * 4) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Partials of a row block's key ranges -> result: a warp per row.
template <int D>
__global__ void __launch_bounds__(256) fa_merge_kernel(Params p, int n_blocks, int n_rows) {
    constexpr int ROWS = Plan<D>::NQ * TM;
    const int lane = threadIdx.x & 31;
    const int64_t i = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);               // row of the launch: (lane x head group, row block, row)
    if (i >= n_rows) return;
    const int m = int(i % ROWS), blk = int(i / ROWS % n_blocks), y = int(i / ROWS / n_blocks);
    const int lane_c = y / p.HG, hg = y - lane_c * p.HG, gl = p.lane0 + lane_c, b = gl / p.Hkv, hkv = gl - b * p.Hkv;
    const int tok = blk * Plan<D>::NQ * p.QT + (m >> 7) * p.QT + (m & 127) / p.GP, hh = (m & 127) % p.GP;
    if (hh >= min(HPG, p.G - hg * HPG) || tok >= p.Tq) return;
    const float* part = p.part + ((int64_t(y) * n_blocks + blk) * p.n_splits * ROWS + m) * (D + 4);
    const int64_t stride = int64_t(ROWS) * (D + 4);
    float mm = -INFINITY, ll = 0.f;
    if (lane < p.n_splits) { mm = part[lane * stride + D]; ll = part[lane * stride + D + 1]; }
    float M = mm;
#pragma unroll
    for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    const float w = ll > 0.f ? ex2(mm - M) : 0.f;
    float sum = w * ll;
#pragma unroll
    for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    float acc[D / 32];
#pragma unroll
    for (int u = 0; u < D / 32; ++u) acc[u] = 0.f;
    for (int s = 0; s < p.n_splits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s);
        if (ws == 0.f) continue;                                                  // (a range without a visible token left no sums)
#pragma unroll
        for (int u = 0; u < D / 32; ++u) acc[u] = fmaf(ws, part[s * stride + u * 32 + lane], acc[u]);
    }
    const int64_t o = ((int64_t(b) * p.Hq + hkv * p.G + hg * HPG + hh) * p.Tq + tok) * D;
    const float il = 1.f / sum;
#pragma unroll
    for (int u = 0; u < D / 32; ++u) store_from_f32(p.out, p.out_dtype, o + u * 32 + lane, acc[u] * il);
}

// Uncompressed tokens into the expanded arrays, a warp per (lane, side, token): float16 rows as they are, float32 / bfloat16
// rows under a power-of-two scale (largest magnitude into [2^7, 2^8)) whose inverse takes the norm's place.  Also zeroes
// the norms of the positions between the last token and the next multiple of 128.
template <int D>
__global__ void __launch_bounds__(256) fa_dense_rows_kernel(DecodeParams c, int lane0, int n_lanes, int total, int ts, __half* k, __half* v, float* kn, float* vn) {
    const int lane = threadIdx.x & 31;
    const int n_dense = int(c.sink_len + c.res_len), n_items = n_dense + (ts - total);
    const int64_t i = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (i >= int64_t(n_lanes) * 2 * n_items) return;
    const int item = int(i % n_items), side = int(i / n_items) & 1, lc = int(i / n_items / 2);
    float* nn = (side ? vn : kn) + int64_t(lc) * ts;
    if (item >= n_dense) {
        if (lane == 0) nn[total + item - n_dense] = 0.f;
        return;
    }
    const bool in_sink = item < c.sink_len;
    const int pos = in_sink ? item : int(c.c_len) + item;
    const int64_t src = (in_sink ? (lane0 + lc) * c.sink_ls + item : (lane0 + lc) * c.res_ls + (item - c.sink_len)) * D;
    const void* base = in_sink ? (side ? c.sink_v : c.sink_k) : (side ? c.res_v : c.res_k);
    __half* dst = (side ? v : k) + (int64_t(lc) * ts + pos) * D;
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
    if (lane == 0) nn[pos] = 1.f / sc;
}

}  // namespace fa

// rowops.cu: with scales, rows c @ R leave without their norms, which are copied there
int dequantize_jobs(const tq_dequantize_args* q, int n, float* const* scales, int64_t scale_lane_stride, const int* parts, const float* tab_scale, cudaStream_t s);

namespace fa {

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

// How a call of n_lanes cache lanes is laid out in the workspace.
struct Layout {
    int GP, QT, n_blocks, n_splits, ts;
    size_t k, v, kn, vn, part, bytes;
};
// n_splits 0: chosen here, for a call (or its first round); a later round of fewer lanes keeps the first one's: left to itself it may
// choose more ranges, whose partials can outweigh the rows it saves (13 sequences of 120,026 tokens at d = 128: 711 MB of 537).
template <int D> static Layout layout(int n_lanes, int G, int64_t total, int t_q, int n_splits = 0) {
    using P = Plan<D>;
    Layout l{};
    const int g = std::min(G, HPG), hg = (G + HPG - 1) / HPG;
    l.GP = g <= 1 ? 1 : g <= 2 ? 2 : g <= 4 ? 4 : 8;
    l.QT = TM / l.GP;
    l.n_blocks = (t_q + P::NQ * l.QT - 1) / (P::NQ * l.QT);
    l.ts = int((total + 127) / 128 * 128);
    // key ranges per row block: as many as shorten the whole launch, a CTA costing its tiles and some twelve more for set-up,
    // first scores and the partials (with four, 512 queries x 32 lanes over 16,384 tokens were split for a merge of 34 us and no gain)
    const int64_t tiles = (total + P::TN - 1) / P::TN, ctas = int64_t(l.n_blocks) * n_lanes * hg, sms = sm_count();
    double best = 0.0;
    l.n_splits = n_splits;
    for (int s = 1; n_splits == 0 && s <= 16 && (s == 1 || tiles >= 2 * s); ++s) {
        const double t = double((ctas * s + sms - 1) / sms) * (double((tiles + s - 1) / s) + 12.0) + (s > 1 ? 8.0 : 0.0);
        if (s == 1 || t < best) { best = t; l.n_splits = s; }
    }
    const size_t rows = size_t(n_lanes) * l.ts;
    l.k = 0;
    l.v = up(rows * D * 2);
    l.kn = l.v + up(rows * D * 2);
    l.vn = l.kn + up(rows * 4);
    l.part = l.vn + up(rows * 4);
    l.bytes = l.part + (l.n_splits > 1 ? up(size_t(n_lanes) * hg * l.n_blocks * l.n_splits * P::NQ * TM * (D + 4) * 4) : 0);
    return l;
}

constexpr size_t WS_CAP = size_t(1) << 29;             // more lanes than fit 512 MB are done in several rounds

template <int D> static size_t workspace(int lanes, int G, int64_t total, int t_q) {
    const size_t all = layout<D>(lanes, G, total, t_q).bytes, one = layout<D>(1, G, total, t_q).bytes;
    return std::max(std::min(all, WS_CAP), one);
}

// The rounds of a call with ws_bytes of workspace: cache lanes of a round (the last one may have fewer) and key ranges of all of them.
template <int D> static int first_round(int lanes, int G, int64_t total, int t_q, size_t ws_bytes, int& n_splits) {
    int chunk = lanes;
    while (chunk > 1 && layout<D>(chunk, G, total, t_q).bytes > ws_bytes) chunk = (chunk + 1) / 2;
    n_splits = layout<D>(chunk, G, total, t_q).n_splits;
    return chunk;
}

template <int D> static size_t most_used(int lanes, int G, int64_t total, int t_q, size_t ws_bytes) {
    int n_splits;
    const int chunk = first_round<D>(lanes, G, total, t_q, ws_bytes, n_splits);
    size_t most = 0;
    for (int lane0 = 0; lane0 < lanes; lane0 += chunk) most = std::max(most, layout<D>(std::min(chunk, lanes - lane0), G, total, t_q, n_splits).bytes);
    return most;
}

template <int D> static int run(const DecodeParams& c, const void* q, int q_dtype, void* out, int out_dtype, int t_q, int64_t q_pos0, unsigned char* ws,
                                size_t ws_bytes, cudaStream_t s) {
    using P = Plan<D>;
    const int64_t total = c.sink_len + c.c_len + c.res_len;
    const int lanes = c.B * c.Hkv;
    int n_splits;
    const int chunk = first_round<D>(lanes, c.G, total, t_q, ws_bytes, n_splits);
    static std::atomic<bool> set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !set[dev].load()) {
        cudaError_t e = cudaFuncSetAttribute(fa_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(P::SMEM));
        if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: shared memory %zu B: %s", P::SMEM, cudaGetErrorString(e));
        set[dev].store(true);
    }
    for (int lane0 = 0; lane0 < lanes; lane0 += chunk) {
        const int n = std::min(chunk, lanes - lane0);
        const Layout l = layout<D>(n, c.G, total, t_q, n_splits);
        if (l.bytes > ws_bytes) return fail(TQ_ERR_INVALID, "tq_prefill_attn: workspace %zu B < %zu B", ws_bytes, l.bytes);
        __half* k = reinterpret_cast<__half*>(ws + l.k);
        __half* v = reinterpret_cast<__half*>(ws + l.v);
        float* kn = reinterpret_cast<float*>(ws + l.kn);
        float* vn = reinterpret_cast<float*>(ws + l.vn);
        const int64_t items = int64_t(n) * 2 * (c.sink_len + c.res_len + (l.ts - total));
        if (items > 0) {
            fa_dense_rows_kernel<D><<<unsigned((items + 7) / 8), 256, 0, s>>>(c, lane0, n, int(total), l.ts, k, v, kn, vn);
            if (int rc = check_launch("tq_prefill_attn")) return rc;
        }
        if (c.c_len > 0) {
            tq_dequantize_args d[2] = {};
            float* scales[2] = {kn + c.sink_len, vn + c.sink_len};
            int parts[2];
            float tab[2];
            for (int side = 0; side < 2; ++side) {
                tq_dequantize_args& a = d[side];
                const int hi = side ? c.vb_hi : c.kb_hi, lo = side ? c.vb_lo : c.kb_lo;
                const int w_hi = packed_bytes(lo ? D / 2 : D, hi), w_lo = lo ? packed_bytes(D / 2, lo) : 0;
                a.packed_hi = (side ? c.v_hi : c.k_hi) + int64_t(lane0) * c.c_ls * w_hi;
                a.packed_lo = lo ? (side ? c.v_lo : c.k_lo) + int64_t(lane0) * c.c_ls * w_lo : nullptr;
                a.norms = (side ? c.v_norms : c.k_norms) + int64_t(lane0) * c.c_ls;
                a.n_lanes = n; a.n_rows = c.c_len; a.in_lane_stride = c.c_ls;
                a.d = D; a.bits_hi = hi; a.bits_lo = lo;
                a.cent_hi = side ? c.vc_hi : c.kc_hi; a.cent_lo = side ? c.vc_lo : c.kc_lo; a.rot = c.rot;
                a.out = (side ? v : k) + c.sink_len * D; a.out_dtype = TQ_F16;
                a.out_lane_stride = int64_t(l.ts) * D; a.out_row_stride = D;
                // fp16 centroids as they are for keys, under their best scale for values (one scale cannot serve two tables: both parts)
                parts[side] = side && lo ? 2 : 1;
                tab[side] = side && !lo ? c.v_scale_hi : 1.f;
            }
            if (int rc = dequantize_jobs(d, 2, scales, l.ts, parts, tab, s)) return rc;
        }
        CUtensorMap maps[2];
        for (int side = 0; side < 2; ++side) {
            const cuuint64_t dims[3] = {cuuint64_t(D), cuuint64_t(total), cuuint64_t(n)};        // rows past the last token read as zeros
            const cuuint64_t strides[2] = {cuuint64_t(D) * 2, cuuint64_t(l.ts) * D * 2};
            const cuuint32_t box[3] = {64, cuuint32_t(P::TN), 1}, es[3] = {1, 1, 1};
            if (encoder()(&maps[side], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, side ? v : k, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: cannot describe the expanded rows to the tensor memory accelerator");
        }
        Params p{};
        p.q = q; p.q_dtype = q_dtype; p.f = c.scale * LOG2E; p.out = out; p.out_dtype = out_dtype;
        p.Hq = c.Hq; p.Hkv = c.Hkv; p.G = c.G; p.HG = c.HG; p.GP = l.GP; p.QT = l.QT; p.Tq = t_q;
        p.lane0 = lane0; p.q_pos0 = int(q_pos0); p.total = int(total);
        p.kn = kn; p.vn = vn; p.ts = l.ts; p.n_splits = l.n_splits;
        p.part = reinterpret_cast<float*>(ws + l.part);
        if (!(p.status = decode_status_ptr())) return fail(TQ_ERR_LAUNCH, "tq_prefill_attn: cannot locate the status word");
        fa_kernel<D><<<dim3(unsigned(l.n_blocks * l.n_splits), unsigned(n * c.HG)), P::NT, P::SMEM, s>>>(p, maps[0], maps[1]);
        if (int rc = check_launch("tq_prefill_attn")) return rc;
        if (l.n_splits > 1) {
            const int rows = n * c.HG * l.n_blocks * P::NQ * TM;
            fa_merge_kernel<D><<<unsigned((rows + 7) / 8), 256, 0, s>>>(p, l.n_blocks, rows);
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

// Whether the two-step kernel takes the call with this workspace; the caller has validated the arguments.
bool prefill_fa_applicable(const tq_decode_args* a, int t_q) {
    const int64_t total = a->c_len + a->sink_len + a->res_len;
    // (a float32 query would be rounded to fp16 beside the rounding of the expanded rows; 16-bit queries are exact: float32 callers
    // stay with the kernels that multiply the rotated query with the centroids, one rounding fewer)
    if (a->q_dtype == TQ_F32) return false;
    if (!a->workspace || !aligned(a->workspace, 256) || total >= (int64_t(1) << 30) || !fa::encoder()) return false;
    if (a->c_len > 0 && ((a->k_bits_lo && a->k_bits_lo != a->k_bits_hi - 1) || (a->v_bits_lo && a->v_bits_lo != a->v_bits_hi - 1))) return false;
    if (!aligned(a->out, 16) || !aligned(a->rot, 16)) return false;
    return a->workspace_bytes >= prefill_fa_workspace(1, a->n_q_heads / a->n_kv_heads, 1, a->d, total, t_q);      // one lane at a time at least
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

extern "C" size_t tq_prefill_workspace_used(int batch, int n_q_heads, int n_kv_heads, int d, int64_t total_len, int t_q, size_t workspace_bytes) {
    using namespace tq;
    if (prefill_fa_workspace(batch, n_q_heads, n_kv_heads, d, total_len, t_q) == 0 ||
        workspace_bytes < prefill_fa_workspace(1, n_q_heads / n_kv_heads, 1, d, total_len, t_q)) return 0;
    const int lanes = batch * n_kv_heads, g = n_q_heads / n_kv_heads;
    if (d == 64) return fa::most_used<64>(lanes, g, total_len, t_q, workspace_bytes);
    if (d == 96) return fa::most_used<96>(lanes, g, total_len, t_q, workspace_bytes);
    if (d == 128) return fa::most_used<128>(lanes, g, total_len, t_q, workspace_bytes);
    return fa::most_used<256>(lanes, g, total_len, t_q, workspace_bytes);
}
