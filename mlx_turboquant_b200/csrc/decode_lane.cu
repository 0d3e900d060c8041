// Decode attention of small and middling calls in ONE launch: a cluster of C CTAs per cache lane (sequence, KV head, head group), with the
// widths, head dims and operands of decode_lut.cu (lookup tables in shared memory, decode_lut.cuh).
//
// Why.  The persistent grid of decode_lut.cu deals the tiles of all lanes out flat, which long contexts need, but pays for it with
// partials in global memory and launches around it (queries, merge): some 20 us per call before the first tile counts.  Here a lane's
// tiles belong to the 8 C warps of its cluster - some warps take packed tiles, the others uncompressed ones, in proportion - and
// nothing leaves the chip before the result: warps fold in shared memory, CTAs over distributed shared memory, and each CTA rotates
// its share of the output columns back.  Eight warps per CTA; an SM to each while the CTAs are few, else two CTAs per SM.
//   us per call on caches that do not come from L2, 4 query heads per lane unless given, other kernels / here: 8 lanes x 600 tokens, 4 / 2
//   bits 11.9 / 8.4; 32 x 11,777, 3.5 / 3.5 38.0 / 32.8; 160 x 1064, 3 / 4 40.3 / 28.4; 3 x 5902 of 8 heads, 4 / 4 25 / 14; 272 x 933 at d = 96,
//   2 / 2 39.7 / 20.7; 72 x 3912 of one head with sketches 39.7 / 30; 16 x 3735 at d = 64 15.3 / 10.
// Where 8.4 us go (stamps from the end of the launch before): dependency wait 0.6, rotated query at 2.0, first tile read 2.7, its products
// 3.7, partial stored 4.3, folded 4.8, cluster barrier 5.4, merged 6.5, rotated back 7.4, stored 8.0.  A tile's products are a chain of
// latencies (0.9 us for a warp alone); two tiles interleaved in a warp took longer (twice the code: 39 against 35 us for 32 x 11,777).
//
// Uncompressed tokens (16-bit) go from global memory into the operand registers: keys as the A operand with the coordinates in the
// order of the packed rows (a thread owns a quarter of a row), values by one byte-permute per register from the rows of two tokens.
// bfloat16 rows take the query and the weights as high + low bfloat16 parts (decode_lut.cu).
//
// Every mbarrier wait is bounded (status 112); the warp whose copies never land drains what is in flight (bounded), leaves its tokens
// out and takes part in the rest, so that the cluster's barriers are always reached by all.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "decode_lut.cuh"

namespace tq {
namespace dl {

using namespace lut;

constexpr int ERR_RING = 112, ERR_LAYOUT = 113;
constexpr int NW = 8, NT = NW * 32, MAX_C = 16, MAX_NS = 3;
constexpr uint32_t LO_BASE = 1024u;                 // where the dynamic allocation starts (checked)
using Tab = Tables<LO_BASE>;

template <int D, bool QJL, int PER_SM> struct Plan {
    static constexpr uint32_t SC = (QJL ? 6u : 2u) * TILE * 4u;                      // a stage's scalars: norms, sign words, residual norms
    static constexpr uint32_t O_KN = 0, O_VN = 64, O_KB = 128, O_KG = 192, O_VB = 256, O_VG = 320;
    static constexpr int NC = (int((SC + 2u * TILE * D / 2) / 16) + 31) / 32;        // 16-byte chunks per lane at most
    static constexpr uint32_t BYTES = (PER_SM == 1 ? 227u : 113u) * 1024u, END = LO_BASE + BYTES;
    static constexpr int QR = D + (QJL ? QM : 0);                                    // rotated query | sketch of a head
    static constexpr uint32_t QROT = END - HPG * QR * 2u, BARS = QROT - 8u * NW * MAX_NS;
    // Behind the loop, from LO_BASE on (tables and rings are dead): warps' partials, the CTA's sums, the lane's, products with R.
    // Partials and sums keep the order of the accumulators: slot 16 mt + 2 g + u is coordinate coord_of(slot).
    static constexpr int PS = QR + 8;                                                // floats per head of a partial: values | sketch rows | max, sum, pad (2 PS = 16 mod 32 banks)
    static constexpr uint32_t RED = LO_BASE, CP = RED + NW * HPG * PS * 4u, CD = CP + HPG * QR * 4u, ML = CD + HPG * D * 4u;
    static constexpr uint32_t WT = ML + HPG * 8u, Y = WT + HPG * (MAX_C + 4) * 4u, YD = Y + HPG * (QR + 1) * 4u, OP = YD + HPG * D * 4u;
    static_assert(OP + NT * HPG * 4u <= BARS && RED % 16 == 0 && Y % 16 == 0 && PS % 4 == 0, "shared-memory plan");
};
__host__ __device__ constexpr uint32_t ring_base(bool any3) { return any3 ? Tab::END : Tab::K3; }

// ---- cluster ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// all of the CTA's threads, from either side of a branch between warps
__device__ __forceinline__ void cta_sync() { asm volatile("barrier.sync 0;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 peer_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 peer_f2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float peer_f1(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void prefetch_l2(const void* ptr) { asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr)); }

// ---- uncompressed tokens ------------------------------------------------------------------------------------
// N words from global memory, 16 (N = 6: 8) bytes at a time; ordered behind the dependency wait
template <int N> __device__ __forceinline__ void load_words(uint32_t (&w)[N], const uint16_t* src) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]) : "l"(src + 2 * i) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(w[i]), "=r"(w[i + 1]) : "l"(src + 2 * i) : "memory");
    }
}
// Rows of the uncompressed tokens of cache lane kvl: sink, recent window, the token that this call appends
struct DenseRows {
    const uint16_t *sink, *res, *fresh;
    int s_len, r_len, n_tok;
    template <int D> __device__ __forceinline__ const uint16_t* row(int tok) const {
        const int rr = tok - s_len;
        return tok < s_len ? sink + int64_t(tok) * D : rr < r_len ? res + int64_t(rr) * D : fresh;
    }
};
__device__ __forceinline__ DenseRows dense_rows(const DecodeParams& p, int64_t kvl, bool keys) {
    DenseRows r;
    r.sink = static_cast<const uint16_t*>(keys ? p.sink_k : p.sink_v) + kvl * p.sink_ls * p.D;
    r.res = static_cast<const uint16_t*>(keys ? p.res_k : p.res_v) + kvl * p.res_ls * p.D;
    r.fresh = static_cast<const uint16_t*>(keys ? p.k_new : p.v_new) + kvl * p.D;
    r.s_len = int(p.sink_len); r.r_len = int(p.res_len); r.n_tok = r.s_len + r.r_len + (p.k_new ? 1 : 0);
    return r;
}
// Elements c0 + step ks + half u, + 1 (u = 0, 1) of a query head, every load in flight at once
template <int D> __device__ __forceinline__ void load_query(const DecodeParams& p, int64_t head, bool live, int c0, int step, int half, float2 (&x)[D / 16][2]) {
    const int64_t e0 = head * D + c0;
    if (p.q_dtype == TQ_F32) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int u = 0; u < 2; ++u) x[ks][u] = live ? *reinterpret_cast<const float2*>(static_cast<const float*>(p.q) + e0 + step * ks + half * u) : make_float2(0.f, 0.f);
        return;
    }
    uint32_t w[D / 16][2];
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int u = 0; u < 2; ++u) w[ks][u] = live ? *reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.q) + e0 + step * ks + half * u) : 0u;
    const bool f16 = p.q_dtype == TQ_F16;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w[ks][u]));
            x[ks][u] = f16 ? h : make_float2(__uint_as_float(w[ks][u] << 16), __uint_as_float(w[ks][u] & 0xffff0000u));
        }
}
// Sixteen rows of R (or S) as fp16 high and 2^-11 low parts, A operands: prepared before the wait, so that behind it a slab costs the
// query's loads and its products.  (Splitting behind the wait: 3.1 us from the wait to the rotated query, 1.4 now.)
template <int D> struct Slab {
    uint32_t h[D / 16][4], l[D / 16][4];
    __device__ __forceinline__ void load(const DecodeParams& p, int slab, int g, int t) {
        float2 rr[D / 16][4];
        load_rows<D>(p, slab, g, t, rr);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int r = 0; r < 4; ++r) split_h2(rr[ks][r], h[ks][r], l[ks][r]);
    }
};

// Tiles [tile0, tile0 + n); k-slots and MMA rows are tokens in their own order.
template <int D, bool BF16>
__device__ __forceinline__ void dense_direct(const DecodeParams& p, int64_t kvl, int tile0, int n, int64_t qhead, bool live_q, WarpAcc<D, 0>& st, int lane) {
    constexpr int KW = D / 8, VW = D / 16;                              // words a thread owns of a key row, of a value row
    const int g = lane >> 2, t = lane & 3;
    const DenseRows kr = dense_rows(p, kvl, true), vr = dense_rows(p, kvl, false);
    uint32_t ka[KW], kb[KW];
    auto load_keys = [&](int tok0) {
        load_words(ka, kr.row<D>(min(tok0 + g, kr.n_tok - 1)) + t * (D / 4));
        load_words(kb, kr.row<D>(min(tok0 + g + 8, kr.n_tok - 1)) + t * (D / 4));
    };
    load_keys(tile0 * TILE);                                            // (in flight beside the query's)
    uint32_t bh[D / 16][2], bl[BF16 ? D / 16 : 1][2];
    {
        float2 x[D / 16][2];
        load_query<D>(p, qhead, live_q, t * (D / 4), 4, 2, x);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float2 y = make_float2(x[ks][u].x * (p.scale * LOG2E), x[ks][u].y * (p.scale * LOG2E));
                if (BF16) {
                    bh[ks][u] = pack_bf2(y.x, y.y);
                    bl[ks][u] = pack_bf2(y.x - __uint_as_float(bh[ks][u] << 16), y.y - __uint_as_float(bh[ks][u] & 0xffff0000u));
                } else {
                    bh[ks][u] = pack_h2(y.x, y.y);
                }
            }
    }
    // Keys of a tile are asked for when the previous tile's have been used, its values likewise: both have about a tile's time to arrive.
    uint32_t w[4][VW];                                                  // tokens 2 t, 2 t + 1, 2 t + 8, 2 t + 9: coordinates g (D / 8), ...
    auto load_values = [&](int tok0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) load_words(w[u], vr.row<D>(min(tok0 + 2 * t + (u & 1) + 4 * (u & 2), kr.n_tok - 1)) + g * (D / 8));
    };
    load_values(tile0 * TILE);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int tok0 = (tile0 + i) * TILE;
        if (i + 2 < n) {                                                // the tile after the next into L2: two lanes a row
            const int tok = min(tok0 + 2 * TILE + (lane >> 1), kr.n_tok - 1);
#pragma unroll
            for (int u = 0; u < (D + 127) / 128; ++u) {
                prefetch_l2(kr.row<D>(tok) + (lane & 1) * (D / 2) + 64 * u);
                prefetch_l2(vr.row<D>(tok) + (lane & 1) * (D / 2) + 64 * u);
            }
        }
        const bool ok0 = tok0 + g < kr.n_tok, ok1 = tok0 + g + 8 < kr.n_tok;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t a[4] = {ka[2 * ks], kb[2 * ks], ka[2 * ks + 1], kb[2 * ks + 1]};
            if (BF16) { mma_bf16(s, a, bh[ks][0], bh[ks][1]); mma_bf16(s, a, bl[ks][0], bl[ks][1]); }
            else mma16816(s, a[0], a[1], a[2], a[3], bh[ks][0], bh[ks][1]);
        }
        if (i + 1 < n) load_keys(tok0 + TILE);
        if (tok0 + TILE > kr.n_tok) {                                   // rows past the end: no weight, and zeros so that no Inf or NaN meets it
            s[0] = ok0 ? s[0] : -INFINITY; s[1] = ok0 ? s[1] : -INFINITY;
            s[2] = ok1 ? s[2] : -INFINITY; s[3] = ok1 ? s[3] : -INFINITY;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (tok0 + 2 * t + (u & 1) + 4 * (u & 2) >= kr.n_tok) {
#pragma unroll
                    for (int m = 0; m < VW; ++m) w[u][m] = 0u;
                }
        }
        float pr[4];
        softmax_scores<D, 0>(s, 1.f, 1.f, 0.f, st, pr);                 // (value norms are 1)
        uint32_t bp[2], bpl[2] = {0u, 0u};
        if (BF16) {
            const uint32_t h0 = pack_bf2(pr[0], pr[1]), h1 = pack_bf2(pr[2], pr[3]);
            bp[0] = movm_t(h0); bp[1] = movm_t(h1);
            bpl[0] = movm_t(pack_bf2(pr[0] - __uint_as_float(h0 << 16), pr[1] - __uint_as_float(h0 & 0xffff0000u)));
            bpl[1] = movm_t(pack_bf2(pr[2] - __uint_as_float(h1 << 16), pr[3] - __uint_as_float(h1 & 0xffff0000u)));
        } else {
            bp[0] = movm_t(pack_h2(pr[0], pr[1])); bp[1] = movm_t(pack_h2(pr[2], pr[3]));
        }
#pragma unroll
        for (int mt = 0; mt < VW; ++mt) {
            const uint32_t a[4] = {__byte_perm(w[0][mt], w[1][mt], 0x5410), __byte_perm(w[0][mt], w[1][mt], 0x7632), __byte_perm(w[2][mt], w[3][mt], 0x5410),
                                   __byte_perm(w[2][mt], w[3][mt], 0x7632)};
            if (BF16) { mma_bf16(st.o[mt], a, bp[0], bp[1]); mma_bf16(st.o[mt], a, bpl[0], bpl[1]); }
            else mma16816(st.o[mt], a[0], a[1], a[2], a[3], bp[0], bp[1]);
        }
        if (i + 1 < n) load_values(tok0 + TILE);
    }
}

// A warp's partial of up to eight heads (PS floats each): values, sketch rows, maximum, sum.  Rows g, g + 8 of m-tile mt are two
// coordinates in a row of this thread's share, slots 16 mt + 2 g, + 1.
template <int D, int NZ, int PS>
__device__ __forceinline__ void store_partial(float* dst, WarpAcc<D, NZ>& st, int heads_here, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const float r = __int_as_float(0x7f000000 - __float_as_int(st.vsc));       // 1 / vsc, a power of two in [2^-120, 2^120]
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
        st.l[0] += __shfl_xor_sync(0xffffffffu, st.l[0], off);
        st.l[1] += __shfl_xor_sync(0xffffffffu, st.l[1], off);
    }
    if (2 * t >= heads_here) return;
    const bool two = 2 * t + 1 < heads_here;
    float* h0 = dst + (2 * t) * PS;
    float* h1 = h0 + PS;
#pragma unroll
    for (int mt = 0; mt < D / 16; ++mt) {
        *reinterpret_cast<float2*>(h0 + 16 * mt + 2 * g) = make_float2(st.o[mt][0] * r, st.o[mt][2] * r);
        if (two) *reinterpret_cast<float2*>(h1 + 16 * mt + 2 * g) = make_float2(st.o[mt][1] * r, st.o[mt][3] * r);
    }
#pragma unroll
    for (int mz = 0; mz < NZ; ++mz) {
        h0[D + 16 * mz + g] = st.z[mz][0] * r; h0[D + 16 * mz + g + 8] = st.z[mz][2] * r;
        if (two) { h1[D + 16 * mz + g] = st.z[mz][1] * r; h1[D + 16 * mz + g + 8] = st.z[mz][3] * r; }
    }
    if (g == 0) {
        *reinterpret_cast<float2*>(h0 + PS - 8) = make_float2(st.m[0], st.l[0]);
        if (two) *reinterpret_cast<float2*>(h1 + PS - 8) = make_float2(st.m[1], st.l[1]);
    }
}
template <int D> __device__ __forceinline__ int coord_of(int slot, bool split) {
    const int mt = slot >> 4, g = (slot >> 1) & 7, u = slot & 1;
    return (split ? (mt < D / 32 ? g * (D / 16) + 2 * mt : D / 2 + g * (D / 16) + 2 * (mt - D / 32)) : g * (D / 8) + 2 * mt) + u;
}
template <int D> __device__ __forceinline__ int slot_of(int c) {       // (unsplit rows)
    const int g = c / (D / 8), x = c - g * (D / 8);
    return 16 * (x >> 1) + 2 * g + (x & 1);
}

// PER_SM: CTAs that share an SM (d = 256: 1).  Alone it has registers enough to keep everything; two have half each and spill some.
template <int D, bool QJL, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) decode_lane_kernel(DecodeParams p) {
    using P = Plan<D, QJL, PER_SM>;
    constexpr int NZ = QJL ? QM / 16 : 0, NC = P::NC, QR = P::QR, PS = P::PS, SLABS = D / 16 + NZ;
    extern __shared__ __align__(16) unsigned char smem[];
    // In a cluster the shared-window address of a CTA's own memory carries its rank in the upper bits: the plan's addresses are offsets
    // from `base`, and the upper half of a table address comes with the lane's copy offset.
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem)), base = sbase & 0xffff0000u, s0 = sbase - base;
    auto gp = [&](uint32_t addr) -> unsigned char* { return smem + (addr - s0); };
    auto fp = [&](uint32_t addr) -> float* { return reinterpret_cast<float*>(smem + (addr - s0)); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    if (s0 > LO_BASE || (s0 & 15u)) {                  // (the same in every CTA) cannot happen after the host-side probe; never run on a bad plan
        if (tid == 0) atomicCAS(p.status, 0, ERR_LAYOUT);
        return;
    }
    pdl_trigger();
    const int C = p.ln_c, a = int(blockIdx.x) / C, rank = int(blockIdx.x) - a * C;
    const int kvl = a / p.HG, hg = a - kvl * p.HG, b = kvl / p.Hkv, hkv = kvl - b * p.Hkv;
    const int heads_here = min(HPG, p.G - hg * HPG), head0 = hkv * p.G + hg * HPG;          // first query head of the group
    const int64_t q0 = int64_t(b) * p.Hq + head0;
    // this warp's tiles: packed ones for the first n_pw warps of the cluster, uncompressed ones for the n_dw after them
    const int wr = rank * NW + warp, n_pw = p.ln_pw, n_dw = p.ln_dw;
    const bool packed = wr < n_pw, has_packed = rank * NW < n_pw;
    int first = 0, n_my = 0;
    {
        const int n_all = packed ? int((p.c_len + TILE - 1) / TILE) : (int(p.sink_len + p.res_len) + (p.k_new ? 1 : 0) + TILE - 1) / TILE;
        const int w = packed ? wr : wr - n_pw, n_w = packed ? n_pw : n_dw;
        if (w < n_w) {
            const int each = n_all / n_w, extra = n_all - each * n_w;
            n_my = each + (w < extra ? 1 : 0);
            first = w * each + min(w, extra);
        }
    }
    // ---------------- constants only, before the wait for the previous launch ----------------
    const int ns = p.ln_ns;
    const uint32_t bar0 = base + P::BARS + 8u * uint32_t(warp) * MAX_NS;
    if (lane == 0) {
        for (int s = 0; s < MAX_NS; ++s) mbar_init(bar0 + 8u * s, 32);       // every lane arrives when its copies into the stage have completed
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int kwh = packed_bytes(p.kb_lo ? D / 2 : D, p.kb_hi), kwl = p.kb_lo ? packed_bytes(D / 2, p.kb_lo) : 0;
    const int vwh = packed_bytes(p.vb_lo ? D / 2 : D, p.vb_hi), vwl = p.vb_lo ? packed_bytes(D / 2, p.vb_lo) : 0;
    const bool any3 = p.kb_hi == 3 || p.kb_lo == 3 || p.vb_hi == 3 || p.vb_lo == 3;
    const uint32_t stage_b = P::SC + 16u * uint32_t(kwh + kwl + vwh + vwl), my_area = base + ring_base(any3) + uint32_t(warp) * (uint32_t(ns) * stage_b + 16u);
    const unsigned char* cp_ptr[NC];
    uint32_t cp_step[NC];
    Slab<D> slab;
    if (has_packed) {
        // (lines of the first tiles are asked for in L2: harmless whoever may still be writing them)
        if (packed) {
            const int n_sc = int(P::SC / 16), n_chunks = n_sc + kwh + kwl + vwh + vwl;
            const int64_t row = int64_t(kvl) * p.c_ls + int64_t(first) * TILE;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                int c = lane + 32 * j, rb;
                const unsigned char* src = chunk_source(p, c, n_sc, kwh, kwl, vwh, rb);
                cp_ptr[j] = src + row * rb + 16 * c;
                cp_step[j] = lane + 32 * j < n_chunks ? uint32_t(TILE * rb) : 0u;
                if (cp_step[j] && n_my > 0) prefetch_l2(cp_ptr[j]);
            }
        }
        fill_tables<Tab, NT>(p, tid, gp);
        if (warp < SLABS) slab.load(p, warp, g, t);
    }
    if (!packed && n_my > 0) {
        const DenseRows kr = dense_rows(p, kvl, true), vr = dense_rows(p, kvl, false);
#pragma unroll 1
        for (int i = 0; i < min(n_my, 2); ++i) {
            const int tok = min((first + i) * TILE + (lane >> 1), kr.s_len + kr.r_len - 1);
            if (tok < 0) break;
#pragma unroll
            for (int u = 0; u < (D + 127) / 128; ++u) {
                prefetch_l2(kr.row<D>(tok) + (lane & 1) * (D / 2) + 64 * u);
                prefetch_l2(vr.row<D>(tok) + (lane & 1) * (D / 2) + 64 * u);
            }
        }
    }
    __syncthreads();
    pdl_wait();        // the query and the cache are settled from here on
    await_gather(p);   // (head-sharded decoding) ... and the peers' heads of an earlier call have arrived
    const unsigned epoch = next_epoch(p, a);

    auto issue = [&](int stage) {
        const uint32_t bar = bar0 + 8u * stage, dst = my_area + uint32_t(stage) * stage_b + 16u * lane;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            if (cp_step[j]) cp_async16(dst + 512u * j, cp_ptr[j], 16);
            cp_ptr[j] += cp_step[j];
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    };
    if (packed) {
#pragma unroll 1
        for (int n = 0; n < min(n_my, ns); ++n) issue(n);
    }
    __half* qrot = reinterpret_cast<__half*>(gp(P::QROT));
    if (has_packed) {
        // q_rot[h][j] = sum_k q[h][k] R[j][k] (rotation.py:81-110) and (S q) (qjl.py:70-94), times scale * log2(e): a slab of sixteen rows per
        // warp.  A float16 query is a B operand as it is; others are scaled and split like R (the low parts' product is below float32 resolution).
        if (warp < SLABS) {
            const float f = p.scale * LOG2E;
            const bool f16 = p.q_dtype == TQ_F16;
            uint32_t bh[D / 16][2], bl[D / 16][2];
            {
                float2 x[D / 16][2];
                load_query<D>(p, q0 + min(g, heads_here - 1), g < heads_here, 2 * t, 16, 8, x);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
                    for (int u = 0; u < 2; ++u) split_h2(f16 ? x[ks][u] : make_float2(x[ks][u].x * f, x[ks][u].y * f), bh[ks][u], bl[ks][u]);
            }
#pragma unroll 1
            for (int un = warp; un < SLABS; un += NW) {
                if (un != warp) slab.load(p, un, g, t);
                float ym[4] = {0.f, 0.f, 0.f, 0.f}, ya[4] = {0.f, 0.f, 0.f, 0.f}, yb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    mma16816(ym, slab.h[ks][0], slab.h[ks][1], slab.h[ks][2], slab.h[ks][3], bh[ks][0], bh[ks][1]);
                    mma16816(ya, slab.l[ks][0], slab.l[ks][1], slab.l[ks][2], slab.l[ks][3], bh[ks][0], bh[ks][1]);
                    if (!f16) mma16816(yb, slab.h[ks][0], slab.h[ks][1], slab.h[ks][2], slab.h[ks][3], bl[ks][0], bl[ks][1]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {              // rows g, g + 8 of the slab x heads 2t, 2t + 1
                    const int h = 2 * t + (r & 1);
                    if (h < heads_here) qrot[h * QR + un * 16 + g + (r >> 1) * 8] = __float2half_rn((ym[r] + (ya[r] + yb[r]) * (1.f / 2048.f)) * (f16 ? f : 1.f));
                }
            }
        }
        __syncthreads();
    }

    float* const red = fp(P::RED);
    float* const my_part = red + warp * (HPG * PS);
    if (packed) {
        const Copies cpy{base | uint32_t(lane * 4), base | uint32_t((lane & 15) * 8)};
        const TileLayout ly = tile_layout<P, D>(p, lane);
        uint32_t bq[D / 16][2], bu[QM / 16][2];
        {
            const __half* qh = qrot + g * QR;
            const bool split = p.kb_lo != 0, live = g < heads_here;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const int c = split ? (ks < D / 32 ? t * (D / 8) + 4 * ks : D / 2 + t * (D / 8) + 4 * (ks - D / 32)) : t * (D / 4) + 4 * ks;
                const uint2 x = live ? *reinterpret_cast<const uint2*>(qh + c) : make_uint2(0u, 0u);
                bq[ks][0] = x.x; bq[ks][1] = x.y;
            }
            // k slot (ks, register hh, half e) of lane t stands for sketch row 4t + 2ks + hh + 16e
#pragma unroll
            for (int ks = 0; ks < QM / 16; ++ks)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const unsigned short* z = reinterpret_cast<const unsigned short*>(qh + D + 4 * t + 2 * ks + hh);
                    bu[ks][hh] = QJL && live ? uint32_t(z[0]) | (uint32_t(z[16]) << 16) : 0u;
                }
        }
        WarpAcc<D, NZ> st;
        st.init();
        const int c_len = int(p.c_len);
        bool failed = false;
#pragma unroll 1
        for (int n = 0, stage = 0, phase = 0; n < n_my; ++n) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar0 + 8u * stage, uint32_t(phase)))) {
                atomicCAS(p.status, 0, ERR_RING);
                failed = true;
                for (int m = n + 1; m < min(n_my, n + ns); ++m) mbar_wait(bar0 + 8u * (m % ns), uint32_t(m / ns) & 1u);
                break;
            }
            packed_tile<Tab, P, D, QJL>(my_area + uint32_t(stage) * stage_b, ly, bq, bu, cpy, c_len - (first + n) * TILE, st, lane);
            if (n + ns < n_my) {
                __syncwarp();
                issue(stage);
            }
            if (++stage == ns) { stage = 0; phase ^= 1; }
        }
        if (failed) st.init();
        cta_sync();            // tables and rings are dead from here on
        store_partial<D, NZ, PS>(my_part, st, heads_here, lane);
    } else {
        WarpAcc<D, 0> st;
        st.init();
        if (n_my > 0) {
            const int64_t qhead = q0 + min(g, heads_here - 1);
            if (p.dense_dtype == TQ_F16) dense_direct<D, false>(p, kvl, first, n_my, qhead, g < heads_here, st, lane);
            else dense_direct<D, true>(p, kvl, first, n_my, qhead, g < heads_here, st, lane);
            const int new_tile = int(p.sink_len + p.res_len) / TILE;
            if (p.k_new && new_tile >= first && new_tile < first + n_my && lane < D / 8) {
                // the warp that owns the new token's tile stores its rows at the end of the recent-token buffer (the caller's slice
                // assignment, cache.py:632-672); head groups write the same bytes
                const int64_t dst = (int64_t(kvl) * p.res_ls + p.res_len) * D, src = int64_t(kvl) * D;
                reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.res_k_w) + dst)[lane] = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.k_new) + src)[lane];
                reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.res_v_w) + dst)[lane] = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.v_new) + src)[lane];
            }
        }
        cta_sync();
        store_partial<D, 0, PS>(my_part, st, heads_here, lane);
    }

    // ---------------- rotation back: this CTA's columns of R (and S), in flight under the folding ----------------
    // (Code behind the loop runs once per call, from a cold instruction cache: short rolled loops.  Fully unrolled: 11.6 us for the 8.4.)
    const int ncol = ((D + C - 1) / C + 1) & ~1, lp = max(32 - __clz(ncol - 1), 3), col0 = rank * ncol;    // columns per CTA; a power of two of threads for them
    const int kg = tid >> lp, oc = tid & ((1 << lp) - 1), KG = NT >> lp, n_k = QR / KG;            // (KG divides QR)
    const float* const r_col = p.rot + min(col0 + oc, D - 1);
    const float* const s_col = QJL ? p.qjl_proj + min(col0 + oc, D - 1) : nullptr;
    constexpr int U = 16;
    float rc[U];
    auto load_cols = [&](int i0) {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int k = kg + KG * (i0 + i);
            rc[i] = k < D ? __ldg(r_col + k * D) : QJL && k < QR ? __ldg(s_col + (k - D) * D) : 0.f;
        }
    };
    if (n_pw > 0) load_cols(0);
    __syncthreads();
    // ---------------- the CTA's warps: packed part (rotated space), uncompressed part ----------------
    const int n_e = heads_here * (QR / 4);                              // items: a head's four slots
    float* const ys = fp(P::Y);                                         // [QR + 1][HPG], by coordinate; a last row of zeros
    float* const yd = fp(P::YD);                                        // [HPG][D]: the uncompressed part, by slot (C = 1) or own columns
    float* const wt = fp(P::WT);                                        // [HPG][MAX_C + 4]: weights of the CTAs, then 1 / sum
    auto put_y = [&](int h, int c, const float4& y) {                   // four slots of the packed part, their scale taken back
        const bool split = p.vb_lo != 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = c >= D ? c + u : coord_of<D>(c + u, split);
            ys[k * HPG + h] = (&y.x)[u] * (c >= D ? QJL_C / D : 1.f / (split && k >= D / 2 ? p.v_scale_lo : p.v_scale_hi));
        }
    };
    if (tid < HPG) ys[QR * HPG + tid] = 0.f;
#pragma unroll 1
    for (int e = tid; e < n_e; e += NT) {
        const int h = e / (QR / 4), c = 4 * (e - h * (QR / 4));
        const float* src = red + h * PS;
        float M = -INFINITY, L = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) M = fmaxf(M, src[w * (HPG * PS) + QR]);
        float4 ap = make_float4(0.f, 0.f, 0.f, 0.f), ad = ap;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float2 ml = *reinterpret_cast<const float2*>(src + w * (HPG * PS) + QR);
            const float x = ml.x == -INFINITY ? 0.f : ex2(ml.x - M);
            const bool pk = rank * NW + w < n_pw;
            L = fmaf(x, ml.y, L);                                       // (weight 0 counts too: 0 x NaN is NaN, and a warp without tokens holds zeros)
            if (!pk && c >= D) continue;                                // (uncompressed tokens have no sketch rows)
            const float4 v = *reinterpret_cast<const float4*>(src + w * (HPG * PS) + c);
            if (pk) { ap.x = fmaf(x, v.x, ap.x); ap.y = fmaf(x, v.y, ap.y); ap.z = fmaf(x, v.z, ap.z); ap.w = fmaf(x, v.w, ap.w); }
            else { ad.x = fmaf(x, v.x, ad.x); ad.y = fmaf(x, v.y, ad.y); ad.z = fmaf(x, v.z, ad.z); ad.w = fmaf(x, v.w, ad.w); }
        }
        if (C > 1) {
            *reinterpret_cast<float4*>(fp(P::CP) + h * QR + c) = ap;
            if (c < D) *reinterpret_cast<float4*>(fp(P::CD) + h * D + c) = ad;
            if (c == 0) *reinterpret_cast<float2*>(fp(P::ML) + 2 * h) = make_float2(M, L);
        } else {
            put_y(h, c, ap);
            if (c < D) *reinterpret_cast<float4*>(yd + h * D + c) = ad;
            if (c == 0) wt[h * (MAX_C + 4) + MAX_C] = 1.f / L;
        }
    }
    // ---------------- the lane's CTAs, over distributed shared memory: every CTA merges all of the packed part, its columns of the other ----
    if (C > 1) {
        cluster_arrive();
        cluster_wait();
        const int n_pc = (n_pw + NW - 1) / NW, d_c0 = n_pw / NW;         // CTAs with packed tiles; the first with uncompressed ones
        const int n_d = heads_here * ncol;
        float4 v[4];
        float u[4];
        auto load_p = [&](int e, int r0) {
            const int h = e / (QR / 4), c = 4 * (e - h * (QR / 4));
#pragma unroll
            for (int r = 0; r < 4; ++r)
                v[r] = r0 + r < n_pc ? peer_f4(peer_addr(base + P::CP + uint32_t(h * QR + c) * 4u, r0 + r)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto load_d = [&](int e, int r0) {
            const int h = e / ncol, c = min(col0 + (e - h * ncol), D - 1);
            const uint32_t addr = base + P::CD + uint32_t(h * D + slot_of<D>(c)) * 4u;
#pragma unroll
            for (int r = 0; r < 4; ++r) u[r] = r0 + r < C ? peer_f1(peer_addr(addr, r0 + r)) : 0.f;
        };
        // one round trip: maxima and sums (sixteen threads a head), the first four sums of every item
        float2 x = make_float2(-INFINITY, 0.f);
        const int wh = tid / MAX_C, wr_ = tid % MAX_C, ed = NT - 1 - tid;
        if (wh < heads_here && wr_ < C) x = peer_f2(peer_addr(base + P::ML + 8u * uint32_t(wh), wr_));
        if (tid < n_e) load_p(tid, 0);
        if (ed < n_d) load_d(ed, d_c0);
        {
            float M = x.x;
#pragma unroll
            for (int off = 8; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
            const float w = x.x == -INFINITY ? 0.f : ex2(x.x - M);
            float sum = w * x.y;
#pragma unroll
            for (int off = 8; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (wh < HPG) {
                wt[wh * (MAX_C + 4) + wr_] = w;
                if (wr_ == 0) wt[wh * (MAX_C + 4) + MAX_C] = 1.f / sum;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int e = tid; e < n_e; e += NT) {
            const int h = e / (QR / 4), c = 4 * (e - h * (QR / 4));
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int r0 = 0; r0 < n_pc; r0 += 4) {
                if (r0 > 0 || e != tid) load_p(e, r0);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float w = wt[h * (MAX_C + 4) + min(r0 + r, MAX_C - 1)];       // (a sum that is not there counts 0, whatever its weight)
                    if (r0 + r >= n_pc) continue;
                    y.x = fmaf(w, v[r].x, y.x); y.y = fmaf(w, v[r].y, y.y); y.z = fmaf(w, v[r].z, y.z); y.w = fmaf(w, v[r].w, y.w);
                }
            }
            put_y(h, c, y);
        }
#pragma unroll 1
        for (int e = ed; e < n_d; e += NT) {
            const int h = e / ncol, c = e - h * ncol;
            float y = 0.f;
#pragma unroll 1
            for (int r0 = d_c0; r0 < C; r0 += 4) {
                if (r0 > d_c0 || e != ed) load_d(e, r0);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float w = wt[h * (MAX_C + 4) + min(r0 + r, MAX_C - 1)];
                    if (r0 + r < C) y = fmaf(w, u[r], y);
                }
            }
            yd[h * D + c] = y;
        }
    }
    __syncthreads();
    if (C > 1) cluster_arrive();                                        // (the peers' sums have been read)
    if (tid == 0 && rank == 0 && p.n_peers > 0) p.epochs[a] = epoch;
    // ---------------- y @ R (rotation.py:68-78), plus (c/d) z @ S (qjl.py:89-92): thread (k group, column) ----------------
    float acc[HPG];
#pragma unroll
    for (int h = 0; h < HPG; ++h) acc[h] = 0.f;
#pragma unroll 1
    for (int i0 = 0; n_pw > 0 && i0 < n_k; i0 += U) {
        if (i0 > 0) load_cols(i0);
#pragma unroll
        for (int j = 0; j < U; j += 4) {
            if (i0 + j >= n_k) break;
#pragma unroll
            for (int i = j; i < j + 4; ++i) {
                const float* y = ys + min(kg + KG * (i0 + i), QR) * HPG;
                const float4 x = *reinterpret_cast<const float4*>(y);
                acc[0] = fmaf(x.x, rc[i], acc[0]); acc[1] = fmaf(x.y, rc[i], acc[1]); acc[2] = fmaf(x.z, rc[i], acc[2]); acc[3] = fmaf(x.w, rc[i], acc[3]);
                if (heads_here > 4) {
                    const float4 z = *reinterpret_cast<const float4*>(y + 4);
                    acc[4] = fmaf(z.x, rc[i], acc[4]); acc[5] = fmaf(z.y, rc[i], acc[5]); acc[6] = fmaf(z.z, rc[i], acc[6]); acc[7] = fmaf(z.w, rc[i], acc[7]);
                }
            }
        }
    }
    float* const op = fp(P::OP);                                        // [KG][HPG][1 << lp]
#pragma unroll
    for (int h = 0; h < HPG; ++h)
        if (h < heads_here) op[(((kg * HPG) + h) << lp) + oc] = acc[h];
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < heads_here * (ncol / 2); e += NT) {           // two columns each
        const int h = e / (ncol / 2), j = 2 * (e - h * (ncol / 2)), c = col0 + j;
        if (c >= D) continue;
        const float* d0 = yd + h * D;
        float o[2] = {C > 1 ? d0[j] : d0[slot_of<D>(c)], C > 1 ? d0[j + 1] : d0[slot_of<D>(c + 1)]};
#pragma unroll 8
        for (int q = 0; q < KG; ++q) {
            const float2 x = *reinterpret_cast<const float2*>(op + (((q * HPG) + h) << lp) + j);
            o[0] += x.x; o[1] += x.y;
        }
        const float il = wt[h * (MAX_C + 4) + MAX_C];
        o[0] *= il; o[1] *= il;
        if (p.n_peers == 0) {
            const int64_t at = (q0 + h) * D + c;
            store_from_f32(p.out, p.out_dtype, at, o[0]);
            store_from_f32(p.out, p.out_dtype, at + 1, o[1]);
            continue;
        }
        // fused gather: the two elements in the result's type, sent to every peer as {payload, epoch} words
        const unsigned long long ep = static_cast<unsigned long long>(epoch) << 32;
        const int64_t at = (int64_t(b) * p.heads_total + p.head_offset + head0 + h) * D + c;
        const bool f32 = p.out_dtype == TQ_F32;
        const uint32_t w0 = f32 ? __float_as_uint(o[0]) : p.out_dtype == TQ_F16 ? pack_h2(o[0], o[1]) : pack_bf2(o[0], o[1]), w1 = __float_as_uint(o[1]);
        for (int q = 0; q < p.n_peers; ++q) {
            unsigned long long* dst = p.peer_ll[q] + (f32 ? at : at / 2);
            asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst), "l"(w0 | ep) : "memory");
            if (f32) asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst + 1), "l"(w1 | ep) : "memory");
        }
    }
    if (C > 1) cluster_wait();                                          // no CTA leaves while its sums may still be read
}

// ---- host side ------------------------------------------------------------------------------------------------
constexpr int SIZES[] = {1, 2, 3, 4, 5, 6, 8, 12, 16}, N_SIZES = 9;
// Clusters of each size that the device runs at once (all 0: the kernel cannot run here); looked up once per device.
struct Room { int clusters[N_SIZES]; };
template <int D, bool QJL, int PER_SM> static size_t smem_bytes() { return Plan<D, QJL, PER_SM>::END - dd::probe_smem_base(); }
template <int D, bool QJL, int PER_SM> static const Room& room() {
    static Room rooms[64];
    static std::atomic<int> known[64];
    static const Room none{};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return none;
    if (known[dev].load(std::memory_order_acquire)) return rooms[dev];
    Room r{};
    const unsigned sb = dd::probe_smem_base();
    if (sb == ~0u) return none;                                // (no answer this time, not no room: asked again at the next call)
    int max_optin = 0;
    auto kernel = decode_lane_kernel<D, QJL, PER_SM>;
    if (sb <= LO_BASE && (sb & 15u) == 0 && cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
        smem_bytes<D, QJL, PER_SM>() <= size_t(max_optin) &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes<D, QJL, PER_SM>())) == cudaSuccess) {
        const bool large = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        for (int i = 0; i < N_SIZES; ++i) {
            if (SIZES[i] > 8 && !large) break;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = unsigned(SIZES[i]); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(unsigned(SIZES[i]));
            cfg.blockDim = dim3(NT);
            cfg.dynamicSmemBytes = smem_bytes<D, QJL, PER_SM>();
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) r.clusters[i] = n;
        }
    }
    cudaGetLastError();
    // (two threads may both have looked it up: the same numbers)
    static std::mutex m;
    std::lock_guard<std::mutex> lock(m);
    if (!known[dev].load(std::memory_order_relaxed)) { rooms[dev] = r; known[dev].store(1, std::memory_order_release); }
    return rooms[dev];
}
static const Room& room(int d, bool qjl, int per_sm) {
    if (d == 256) return qjl ? room<256, true, 1>() : room<256, false, 1>();
    if (d == 64) return per_sm == 1 ? (qjl ? room<64, true, 1>() : room<64, false, 1>()) : (qjl ? room<64, true, 2>() : room<64, false, 2>());
    if (d == 96) return per_sm == 1 ? (qjl ? room<96, true, 1>() : room<96, false, 1>()) : (qjl ? room<96, true, 2>() : room<96, false, 2>());
    return per_sm == 1 ? (qjl ? room<128, true, 1>() : room<128, false, 1>()) : (qjl ? room<128, true, 2>() : room<128, false, 2>());
}
// Ring stages per warp beside the tables of the call's widths
template <int D, bool QJL, int PER_SM> static int stages(bool any3, int row_bytes) {
    using P = Plan<D, QJL, PER_SM>;
    return std::min(MAX_NS, int(((P::BARS - ring_base(any3)) / NW - 16u) / (P::SC + 16u * uint32_t(row_bytes))));
}
static int stages(int d, bool qjl, int per_sm, bool any3, int rows) {
    if (d == 256) return qjl ? stages<256, true, 1>(any3, rows) : stages<256, false, 1>(any3, rows);
    if (d == 64) return per_sm == 1 ? (qjl ? stages<64, true, 1>(any3, rows) : stages<64, false, 1>(any3, rows)) : (qjl ? stages<64, true, 2>(any3, rows) : stages<64, false, 2>(any3, rows));
    if (d == 96) return per_sm == 1 ? (qjl ? stages<96, true, 1>(any3, rows) : stages<96, false, 1>(any3, rows)) : (qjl ? stages<96, true, 2>(any3, rows) : stages<96, false, 2>(any3, rows));
    return per_sm == 1 ? (qjl ? stages<128, true, 1>(any3, rows) : stages<128, false, 1>(any3, rows)) : (qjl ? stages<128, true, 2>(any3, rows) : stages<128, false, 2>(any3, rows));
}

template <int D, bool QJL, int PER_SM> static int launch(const DecodeParams& p, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(p.B * p.Hkv * p.HG * p.ln_c));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem_bytes<D, QJL, PER_SM>();
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = p.pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = unsigned(p.ln_c); attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.ln_c > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_lane_kernel<D, QJL, PER_SM>, p);
    if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_decode_attn: %s", cudaGetErrorString(e));
    return TQ_OK;
}
template <int D> static int launch(const DecodeParams& p, cudaStream_t s) {
    const bool qjl = p.qjl_proj != nullptr;
    if constexpr (D == 256) return qjl ? launch<D, true, 1>(p, s) : launch<D, false, 1>(p, s);
    else if (p.ln_per_sm == 1) return qjl ? launch<D, true, 1>(p, s) : launch<D, false, 1>(p, s);
    else return qjl ? launch<D, true, 2>(p, s) : launch<D, false, 2>(p, s);
}

}  // namespace dl

// CTAs per lane, CTAs per SM, and the split of a cluster's warps between packed and uncompressed tiles.  Cost in us, fitted to 965 measured
// calls (log error 0.10): waves of clusters; per wave a base, the cluster's size, 4.2 at d = 128 once the CTAs leave no room for the next
// call's, whose tables are then no longer filled under this one (64 lanes x 34 tiles, 128 CTAs: 12.9; 8 x 38, 32 CTAs: 8.4), and the tiles
// of the busiest warp: twice as much each when two CTAs share an SM (32 lanes x 737 tiles at 3.5 bits: 32.8 with 128 CTAs, 33.3 with 256
// on as many SMs: clusters are packed onto pairs even where SMs are free); an uncompressed tile counts as 1.6.
// below: only a plan that costs less is of use.  A long context is turned away by a bound that takes no division: every warp has its share of
// the tiles at least, and so has every SM.  (Host time of a call's checks and choice: 8 lanes x 32,768 tokens 1.35 us with all plans made, 0.71 now, 0.61
// without this kernel; 8 lanes x 600, which it takes, 0.97 / 0.78 / 0.49.)
LanePlan lane_plan(int64_t lanes, int d, bool qjl, int kb_hi, int kb_lo, int vb_hi, int vb_lo, int64_t c_len, int64_t dense_len, int force_c, int sms, double below) {
    LanePlan best{};
    const int64_t p_tiles = (c_len + TILE - 1) / TILE, d_tiles = (dense_len + TILE - 1) / TILE;
    const bool any3 = kb_hi == 3 || kb_lo == 3 || vb_hi == 3 || vb_lo == 3;
    const int rows = c_len > 0 ? packed_bytes(kb_lo ? d / 2 : d, kb_hi) + (kb_lo ? packed_bytes(d / 2, kb_lo) : 0) + packed_bytes(vb_lo ? d / 2 : d, vb_hi) +
                                     (vb_lo ? packed_bytes(d / 2, vb_lo) : 0) : 0;
    if (lanes <= 0 || p_tiles + d_tiles == 0 || p_tiles + d_tiles > (int64_t(1) << 24)) return best;
    const int max_per_sm = d == 256 ? 1 : 2;
    const double dd = double(d) / 128.0, work = double(p_tiles) + 1.6 * double(d_tiles);       // packed tiles' worth
    double tile_us[3], least[3];                                       // per tile; per tile of a lane, at least, by the share of a warp and of an SM
    for (int per_sm = 1; per_sm <= max_per_sm; ++per_sm) {
        tile_us[per_sm] = 0.15 + (per_sm == 1 ? 0.61 : 1.29) * dd + 0.45 * dd * qjl + 0.09 * dd * (rows * 16 >= d * 13);
        least[per_sm] = tile_us[per_sm] / dl::NW * std::max(1.0 / dl::MAX_C, double(lanes) / double(sms * per_sm));
    }
    if (2.25 + 5.4 * dd + work * std::min(least[1], least[max_per_sm]) >= below) return best;
    const dl::Room* room[3];
    int ns[3];
    for (int per_sm = 1; per_sm <= max_per_sm; ++per_sm) {
        room[per_sm] = &dl::room(d, qjl, per_sm);
        ns[per_sm] = dl::stages(d, qjl, per_sm, any3, rows);
    }
    best.cost = below;
    for (int i = 0; i < dl::N_SIZES; ++i) {
        const int c = dl::SIZES[i], nw = dl::NW * c;
        if (force_c > 0 ? c != force_c : c > 1 && dl::NW * dl::SIZES[i - 1] >= p_tiles + d_tiles) continue;       // (a tile per warp already)
        if (lanes * c >= (int64_t(1) << 31)) break;
        if (2.1 + 0.15 * c + 5.4 * dd + work / nw * std::min(tile_us[1], tile_us[max_per_sm]) >= best.cost * 1.000001) continue;
        // packed warps so that both kinds take as long; costs in tenths of a packed tile
        const int64_t dc = d_tiles * 16, w0 = nw * p_tiles * 10 / (p_tiles * 10 + dc);
        const int lo = p_tiles > 0 ? 1 : 0, hi = d_tiles > 0 ? nw - 1 : nw;
        auto load = [&](int w) { return std::max<int64_t>(w > 0 ? (p_tiles + w - 1) / w * 10 : 0, nw > w ? (d_tiles + nw - w - 1) / (nw - w) * 16 : 0); };
        int pw = nw;
        if (nw > 1) {
            pw = std::clamp(int(w0), lo, hi);
            if (pw + 1 <= hi && load(pw + 1) < load(pw)) ++pw;
            else if (pw - 1 >= lo && load(pw - 1) < load(pw)) --pw;
        }
        const double tiles = 0.1 * double(load(pw));
        for (int per_sm = 1; per_sm <= max_per_sm; ++per_sm) {
            // (the last few clusters of pairs do not find their places: 72 lanes x 4 CTAs, of 74 that fit, take two waves)
            const int fit = room[per_sm]->clusters[i], at_once = per_sm == 2 && c > 2 ? fit * 15 / 16 : fit;
            if (at_once == 0 || ns[per_sm] < 2) continue;              // (two stages at least: 3.5 / 3.5 bits with sketches have an SM to themselves)
            const int64_t waves = (lanes + at_once - 1) / at_once;
            const double full = std::clamp((double(lanes) / double(at_once) - 0.4) / 0.3, 0.0, 1.0);
            const double cost = double(waves) * (2.1 + 0.15 * c + 5.4 * dd + full * (1.3 + 2.9 * dd) + tile_us[per_sm] * tiles);
            if (cost >= best.cost) continue;
            best.c = c; best.per_sm = per_sm; best.ns = ns[per_sm]; best.cost = cost;
            best.pw = int(std::min<int64_t>(pw, p_tiles)); best.dw = int(std::min<int64_t>(nw - pw, d_tiles));
        }
    }
    return best;
}

int launch_decode_lane(const DecodeParams& p, cudaStream_t s) {
    if (p.D == 64) return dl::launch<64>(p, s);
    if (p.D == 96) return dl::launch<96>(p, s);
    return p.D == 128 ? dl::launch<128>(p, s) : dl::launch<256>(p, s);
}

}  // namespace tq
