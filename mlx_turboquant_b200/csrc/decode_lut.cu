// Decode attention for the widths and head dims without a kernel of their own: keys and values at 2, 3 or 4 bits or a
// fractional split (4 | 3 or 3 | 2 bits), head_dim 64 / 96 / 128 / 256, with or without the QJL sign sketches.
//
// One persistent CTA per SM; the packed 16-token tiles of ALL cache lanes (sequence, KV head, head group) are dealt out as
// one flat sequence, an equal contiguous run per warp (as decode_stream.cu does for 4-bit keys / 2-bit values).  Two
// launches chained with programmatic dependent launch: decode_lut_kernel and lut_merge_kernel (log-sum-exp merge, rotation
// back, normalisation).  A CTA rotates the queries of its lanes itself where it has two lanes at most; many short lanes, and a
// fused gather, have lut_query_kernel rotate all of them in a launch before (on mma.sync).
//
// Operands come from shared-memory tables: decode_lut.cuh.
//   (The general kernel of decode.cu takes codes one by one through a 16-entry table and shared-memory staging: 906 us per
//   call for 4 sequences x 8 KV heads x 11,777 tokens at 3.5 / 3.5 bits.)
//
// Tiles reach a warp through its own ring of NS stages in shared memory (16-byte asynchronous copies, an mbarrier per
// stage).  A lane reads the bits it owns of a row as aligned words and shifts them into place, so any row length works.
//
// Partials.  Long lanes (a CTA's tiles span at most two of them): the warps of a CTA fold their partials of a lane into
// one before it leaves the SM, so that few lanes of many tiles do not flood the merge.  Short lanes: a warp writes a
// partial per lane it touches.
//
// Every mbarrier wait is bounded; a wait that runs out records a status (tq_device_status), the warp drains the copies it
// still has in flight (bounded again) and stops.
#include <algorithm>
#include <atomic>

#include "decode_lut.cuh"

namespace tq {
namespace lut {

constexpr int ERR_RING = 109, ERR_LAYOUT = 110;
constexpr int MAX_PARTS = 192;                 // partial slots per lane the merge handles

// Shared-window addresses are compile-time constants (they travel in the instructions): the dynamic allocation starts at
// sbase <= LO_BASE.
constexpr uint32_t LO_BASE = 2048u;
using Tab = Tables<LO_BASE>;
constexpr uint32_t AREA0 = Tab::END;

template <int D, bool QJL> struct Plan {
    static constexpr int NW = D == 256 ? 8 : 16, NT = NW * 32;                       // (d = 256: 128 accumulator / query registers per thread)
    static constexpr uint32_t SC = (QJL ? 6u : 2u) * TILE * 4u;                      // scalars first: norms, sign words, residual norms
    static constexpr uint32_t O_KN = 0, O_VN = 64, O_KB = 128, O_KG = 192, O_VB = 256, O_VG = 320;
    static constexpr uint32_t STAGE = SC + 2u * TILE * D / 2;                        // 4-bit keys and values fill it
    static constexpr int NC = (int(STAGE / 16) + 31) / 32;                           // 16-byte chunks per lane at most
    static constexpr int NS = 3;
    static constexpr uint32_t RING = NS * STAGE + 16u;                               // (+ a word that is read but not used past the last row)
    static constexpr uint32_t DSTAGE = 2u * TILE * stage_ld<D>() * 2u;               // 16-bit keys + values of one uncompressed tile
    static constexpr uint32_t PART = HPG * (D + QM + 4) * 4u;                        // one warp's partial of up to eight heads
    static constexpr uint32_t A0 = RING > DSTAGE ? RING : DSTAGE;
    static constexpr uint32_t AREA = ((A0 > PART ? A0 : PART) + 127u) / 128u * 128u;
    static constexpr uint32_t SPILL = AREA0 + NW * AREA;                             // partial of the lane a warp leaves (one warp per CTA can)
    static constexpr uint32_t BARS = SPILL + (PART + 127u) / 128u * 128u;
    static constexpr uint32_t OWNER = BARS + 8u * NW * NS;                           // lane of each warp's partial, then of the spilled one
    static constexpr uint32_t META = (OWNER + 4u * (NW + 1) + 15u) / 16u * 16u;      // per lane of a folding CTA: its heads, first query head, partial slot
    static constexpr uint32_t QROT = META + 32u;                                     // rotated queries (and sketches) of the CTA's two lanes
    static constexpr int QR = D + (QJL ? QM : 0);                                    // halves per head there
    static constexpr uint32_t QLANE = HPG * QR * 2u;                                 // bytes per lane, eight heads
    static constexpr uint32_t QCAP = 227u * 1024u - QROT < 2u * QLANE ? 227u * 1024u - QROT : 2u * QLANE;
    static constexpr uint32_t SMEM_END = QROT + QCAP;
    static_assert(SMEM_END <= 227u * 1024u, "shared-memory plan");
    static_assert(STAGE % 16 == 0 && AREA % 128 == 0, "copies need 16-byte alignment");
};

// Query heads in the workspace, halves: rotated | sketch (launches whose CTAs do not rotate their own)
__host__ __device__ constexpr int q_stride(int d) { return d + QM; }
__host__ __device__ constexpr int part_stride(int d) { return d + QM + 4; }    // floats per head of a partial: values | sketch rows | max, sum, pad

// Uncompressed tokens (sink, recent window, the token a step appends) of cache lane kvl, tiles [tile_lo, tile_hi), 16-bit
// caches: a tile's rows come in with asynchronous copies and feed the MMAs in their own type.  bf16 rows take the
// query and the weights as high + low bf16 parts (16 bits between them), so nothing is converted and any magnitude works.
template <int D, bool BF16>
__device__ __forceinline__ void dense_run(const DecodeParams& p, int64_t kvl, int tile_lo, int tile_hi, uint32_t stage, int64_t qhead, bool live_q,
                                          WarpAcc<D, 0>& st, int lane) {
    constexpr int LD = stage_ld<D>(), CPR = D / 8;                       // halves per staged row, 16-byte chunks per row
    const int g = lane >> 2, t = lane & 3;
    const int n_tok = int(p.sink_len + p.res_len) + (p.k_new ? 1 : 0);
    uint32_t bh[D / 16][2], bl[BF16 ? D / 16 : 1][2];
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = ks * 16 + 2 * t + 8 * u;
            const float2 x = live_q ? q_pair(p, qhead, c) : make_float2(0.f, 0.f);
            if (BF16) {
                bh[ks][u] = pack_bf2(x.x, x.y);
                bl[ks][u] = pack_bf2(x.x - __uint_as_float(bh[ks][u] << 16), x.y - __uint_as_float(bh[ks][u] & 0xffff0000u));
            } else {
                bh[ks][u] = pack_h2(x.x, x.y);
            }
        }
    const uint32_t vstage = stage + TILE * LD * 2;
    // rows of one side of a tile; the warp that owns the new token's tile also stores the row at the end of the recent-token
    // buffer (the caller's slice assignment, cache.py:632-672); head groups write the same bytes
    auto load = [&](int tile, uint32_t dst, const void* sink, const void* res, const void* neu, void* res_w) {
        const int tok0 = tile * TILE, s_len = int(p.sink_len), r_len = int(p.res_len);
        if (tile < tile_hi && tok0 < n_tok) {
#pragma unroll 4
            for (int i = lane; i < TILE * CPR; i += 32) {
                const int r = i / CPR, c = i - r * CPR, tok = tok0 + r, rr = tok - s_len;
                const bool in_sink = tok < s_len, fresh = rr >= r_len;
                const int64_t e = in_sink ? (kvl * p.sink_ls + tok) * D : fresh ? kvl * D : (kvl * p.res_ls + rr) * D;
                const uint16_t* base = static_cast<const uint16_t*>(in_sink ? sink : fresh ? neu : res);
                const int n = tok < n_tok ? 16 : 0;                          // rows past the end are zero-filled
                const uint16_t* src = n ? base + e + c * 8 : reinterpret_cast<const uint16_t*>(p.rot);
                cp_async16(dst + (r * LD + c * 8) * 2, src, n);
                if (n && fresh && !in_sink)
                    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(res_w) + (kvl * p.res_ls + r_len) * D + c * 8) = __ldg(reinterpret_cast<const uint4*>(src));
            }
        }
        cp_async_commit();
    };
    // the next tile's keys are on their way from when this one's have been used, its values likewise
    load(tile_lo, stage, p.sink_k, p.res_k, p.k_new, p.res_k_w);
    load(tile_lo, vstage, p.sink_v, p.res_v, p.v_new, p.res_v_w);
    for (int tile = tile_lo; tile < tile_hi; ++tile) {
        const int tok0 = tile * TILE;
        if (tok0 >= n_tok) break;
        cp_async_wait<1>();
        __syncwarp();
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t ka = stage + ((lane & 15) * LD + (lane >> 4) * 8) * 2;
        auto ldsm = [](uint32_t (&r)[4], uint32_t addr) {
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
        };
        auto ldsm_t = [](uint32_t (&r)[4], uint32_t addr) {
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
        };
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t a[4];
            ldsm(a, ka + ks * 32);
            if (BF16) { mma_bf16(s, a, bh[ks][0], bh[ks][1]); mma_bf16(s, a, bl[ks][0], bl[ks][1]); }
            else mma16816(s, a[0], a[1], a[2], a[3], bh[ks][0], bh[ks][1]);
        }
        const bool ok0 = tok0 + g < n_tok, ok1 = tok0 + g + 8 < n_tok;
        s[0] = ok0 ? s[0] : -INFINITY; s[1] = ok0 ? s[1] : -INFINITY;
        s[2] = ok1 ? s[2] : -INFINITY; s[3] = ok1 ? s[3] : -INFINITY;
        __syncwarp();
        load(tile + 1, stage, p.sink_k, p.res_k, p.k_new, p.res_k_w);
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
        cp_async_wait<1>();
        __syncwarp();
        const uint32_t vaddr = vstage + (((lane & 7) + ((lane >> 4) & 1) * 8) * LD + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
        for (int mt = 0; mt < D / 16; ++mt) {
            uint32_t a[4];
            ldsm_t(a, vaddr + mt * 32);
            if (BF16) { mma_bf16(st.o[mt], a, bp[0], bp[1]); mma_bf16(st.o[mt], a, bpl[0], bpl[1]); }
            else mma16816(st.o[mt], a[0], a[1], a[2], a[3], bp[0], bp[1]);
        }
        __syncwarp();
        load(tile + 1, vstage, p.sink_v, p.res_v, p.v_new, p.res_v_w);
    }
    cp_async_wait<0>();
}

// The launch before the persistent grid when its CTAs do not rotate their own queries: many short lanes, or a fused gather.
// Grid (eight heads, groups of four warps' slabs).
template <int D>
__global__ void __launch_bounds__(128) lut_query_kernel(DecodeParams p) {
    constexpr int QS = q_stride(D), KS = D / 16;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int slab = blockIdx.y * 4 + (threadIdx.x >> 5), n_slabs = KS + (p.qjl_proj ? 2 : 0);
    const int64_t n_q = int64_t(p.B) * p.Hq, q0 = int64_t(blockIdx.x) * 8;
    pdl_trigger();
    float2 rr[KS][4];
    load_rows<D>(p, min(slab, n_slabs - 1), g, t, rr);       // constants, so they are in registers before the wait
    pdl_wait();
    await_gather(p);   // (head-sharded decoding) the peers' heads of an earlier call have arrived
    if (p.n_peers > 0 && blockIdx.y == 0) {           // this call's epoch of every group, for the merge launch
        const int n_groups = p.B * p.Hkv * p.HG;
        for (int i = blockIdx.x * 128 + threadIdx.x; i < n_groups; i += gridDim.x * 128) ++p.epochs[i];
    }
    float y[4];
    rotate_rows<D>(p, q0, n_q - q0, g, t, rr, y);
    if (slab >= n_slabs) return;
#pragma unroll
    for (int r = 0; r < 4; ++r) {              // rows g, g + 8 of the slab x heads 2t, 2t + 1
        const int64_t h = q0 + 2 * t + (r & 1);
        if (h < n_q) p.st_q16[h * QS + slab * 16 + g + (r >> 1) * 8] = __float2half_rn(y[r]);
    }
}

// ---- launch 2: the persistent grid ----------------------------------------------------------------------
// INQ: the CTA rotates the queries of its lanes itself.
template <int D, bool QJL, bool INQ>
__global__ void __launch_bounds__(Plan<D, QJL>::NT, 1) decode_lut_kernel(DecodeParams p) {
    using P = Plan<D, QJL>;
    constexpr int NZ = QJL ? QM / 16 : 0, NS = P::NS, NW = P::NW, NT = P::NT, NC = P::NC;
    constexpr int QS = q_stride(D), PS = part_stride(D);
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    auto gp = [&](uint32_t addr) -> unsigned char* { return smem + (addr - sbase); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    if (sbase > LO_BASE || (sbase & 15u)) {            // cannot happen after the host-side probe; never run on a bad plan
        if (tid == 0) atomicCAS(p.status, 0, ERR_LAYOUT);
        return;
    }
    pdl_trigger();
    const uint32_t bar0 = P::BARS + 8u * uint32_t(warp) * NS, my_area = AREA0 + uint32_t(warp) * P::AREA;
    int* owner = reinterpret_cast<int*>(gp(P::OWNER));
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < NS; ++s) mbar_init(bar0 + 8u * s, 32);      // every lane arrives when its copies into the stage have completed
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        owner[warp] = -1;
        if (warp == 0) owner[NW] = -1;
    }
    const int kf = fmt_of(p.kb_hi, p.kb_lo), vf = fmt_of(p.vb_hi, p.vb_lo);
    // ---------------- tables: constants only, before the wait for the previous launch ----------------
    if (p.c_len > 0) fill_tables<Tab, NT>(p, tid, gp);
    const int L = p.B * p.Hkv * p.HG;                          // cache lanes x head groups
    const int n_tiles = int((p.c_len + TILE - 1) / TILE);      // packed tiles per lane
    const bool fold = p.st_fold != 0;                          // the warps of the CTA fold their partials of a lane into one
    const uint32_t total = uint32_t(L) * n_tiles, range = uint32_t(p.st_range), unit = fold ? range * NW : range;       // (below 2^31) unit: tiles behind one partial slot
    const int n_slots = p.st_npp + p.st_nd;                    // partial slots per lane
    const int wg = blockIdx.x * NW + warp, n_warps = gridDim.x * NW;
    const int c_len = int(p.c_len);
    auto heads_of = [&](int a) { return min(HPG, p.G - (a % p.HG) * HPG); };
    auto qhead_of = [&](int a) -> int {                        // first query head of lane a
        const int kvl = a / p.HG, hg = a - kvl * p.HG, b = kvl / p.Hkv, hkv = kvl - b * p.Hkv;
        return b * p.Hq + hkv * p.G + hg * HPG;
    };
    // Everything that follows from the parameters alone is worked out before the wait: integer divisions in code that is cold
    // in the instruction cache cost 5 us of a small call after it.
    int a_first = 0, n_la = 0;                                 // (if it folds) the lanes of the CTA's tiles: two at most
    int4* meta = reinterpret_cast<int4*>(gp(P::META));
    if (fold) {
        const uint32_t c0 = min(blockIdx.x * unit, total), c1 = min(c0 + unit, total);
        a_first = c0 < c1 ? int(c0 / uint32_t(n_tiles)) : 0;
        n_la = c0 < c1 ? int((c1 - 1) / uint32_t(n_tiles)) - a_first + 1 : 0;
        if (tid < n_la) meta[tid] = make_int4(heads_of(a_first + tid), qhead_of(a_first + tid), int(blockIdx.x) - int(uint32_t(a_first + tid) * n_tiles / unit), 0);
    }
    // uncompressed tokens: items i in [i0, i1) of the L * nd (lane, run of dt tiles) pairs, dealt from the far end: with few
    // items the warps that have none are the ones whose packed runs are full
    const uint32_t n_items = uint32_t(L) * p.st_nd, wr = uint32_t(n_warps - 1 - wg);
    const uint32_t i0 = (wr * n_items + n_warps - 1) / n_warps, i1 = ((wr + 1) * n_items + n_warps - 1) / n_warps;
    int da = p.st_nd > 0 ? int(i0 / uint32_t(p.st_nd)) : 0, dpart = int(i0) - da * p.st_nd, dheads = heads_of(da), dq = qhead_of(da);
    // ---------------- queries of the CTA's lanes, by units: sixteen rows of R (or S) x the heads of a lane ----------------
    constexpr int SLABS = D / 16 + (QJL ? QM / 16 : 0);
    const int n_units = INQ ? n_la * SLABS : 0;
    float2 rr[D / 16][4];
    if (INQ && warp < n_units) load_rows<D>(p, warp % SLABS, g, t, rr);           // constants as well
    __syncthreads();
    pdl_wait();        // the prepared queries, the cache and the workspace are settled from here on
    bool failed = false;

    __half* qrot = reinterpret_cast<__half*>(gp(P::QROT));
    for (int un = warp; un < n_units; un += NW) {
        const int la = un / SLABS, slab = un - la * SLABS;
        const int4 lm = meta[la];
        if (un != warp) load_rows<D>(p, slab, g, t, rr);
        float y[4];
        rotate_rows<D>(p, lm.y, lm.x, g, t, rr, y);
#pragma unroll
        for (int r = 0; r < 4; ++r) {              // rows g, g + 8 of the slab x heads 2t, 2t + 1
            const int h = 2 * t + (r & 1);
            if (h < p.slots) qrot[(la * p.slots + h) * P::QR + slab * 16 + g + (r >> 1) * 8] = __float2half_rn(y[r]);
        }
    }
    if (INQ) __syncthreads();

    // ---------------- uncompressed tokens ----------------
    {
        for (uint32_t i = i0; i < i1; ++i) {
            const int a = da, part = dpart, heads_here = dheads;
            const int64_t qhead = dq + min(g, heads_here - 1);
            if (++dpart == p.st_nd) { dpart = 0; ++da; dheads = heads_of(da); dq = qhead_of(da); }
            WarpAcc<D, 0> sd;
            sd.init();
            if (p.dense_dtype == TQ_F16) {
                dense_run<D, false>(p, a / p.HG, part * p.st_dt, (part + 1) * p.st_dt, my_area, qhead, g < heads_here, sd, lane);
            } else if (p.dense_dtype == TQ_BF16) {
                dense_run<D, true>(p, a / p.HG, part * p.st_dt, (part + 1) * p.st_dt, my_area, qhead, g < heads_here, sd, lane);
            } else {
                uint32_t bq[D / 16][2];
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float2 x = q_pair(p, qhead, ks * 16 + 2 * t + 8 * u);
                        bq[ks][u] = g < heads_here ? pack_h2(x.x, x.y) : 0u;
                    }
                }
                __half* Ks = reinterpret_cast<__half*>(gp(my_area));
                dense_tiles<D, 1, 0>(p, a / p.HG, int64_t(part) * p.st_dt, int64_t(part + 1) * p.st_dt, Ks, Ks + TILE * stage_ld<D>(), bq, sd, 0, lane);
            }
            sd.finish();
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) {
                sd.l[0] += __shfl_xor_sync(0xffffffffu, sd.l[0], off);
                sd.l[1] += __shfl_xor_sync(0xffffffffu, sd.l[1], off);
            }
            float* pp = p.st_part + (int64_t(a) * n_slots + p.st_npp + part) * p.slots * PS;
            if (2 * t < heads_here) {
                const bool two = 2 * t + 1 < heads_here;
                float* h0 = pp + (2 * t) * PS;
                float* h1 = h0 + PS;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {           // rows are coordinates mt * 16 + g and + 8
                    const int c = mt * 16 + g;
                    h0[c] = sd.o[mt][0]; h0[c + 8] = sd.o[mt][2];
                    if (two) { h1[c] = sd.o[mt][1]; h1[c + 8] = sd.o[mt][3]; }
                }
                if (g == 0) {
                    h0[D + QM] = sd.m[0]; h0[D + QM + 1] = sd.l[0];
                    if (two) { h1[D + QM] = sd.m[1]; h1[D + QM + 1] = sd.l[1]; }
                }
            }
            __syncwarp();
        }
    }

    // ---------------- packed tokens: flat tiles [T0, T1) of the L * n_tiles ----------------------------------
    const uint32_t T0 = min(uint32_t(wg) * range, total), T1 = min(T0 + range, total);
    const int n_my = int(T1 - T0);
    if (n_my > 0) {
        const int kwh = packed_bytes(p.kb_lo ? D / 2 : D, p.kb_hi), kwl = p.kb_lo ? packed_bytes(D / 2, p.kb_lo) : 0;
        const int vwh = packed_bytes(p.vb_lo ? D / 2 : D, p.vb_hi), vwl = p.vb_lo ? packed_bytes(D / 2, p.vb_lo) : 0;
        // A stage holds the tile's scalars, then its key rows (first part, second part) and value rows, back to back; lane l
        // copies 16-byte chunks l, l + 32, ...  (16 rows of w bytes are w chunks.)  Sources advance by 16 rows per tile.
        const int n_sc = int(P::SC / 16), n_chunks = n_sc + kwh + kwl + vwh + vwl;
        const unsigned char* cp_ptr[NC];
        uint32_t cp_step[NC];
        int ia = int(T0 / uint32_t(n_tiles)), iti = int(T0) - ia * n_tiles;    // lane and tile of the next copy
        {
            const int64_t row = int64_t(ia / p.HG) * p.c_ls + int64_t(iti) * TILE;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                int c = lane + 32 * j, rb;
                const unsigned char* base = chunk_source(p, c, n_sc, kwh, kwl, vwh, rb);
                cp_ptr[j] = base + row * rb + 16 * c;
                cp_step[j] = lane + 32 * j < n_chunks ? uint32_t(TILE * rb) : 0u;
            }
        }
        auto issue = [&](int stage) {
            const uint32_t bar = bar0 + 8u * stage, dst = my_area + uint32_t(stage) * P::STAGE + 16u * lane;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                if (cp_step[j]) cp_async16(dst + 512u * j, cp_ptr[j], 16);
                cp_ptr[j] += cp_step[j];
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
            if (++iti == n_tiles) {          // the next copy starts the next lane: same rows again (next head group) or the next lane's storage
                const int64_t jump = ((ia + 1) / p.HG != ia / p.HG ? p.c_ls : 0) - int64_t(n_tiles) * TILE;
#pragma unroll
                for (int j = 0; j < NC; ++j) cp_ptr[j] += jump * int64_t(cp_step[j] / TILE);
                iti = 0; ++ia;
            }
        };
        __syncwarp();
#pragma unroll 1
        for (int n = 0; n < min(n_my, NS); ++n) issue(n);

        const Copies cpy{uint32_t(lane * 4), uint32_t((lane & 15) * 8)};
        const TileLayout ly = tile_layout<P, D>(p, lane);
        int a = int(T0 / uint32_t(n_tiles)), ti = int(T0) - a * n_tiles;       // lane and tile being computed
        int slot = int(T0 / unit) - int(uint32_t(a) * n_tiles / unit);       // partial slot = rank of this warp (CTA) among the lane's
        int heads_here = 0;
        uint32_t bq[D / 16][2];
        uint32_t bu[QM / 16][2];
        auto load_query = [&]() {
            heads_here = fold ? meta[a - a_first].x : heads_of(a);
            const __half* qh = INQ ? qrot + ((a - a_first) * p.slots + g) * P::QR : p.st_q16 + (qhead_of(a) + g) * QS;
            // this lane's coordinates of k-step ks: four in a row
            const bool split = p.kb_lo != 0;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const int c = split ? (ks < D / 32 ? t * (D / 8) + 4 * ks : D / 2 + t * (D / 8) + 4 * (ks - D / 32)) : t * (D / 4) + 4 * ks;
                // (written by the launch before this one while this grid may already have been resident: read at L2, never through a non-coherent path)
                uint2 x = make_uint2(0u, 0u);
                if (g < heads_here) x = INQ ? *reinterpret_cast<const uint2*>(qh + c) : __ldcg(reinterpret_cast<const uint2*>(qh + c));
                bq[ks][0] = x.x; bq[ks][1] = x.y;
            }
            if (QJL) {
                // k slot (ks, register hh, half e) of lane t stands for sketch row 4t + 2ks + hh + 16e: the halves of an
                // operand register are then bits 16 apart in a token's sign word
#pragma unroll
                for (int ks = 0; ks < QM / 16; ++ks)
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int pi = 4 * t + 2 * ks + hh;
                        bu[ks][hh] = 0u;
                        if (g < heads_here) {
                            const unsigned short* z = reinterpret_cast<const unsigned short*>(qh + D + pi);
                            const unsigned short lo16 = INQ ? z[0] : __ldcg(z), hi16 = INQ ? z[16] : __ldcg(z + 16);
                            bu[ks][hh] = uint32_t(lo16) | (uint32_t(hi16) << 16);
                        }
                    }
            }
        };
        WarpAcc<D, NZ> st;
        st.init();
        load_query();
        // one partial (up to eight heads of PS floats) to dst: values, sketch rows, maximum, sum
        auto write_partial = [&](float* dst) {
            st.finish();
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) {
                st.l[0] += __shfl_xor_sync(0xffffffffu, st.l[0], off);
                st.l[1] += __shfl_xor_sync(0xffffffffu, st.l[1], off);
            }
            if (2 * t < heads_here) {
                const bool two = 2 * t + 1 < heads_here, split = p.vb_lo != 0;
                float* h0 = dst + (2 * t) * PS;
                float* h1 = h0 + PS;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {              // rows g, g + 8 of m-tile mt: two coordinates in a row of this lane's share
                    const int c = split ? (mt < D / 32 ? g * (D / 16) + 2 * mt : D / 2 + g * (D / 16) + 2 * (mt - D / 32)) : g * (D / 8) + 2 * mt;
                    *reinterpret_cast<float2*>(h0 + c) = make_float2(st.o[mt][0], st.o[mt][2]);
                    if (two) *reinterpret_cast<float2*>(h1 + c) = make_float2(st.o[mt][1], st.o[mt][3]);
                }
#pragma unroll
                for (int mz = 0; mz < NZ; ++mz) {
                    h0[D + 16 * mz + g] = st.z[mz][0]; h0[D + 16 * mz + g + 8] = st.z[mz][2];
                    if (two) { h1[D + 16 * mz + g] = st.z[mz][1]; h1[D + 16 * mz + g + 8] = st.z[mz][3]; }
                }
                if (g == 0) {
                    h0[D + QM] = st.m[0]; h0[D + QM + 1] = st.l[0];
                    if (two) { h1[D + QM] = st.m[1]; h1[D + QM + 1] = st.l[1]; }
                }
            }
        };
        auto slot_ptr = [&]() -> float* { return p.st_part + (int64_t(a) * n_slots + slot) * p.slots * PS; };

#pragma unroll 1
        for (int n = 0, stage = 0, phase = 0; n < n_my; ++n) {
            const uint32_t sa = my_area + uint32_t(stage) * P::STAGE;
            if (!__all_sync(0xffffffffu, mbar_wait(bar0 + 8u * stage, uint32_t(phase)))) {
                // the copies never landed: record it, drain what is still in flight (bounded), stop - nothing may land in
                // this CTA's memory after it has gone
                atomicCAS(p.status, 0, ERR_RING);
                failed = true;
                for (int m = n + 1; m < min(n_my, n + NS); ++m) mbar_wait(bar0 + 8u * (m % NS), uint32_t(m / NS) & 1u);
                break;
            }

            packed_tile<Tab, P, D, QJL>(sa, ly, bq, bu, cpy, c_len - ti * TILE, st, lane);

            // ---- the stage is free: ask for the tile NS further on ----
            if (n + NS < n_my) {
                __syncwarp();
                issue(stage);
            }
            if (++stage == NS) { stage = 0; phase ^= 1; }
            if (++ti == n_tiles) {       // the next tile belongs to the next lane
                if (!fold) {
                    write_partial(slot_ptr());
                    ti = 0; ++a; slot = 0;
                    if (n + 1 < n_my) { st.init(); load_query(); }
                } else if (n + 1 < n_my) {               // this warp is the CTA's one that crosses into the next lane
                    write_partial(reinterpret_cast<float*>(gp(P::SPILL)));
                    if (lane == 0) owner[NW] = a;
                    ti = 0; ++a;
                    st.init();
                    load_query();
                }
            }
        }
        if (!failed) {
            if (fold) {
                __syncwarp();
                write_partial(reinterpret_cast<float*>(gp(my_area)));        // (the ring is drained: every copy was waited for)
                if (lane == 0) owner[warp] = a;
            } else if (ti != 0) write_partial(slot_ptr());
        }
    }
    if (!fold) return;

    // ---------------- fold: one partial per (CTA, lane), from the warps' partials in shared memory ----------------
    __syncthreads();
    // (the tables are free: every warp has left its loop)  Weights: a warp per (lane, head), lane w of it = partial w.
    constexpr int NE = D + (QJL ? QM : 0), FW = 20;
    float* fw = reinterpret_cast<float*>(gp(Tab::B));
    auto partial_of = [&](int w, int h) -> const float* {
        return reinterpret_cast<const float*>(gp(w < NW ? AREA0 + uint32_t(w) * P::AREA : P::SPILL)) + h * PS;
    };
    auto dst_of = [&](int la) -> float* {
        return p.st_part + (int64_t(a_first + la) * n_slots + meta[la].z) * p.slots * PS;
    };
    for (int i = warp; i < n_la * p.slots; i += NW) {
        const int la = i >= p.slots ? 1 : 0, h = i - la * p.slots;
        const bool mine = lane <= NW && owner[lane <= NW ? lane : 0] == a_first + la && h < meta[la].x;
        const float* src = partial_of(lane <= NW ? lane : 0, h);
        const float m = mine ? src[D + QM] : -INFINITY, l = mine ? src[D + QM + 1] : 0.f;
        float M = m;
#pragma unroll
        for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        const float w = m == -INFINITY ? 0.f : ex2(m - M);
        float sum = w * l;
#pragma unroll
        for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane <= NW) fw[i * FW + lane] = w;
        if (lane == 0 && h < meta[la].x) *reinterpret_cast<float2*>(dst_of(la) + h * PS + D + QM) = make_float2(M, sum);
    }
    __syncthreads();
    for (int e = tid; e < n_la * p.slots * (NE / 4); e += NT) {
        const int i = e / (NE / 4), c = 4 * (e - i * (NE / 4)), la = i >= p.slots ? 1 : 0, h = i - la * p.slots;
        if (h >= meta[la].x) continue;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w <= NW; ++w) {
            const float x = fw[i * FW + w];
            // (a partial of another lane has weight 0 and may hold anything: skipped, not multiplied)
            const float4 v = x != 0.f ? *reinterpret_cast<const float4*>(partial_of(w, h) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            acc.x = fmaf(x, v.x, acc.x); acc.y = fmaf(x, v.y, acc.y); acc.z = fmaf(x, v.z, acc.z); acc.w = fmaf(x, v.w, acc.w);
        }
        *reinterpret_cast<float4*>(dst_of(la) + h * PS + c) = acc;
    }
}

// ---- launch 3: merge --------------------------------------------------------------------------------------
// Latency is all there is to it: one round trip for the partials' maxima and sums together with the first sixteen partials
// of every thread, one step of weights, one of sums, one of rotation.  A block takes `rp` (lane, query head) rows at a time
// (1, 2 or 4): its NG groups of D threads share a row's slots NG / rp ways.  The rotation back (y @ R, rotation.py:68-78; plus
// (c/d) z @ S for the sketches, qjl.py:89-92) is float32: thread (k group, column) holds its quarter of the column of R in
// registers from before the wait.  (R staged in shared memory by every block, a thread per coordinate over all slots: 12 to
// 20 us per launch whatever the size; now 5 to 7.)  d = 256: two blocks share a row's columns.
template <int D> __host__ __device__ constexpr int merge_cols() { return D > 128 ? 128 : D; }
template <int D> __host__ __device__ constexpr int merge_threads() { return 4 * merge_cols<D>(); }
template <int D, bool QJL>
__global__ void __launch_bounds__(merge_threads<D>(), 1) lut_merge_kernel(DecodeParams p, int nw, int rp) {
    constexpr int PS = part_stride(D), NT = merge_threads<D>(), NCOL = merge_cols<D>(), NG = NT / D, KR = D / 4, SR = QJL ? QM / 4 : 0, U = 16;
    __shared__ float s_w[4][MAX_PARTS], s_il[4];
    __shared__ __align__(16) float s_a[4][D + QM], s_p[2][NG][D], s_o[4][4][NCOL];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_trigger();
    const int n0 = blockIdx.y * NCOL, kg = tid / NCOL, oc = tid - kg * NCOL;       // rotation: k group, output column
    float rr[KR], sr[SR ? SR : 1];
#pragma unroll
    for (int j = 0; j < KR; ++j) rr[j] = __ldg(p.rot + (kg * KR + j) * D + n0 + oc);
#pragma unroll
    for (int j = 0; j < SR; ++j) sr[j] = __ldg(p.qjl_proj + (kg * SR + j) * D + n0 + oc);
    const int n_tiles = int((p.c_len + TILE - 1) / TILE);
    const int n_slots = p.st_npp + p.st_nd;
    const uint32_t unit = uint32_t(p.st_fold ? p.st_range * nw : p.st_range);       // (fewer than 2^31 tiles in all)
    const uint32_t n_rows = uint32_t(p.B * p.Hkv * p.HG * p.slots), slots = uint32_t(p.slots);
    const int sstride = p.slots * PS;
    const int sg = tid / D, c = tid - sg * D, ns = NG / rp, r_of = sg / ns, part = sg - r_of * ns;      // sums: row of the pass, share of its slots
    for (uint32_t row0 = blockIdx.x * uint32_t(rp); row0 < n_rows; row0 += gridDim.x * uint32_t(rp)) {
        auto row_ptr = [&](int r) -> const float* {                   // the row's first partial
            const uint32_t i = min(row0 + r, n_rows - 1), a = i / slots;
            return p.st_part + (int64_t(a) * n_slots * p.slots + (i - a * slots)) * PS;
        };
        auto row_live = [&](int r) -> bool {
            const uint32_t i = row0 + r, a = i / slots;
            return i < n_rows && int(i - a * slots) < min(HPG, p.G - int(a % uint32_t(p.HG)) * HPG);
        };
        const float* src = row_ptr(r_of) + c;
        const uint32_t wa = min(row0 + min(warp, rp - 1), n_rows - 1) / slots;
        // the warps (CTAs) whose runs touch this lane's tiles [wa * n_tiles, (wa + 1) * n_tiles)
        const int n_pp = n_tiles > 0 ? int(((wa + 1) * uint32_t(n_tiles) - 1) / unit) - int((wa * uint32_t(n_tiles)) / unit) + 1 : 0;
        const bool live = row_live(min(warp, rp - 1));
        const float* ml_src = row_ptr(min(warp, rp - 1)) + D + QM;
        if (row0 == blockIdx.x * uint32_t(rp)) pdl_wait();            // (everything above only needs the parameters)
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = part + ns * u < n_slots ? __ldcg(src + (part + ns * u) * sstride) : 0.f;
        if (warp < rp) {
            constexpr int NI = (MAX_PARTS + 31) / 32;
            float2 ml[NI];
            float M = -INFINITY, sum = 0.f;
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                ml[k] = make_float2(-INFINITY, 0.f);
                if (32 * k >= n_slots) continue;
                const int j = lane + 32 * k;
                const bool valid = live && j < n_slots && (j < n_pp || j >= p.st_npp);
                ml[k] = valid ? __ldcg(reinterpret_cast<const float2*>(ml_src + j * sstride)) : make_float2(-INFINITY, 0.f);
            }
#pragma unroll
            for (int k = 0; k < NI; ++k) M = fmaxf(M, ml[k].x);
#pragma unroll
            for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                if (32 * k >= n_slots) continue;
                const int j = lane + 32 * k;
                const float w = ml[k].x == -INFINITY ? 0.f : ex2(ml[k].x - M);
                sum = fmaf(w, ml[k].y, sum);
                if (j < n_slots) s_w[warp][j] = w;
            }
#pragma unroll
            for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (lane == 0) s_il[warp] = 1.f / sum;
        }
        __syncthreads();
        // weighted sums: the packed part in rotated space, the uncompressed part.  A slot without a partial has weight 0 and
        // whatever bytes the workspace holds: it is skipped, not multiplied.
        float ar = 0.f, ad = 0.f;
        auto add = [&](int i, float x) {
            const float w = i < n_slots ? s_w[r_of][i] : 0.f;
            const float y = w != 0.f ? w * x : 0.f;
            if (i < p.st_npp) ar += y; else ad += y;
        };
#pragma unroll
        for (int u = 0; u < U; ++u) add(part + ns * u, v[u]);
#pragma unroll 1
        for (int i0 = part + ns * U; i0 < n_slots; i0 += ns * U) {
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = i0 + ns * u < n_slots ? __ldcg(src + (i0 + ns * u) * sstride) : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) add(i0 + ns * u, v[u]);
        }
        s_p[0][sg][c] = ar;
        s_p[1][sg][c] = ad;
        if (QJL) {
            for (int e = tid; e < rp * QM; e += NT) {
                const int r = e / QM, z = e - r * QM;
                const float* zs = row_ptr(r) + D + z;
                float az = 0.f;
#pragma unroll 8
                for (int i = 0; i < p.st_npp; ++i) {
                    const float w = s_w[r][i];
                    const float x = __ldcg(zs + i * sstride);
                    az += w != 0.f ? w * x : 0.f;
                }
                s_a[r][D + z] = az * (QJL_C / D);
            }
        }
        __syncthreads();
        for (int e = tid; e < rp * D; e += NT) {
            const int r = e / D, k = e - r * D;
            float x = 0.f;
            for (int q = 0; q < ns; ++q) x += s_p[0][r * ns + q][k];
            s_a[r][k] = x * (1.f / (p.vb_lo != 0 && k >= D / 2 ? p.v_scale_lo : p.v_scale_hi));
        }
        __syncthreads();
        for (int r = 0; r < rp; ++r) {
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int j = 0; j < KR; j += 4) {
                const float4 q = *reinterpret_cast<const float4*>(&s_a[r][kg * KR + j]);
                x = fmaf(q.x, rr[j], x); y = fmaf(q.y, rr[j + 1], y); x = fmaf(q.z, rr[j + 2], x); y = fmaf(q.w, rr[j + 3], y);
            }
#pragma unroll
            for (int j = 0; j < SR; ++j) x = fmaf(s_a[r][D + kg * SR + j], sr[j], x);
            s_o[kg][r][oc] = x + y;
        }
        __syncthreads();
        for (int e = tid; e < rp * (NCOL / 2); e += NT) {              // two columns each
            const int r = e / (NCOL / 2), o0 = 2 * (e - r * (NCOL / 2)), col = n0 + o0;
            if (!row_live(r)) continue;
            float o[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float x = (s_o[0][r][o0 + u] + s_o[1][r][o0 + u]) + (s_o[2][r][o0 + u] + s_o[3][r][o0 + u]);
                for (int q = 0; q < ns; ++q) x += s_p[1][r * ns + q][col + u];
                o[u] = x * s_il[r];
            }
            const int ir = int(row0) + r;
            const int a = ir / p.slots, h = ir - a * p.slots, kvl = a / p.HG, hg = a - kvl * p.HG, b = kvl / p.Hkv, hkv = kvl - b * p.Hkv;
            const int head = hkv * p.G + hg * HPG + h;
            if (p.n_peers == 0) {
                const int64_t at = (int64_t(b) * p.Hq + head) * D + col;
                store_from_f32(p.out, p.out_dtype, at, o[0]);
                store_from_f32(p.out, p.out_dtype, at + 1, o[1]);
                continue;
            }
            // fused gather: the two elements in the result's type, sent to every peer as {payload, epoch} words (the query launch
            // counted the call)
            const unsigned long long epoch = static_cast<unsigned long long>(p.epochs[a]) << 32;
            const int64_t at = (int64_t(b) * p.heads_total + p.head_offset + head) * D + col;
            const bool f32 = p.out_dtype == TQ_F32;
            const uint32_t w0 = f32 ? __float_as_uint(o[0]) : p.out_dtype == TQ_F16 ? pack_h2(o[0], o[1]) : pack_bf2(o[0], o[1]), w1 = __float_as_uint(o[1]);
            for (int q = 0; q < p.n_peers; ++q) {
                unsigned long long* dst = p.peer_ll[q] + (f32 ? at : at / 2);
                asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst), "l"(w0 | epoch) : "memory");
                if (f32) asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst + 1), "l"(w1 | epoch) : "memory");
            }
        }
        __syncthreads();
    }
}

// ---- host side ------------------------------------------------------------------------------------------------
template <int D, bool QJL> static bool fits() {
    const unsigned sb = dd::probe_smem_base();
    if (sb == ~0u || sb > LO_BASE || (sb & 15u)) return false;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return false;
    return size_t(Plan<D, QJL>::SMEM_END - sb) <= size_t(max_optin);
}

template <int D, bool QJL> static int launch(const DecodeParams& p, cudaStream_t s) {
    using P = Plan<D, QJL>;
    const size_t smem = P::SMEM_END - dd::probe_smem_base();
    static std::atomic<bool> set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !set[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(decode_lut_kernel<D, QJL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_lut_kernel<D, QJL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_decode_attn: shared memory %zu B: %s", smem, cudaGetErrorString(e));
        set[dev].store(true, std::memory_order_release);
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = p.pdl ? 1 : 0;
    cudaLaunchConfig_t cfg{};
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int64_t n_q = int64_t(p.B) * p.Hq;
    cudaError_t e = cudaSuccess;
    // CTAs that touch two lanes at most rotate those lanes' queries themselves: it takes them 2 us, a launch 5 (with four
    // lanes: 8)
    const bool inq = p.n_peers == 0 && !p.await_ll && (p.c_len == 0 || (p.st_fold && 2u * uint32_t(p.slots) * P::QR * 2u <= P::QCAP));
    if (!inq) {
        cfg.gridDim = dim3(unsigned((n_q + 7) / 8), unsigned((D / 16 + (QJL ? 2 : 0) + 3) / 4));
        cfg.blockDim = dim3(128);
        e = cudaLaunchKernelEx(&cfg, lut_query_kernel<D>, p);
    }
    if (e == cudaSuccess) {
        cfg.gridDim = dim3(unsigned(p.st_grid));
        cfg.blockDim = dim3(P::NT);
        cfg.dynamicSmemBytes = smem;
        e = inq ? cudaLaunchKernelEx(&cfg, decode_lut_kernel<D, QJL, true>, p) : cudaLaunchKernelEx(&cfg, decode_lut_kernel<D, QJL, false>, p);
    }
    if (e == cudaSuccess) {
        // one row at a time spreads few rows over the SMs and many slots over a block; else as many as the groups share evenly
        const int64_t rows = int64_t(p.B) * p.Hkv * p.HG * p.slots;
        constexpr int NG = merge_threads<D>() / D;
        const int n_slots = p.st_npp + p.st_nd;
        const int rp = rows <= p.st_grid || n_slots > 32 ? 1 : std::min(NG, n_slots > 16 ? 2 : 4);
        cfg.gridDim = dim3(unsigned(std::min<int64_t>((rows + rp - 1) / rp, 4 * int64_t(p.st_grid))), D / merge_cols<D>());
        cfg.blockDim = dim3(merge_threads<D>());
        cfg.dynamicSmemBytes = 0;
        e = cudaLaunchKernelEx(&cfg, lut_merge_kernel<D, QJL>, p, P::NW, rp);
    }
    if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_decode_attn: %s", cudaGetErrorString(e));
    return TQ_OK;
}

}  // namespace lut

static bool lut_width(int hi, int lo) { return lo ? (hi == 4 && lo == 3) || (hi == 3 && lo == 2) : hi >= 2 && hi <= 4; }

bool lut_supported(int d, bool qjl, int kb_hi, int kb_lo, int vb_hi, int vb_lo) {
    if (!lut_width(kb_hi, kb_lo) || !lut_width(vb_hi, vb_lo)) return false;
    if (d == 64) return qjl ? lut::fits<64, true>() : lut::fits<64, false>();
    if (d == 96) return qjl ? lut::fits<96, true>() : lut::fits<96, false>();
    if (d == 128) return qjl ? lut::fits<128, true>() : lut::fits<128, false>();
    if (d == 256) return qjl ? lut::fits<256, true>() : lut::fits<256, false>();
    return false;
}

StreamPlan lut_plan(int batch, int n_q_heads, int n_kv_heads, int d, int64_t c_len, int64_t dense_len, int sms) {
    StreamPlan s{};
    const int nw = d == 256 ? 8 : 16;
    const int G = n_q_heads / n_kv_heads, hg = (G + HPG - 1) / HPG;
    const int64_t L = int64_t(batch) * n_kv_heads * hg;
    const int64_t p_tiles = (c_len + TILE - 1) / TILE, d_tiles = (dense_len + TILE - 1) / TILE;
    s.grid = sms;
    const int64_t n_warps = int64_t(s.grid) * nw;
    s.range = std::max<int64_t>((L * p_tiles + n_warps - 1) / n_warps, 1);
    // a CTA's run of tiles no longer than a lane: it touches two lanes at most and folds its warps' partials
    s.fold = p_tiles >= s.range * nw ? 1 : 0;
    const int64_t unit = s.fold ? s.range * nw : s.range;
    s.npp = p_tiles > 0 ? int((p_tiles + unit - 1) / unit) + 1 : 0;
    if (d_tiles > 0) {
        int64_t nd = std::min<int64_t>(d_tiles, std::max<int64_t>(n_warps / L, 1));
        s.dt = int((d_tiles + nd - 1) / nd);
        s.nd = int((d_tiles + s.dt - 1) / s.dt);
    }
    s.q16_bytes = (size_t(batch) * n_q_heads * lut::q_stride(d) * sizeof(__half) + 255) / 256 * 256;
    s.part_bytes = size_t(L) * size_t(s.npp + s.nd) * size_t(std::min(G, HPG)) * lut::part_stride(d) * sizeof(float);
    s.ok = s.npp + s.nd <= lut::MAX_PARTS && (L + 1) * (p_tiles + 1) < (int64_t(1) << 31) && L < (int64_t(1) << 20) && dense_len < (int64_t(1) << 30);
    return s;
}

int launch_decode_lut(const DecodeParams& p, cudaStream_t s) {
    const bool qjl = p.qjl_proj != nullptr;
    if (p.D == 64) return qjl ? lut::launch<64, true>(p, s) : lut::launch<64, false>(p, s);
    if (p.D == 96) return qjl ? lut::launch<96, true>(p, s) : lut::launch<96, false>(p, s);
    if (p.D == 128) return qjl ? lut::launch<128, true>(p, s) : lut::launch<128, false>(p, s);
    return qjl ? lut::launch<256, true>(p, s) : lut::launch<256, false>(p, s);
}

}  // namespace tq
