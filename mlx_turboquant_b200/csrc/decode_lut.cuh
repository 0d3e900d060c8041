// Device code shared by the kernels that turn packed codes into operand registers through lookup tables in shared memory
// (decode_lut.cu: persistent grid over many tiles; decode_lane.cu: a cluster per cache lane in one launch): the tables, the products of a
// 16-token tile, the rotation of the queries.
//
// Operands.  What bounds a decode step at these widths is how packed codes become fp16 operand registers, so no code is
// ever looked at on its own: one shared-memory lookup turns a PAIR of codes (4 bits: a byte; 3 bits: a six-bit field) or
// four codes (2 bits: a byte) into one or two half2 registers, every lane reading its own copy of the table (no bank
// conflicts).  Keys pair neighbouring coordinates of a token, as the A operand of S = K q^T wants them; values pair the
// same coordinate of two tokens, as the A operand of O^T = V^T P^T wants them - the codes of two tokens are interleaved
// with one three-input logic op per eight (bytes at 4 and 2 bits; alternate octal digits at 3 bits).  Per 16-token tile,
// d = 128 and lane: 32 half2 a side = 32 lookups at 4 bits, 32 at 3 bits, 16 (of 64 bits) at 2 bits.
#pragma once

#include "decode_dev.cuh"

namespace tq {
namespace lut {

constexpr int QM = 32;                         // sketch rows (one 32-bit sign word per token)
constexpr float QJL_C = 1.2533141373155003f;   // sqrt(pi / 2), qjl.py:91-92
constexpr uint32_t WAIT_LIMIT = 4u << 20;

// Code formats of a side: the bits of its coordinates, or of its two halves (hi * 10 + lo).
enum Fmt { F2 = 2, F3 = 3, F4 = 4, F43 = 43, F32 = 32 };
__device__ __forceinline__ int fmt_of(int hi, int lo) { return lo ? hi * 10 + lo : hi; }

// Byte tables: slot e (256 B) holds the key entry of byte e (32 copies of a half2 at 4 bits, 16 of a pair of half2 at 2 bits), then the
// value entry likewise; the six-bit tables have 64 entries of 128 B.  Their shared-window addresses travel in the instructions.
template <uint32_t BASE> struct Tables {
    static constexpr uint32_t B = BASE, K3 = BASE + 65536u, V3 = K3 + 8192u, END = V3 + 8192u;
};

// ---- PTX wrappers ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i)
        if (mbar_try(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Table lookups: the table's address is an immediate of the load.
template <uint32_t OFF> __device__ __forceinline__ uint32_t tab32(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1 + %2];" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}
template <uint32_t OFF> __device__ __forceinline__ uint2 tab64(uint32_t addr) {
    uint2 v;
    asm("ld.shared.v2.b32 {%0,%1}, [%2 + %3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFF));
    return v;
}
// Ring reads: ordered after the wait that made the stage visible.
template <uint32_t OFF> __device__ __forceinline__ uint32_t ring32o(uint32_t base) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1 + %2];" : "=r"(v) : "r"(base), "n"(OFF) : "memory");
    return v;
}
template <uint32_t OFF> __device__ __forceinline__ float ring_f32o(uint32_t base) { return __uint_as_float(ring32o<OFF>(base)); }
template <int LUT> __device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return d;
}
// (a & m) | (b & ~m)
__device__ __forceinline__ uint32_t pick(uint32_t a, uint32_t b, uint32_t m) { return lop3<0xE4>(a, b, m); }
// half2 of two signs (+1 for a set bit) from bits 15 and 31
__device__ __forceinline__ uint32_t sign_pair16(uint32_t x) { return lop3<0x6A>(x, 0x80008000u, 0xBC00BC00u); }

// Token in MMA row / k slot s: slots 2a + e of a half hold tokens a + 4 e, so the four lanes of a thread group read value
// rows of four consecutive tokens and the eight row groups key rows of eight consecutive tokens.
__device__ __forceinline__ int tok_of_slot(int s) { return ((s & 7) >> 1) + 4 * (s & 1) + (s & 8); }

// Compile-time loop: f(Ic<0>{}), f(Ic<1>{}), ...
template <int I> struct Ic { static constexpr int v = I; };
template <int N, int I = 0, typename F> __device__ __forceinline__ void each(F&& f) {
    if constexpr (I < N) {
        f(Ic<I>{});
        each<N, I + 1>(f);
    }
}

__host__ __device__ constexpr int gcd32(int x) { return x % 32 == 0 ? 32 : x % 16 == 0 ? 16 : x % 8 == 0 ? 8 : x % 4 == 0 ? 4 : x % 2 == 0 ? 2 : 1; }
__host__ __device__ constexpr int words_of(int bits) { return (bits + 31) / 32; }
// BITS bits that start `sh` bits into the word at addr (shared memory), as words; sh is a multiple of gcd(BITS, 32).
template <int BITS> __device__ __forceinline__ void read_bits(uint32_t* w, uint32_t addr, uint32_t sh) {
    constexpr int NW = words_of(BITS);
    if constexpr (BITS % 128 == 0) {
        each<NW / 4>([&](auto ic) {
            constexpr int i = 4 * decltype(ic)::v;
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4 + %5];" : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]) : "r"(addr), "n"(4 * i) : "memory");
        });
    } else if constexpr (BITS == 64) {
        asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr) : "memory");
    } else {
        constexpr bool ALIGNED = BITS % 32 == 0;
        constexpr int NR = ALIGNED ? NW : (32 - gcd32(BITS) + BITS + 31) / 32;     // words that can hold a part of them
        uint32_t r[NR + 1];
        each<NR>([&](auto ic) {
            constexpr int i = decltype(ic)::v;
            r[i] = ring32o<4 * i>(addr);
        });
        r[NR] = 0;
#pragma unroll
        for (int i = 0; i < NW; ++i) w[i] = ALIGNED ? r[i] : NR == 1 ? r[i] >> sh : __funnelshift_r(r[i], r[i + 1], sh);
    }
}
// bits [P, ...) of NW words moved to bit TO; callers mask
template <int NW, int P, int TO> __device__ __forceinline__ uint32_t bits_at(const uint32_t* w) {
    constexpr int base = P - TO;
    if constexpr (base < 0) return w[0] << (-base);
    else {
        constexpr int i = base / 32, r = base % 32;
        if constexpr (r == 0) return w[i];
        else if constexpr (i + 1 < NW) return __funnelshift_r(w[i], w[i + 1], r);
        else return w[i] >> r;
    }
}
// Per-lane constants: copy offsets inside an entry (and the upper half of the tables' address, where that is not zero).
struct Copies { uint32_t c4, c2; };            // 4 lane, 8 (lane & 15)
constexpr uint32_t M3 = 63u << 7;              // six-bit field in entry position

// Scores of NK k-steps: this lane's 4 NK coordinates (B bits each, `sh` bits into the word at `addr`) of token row g, and of
// row g + 8, `row8` bytes further.  bq: the query fragments of these k-steps.
template <typename T, int B, int NK>
__device__ __forceinline__ void key_part(float (&s)[4], uint32_t addr, uint32_t row8, uint32_t sh, const uint32_t (*bq)[2], const Copies& c) {
    constexpr int NW = words_of(4 * NK * B);
    uint32_t a[NW], b[NW];
    read_bits<4 * NK * B>(a, addr, sh);
    read_bits<4 * NK * B>(b, addr + row8, sh);
    each<NK>([&](auto ic) {
        constexpr int ks = decltype(ic)::v;
        uint32_t a0, a1, a2, a3;
        if constexpr (B == 4) {
            constexpr uint32_t s0 = 0x7604u | uint32_t((2 * ks) & 3) << 4, s1 = 0x7604u | uint32_t((2 * ks + 1) & 3) << 4;
            a0 = tab32<T::B>(__byte_perm(a[ks / 2], c.c4, s0));
            a1 = tab32<T::B>(__byte_perm(b[ks / 2], c.c4, s0));
            a2 = tab32<T::B>(__byte_perm(a[ks / 2], c.c4, s1));
            a3 = tab32<T::B>(__byte_perm(b[ks / 2], c.c4, s1));
        } else if constexpr (B == 3) {
            a0 = tab32<T::K3>((bits_at<NW, 12 * ks, 7>(a) & M3) | c.c4);
            a1 = tab32<T::K3>((bits_at<NW, 12 * ks, 7>(b) & M3) | c.c4);
            a2 = tab32<T::K3>((bits_at<NW, 12 * ks + 6, 7>(a) & M3) | c.c4);
            a3 = tab32<T::K3>((bits_at<NW, 12 * ks + 6, 7>(b) & M3) | c.c4);
        } else {
            constexpr uint32_t s0 = 0x7604u | uint32_t(ks & 3) << 4;
            const uint2 x = tab64<T::B>(__byte_perm(a[ks / 4], c.c2, s0)), y = tab64<T::B>(__byte_perm(b[ks / 4], c.c2, s0));
            a0 = x.x; a2 = x.y; a1 = y.x; a3 = y.y;
        }
        mma16816(s, a0, a1, a2, a3, bq[ks][0], bq[ks][1]);
    });
}

// O^T += V^T P^T for MT m-tiles: this lane's 2 MT coordinates of tokens t, t + 4 (k slots 2t, 2t + 1) and t + 8, t + 12;
// token rows `row4` bytes apart.
template <typename T, int B, int MT>
__device__ __forceinline__ void value_part(float (*o)[4], uint32_t addr, uint32_t row4, uint32_t sh, const uint32_t (&bp)[2], const Copies& c) {
    constexpr int NW = words_of(2 * MT * B);
    uint32_t va[NW], vb[NW], vc[NW], vd[NW];
    read_bits<2 * MT * B>(va, addr, sh);
    read_bits<2 * MT * B>(vb, addr + row4, sh);
    read_bits<2 * MT * B>(vc, addr + 2 * row4, sh);
    read_bits<2 * MT * B>(vd, addr + 3 * row4, sh);
    if constexpr (B == 3) {
        constexpr uint32_t even = 0x1C71C7u;                     // octal digits 0, 2, 4, 6
        each<(MT + 3) / 4>([&](auto ic) {                        // groups of eight coordinates (24 bits)
            constexpr int gq = decltype(ic)::v;
            const uint32_t a = bits_at<NW, 24 * gq, 0>(va), b = bits_at<NW, 24 * gq, 0>(vb), cc = bits_at<NW, 24 * gq, 0>(vc), d = bits_at<NW, 24 * gq, 0>(vd);
            const uint32_t e0 = pick(a, b << 3, even), o0 = pick(a >> 3, b, even), e1 = pick(cc, d << 3, even), o1 = pick(cc >> 3, d, even);
            each<4>([&](auto jc) {
                constexpr int j = decltype(jc)::v, m = 4 * gq + j;
                if constexpr (m < MT) {
                    auto idx = [&](uint32_t x) -> uint32_t {
                        if constexpr (j < 2) return ((x << (7 - 6 * j)) & M3) | c.c4;
                        else return ((x >> (6 * j - 7)) & M3) | c.c4;
                    };
                    mma16816(o[m], tab32<T::V3>(idx(e0)), tab32<T::V3>(idx(o0)), tab32<T::V3>(idx(e1)), tab32<T::V3>(idx(o1)), bp[0], bp[1]);
                }
            });
        });
    } else {
        constexpr uint32_t low = 0x0F0F0F0Fu;
        each<NW>([&](auto ic) {
            constexpr int w = decltype(ic)::v;
            const uint32_t z0 = pick(va[w], vb[w] << 4, low), z1 = pick(va[w] >> 4, vb[w], low);
            const uint32_t y0 = pick(vc[w], vd[w] << 4, low), y1 = pick(vc[w] >> 4, vd[w], low);
            each<4>([&](auto jc) {
                constexpr int j = decltype(jc)::v;
                constexpr uint32_t sel = 0x7604u | uint32_t(j) << 4;
                if constexpr (B == 4) {                          // byte j of z0 / z1: coordinates 8 w + 2 j, + 1 of the two tokens
                    constexpr int m = 4 * w + j;
                    if constexpr (m < MT)
                        mma16816(o[m], tab32<T::B + 128>(__byte_perm(z0, c.c4, sel)), tab32<T::B + 128>(__byte_perm(z1, c.c4, sel)),
                              tab32<T::B + 128>(__byte_perm(y0, c.c4, sel)), tab32<T::B + 128>(__byte_perm(y1, c.c4, sel)), bp[0], bp[1]);
                } else {                                         // byte j of z0: coordinates 16 w + 4 j, + 1 of the two tokens; z1: + 2, + 3
                    constexpr int m = 8 * w + 2 * j;
                    if constexpr (m < MT) {
                        const uint2 e = tab64<T::B + 128>(__byte_perm(z0, c.c2, sel)), f = tab64<T::B + 128>(__byte_perm(y0, c.c2, sel));
                        mma16816(o[m], e.x, e.y, f.x, f.y, bp[0], bp[1]);
                    }
                    if constexpr (m + 1 < MT) {
                        const uint2 e = tab64<T::B + 128>(__byte_perm(z1, c.c2, sel)), f = tab64<T::B + 128>(__byte_perm(y1, c.c2, sel));
                        mma16816(o[m + 1], e.x, e.y, f.x, f.y, bp[0], bp[1]);
                    }
                }
            });
        });
    }
}

// Query elements c, c + 1 of a head times scale * log2(e)
__device__ __forceinline__ float2 q_pair(const DecodeParams& p, int64_t head, int c) {
    const int64_t e = head * p.D + c;
    const float f = p.scale * LOG2E;
    float2 x;
    if (p.q_dtype == TQ_F32) x = *reinterpret_cast<const float2*>(static_cast<const float*>(p.q) + e);
    else {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.q) + e);
        if (p.q_dtype == TQ_F16) x = __half22float2(*reinterpret_cast<const __half2*>(&w));
        else x = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    return make_float2(x.x * f, x.y * f);
}

// Softmax step on scores that already carry the key norms (and the sketch term); tokens past the end come in with score
// -inf and norm 0.  pr: the four weights times the value scale.
template <int D, int NZ>
__device__ __forceinline__ void softmax_scores(float (&s)[4], float vn0, float vn1, float vx, WarpAcc<D, NZ>& st, float (&pr)[4]) {
    const float mx0 = fmaxf(s[0], s[2]), mx1 = fmaxf(s[1], s[3]), vmax = fmaxf(fmaxf(vn0, vn1), vx);
    if (__any_sync(0xffffffffu, mx0 > st.mt[0] || mx1 > st.mt[1] || vmax > st.vt)) softmax_refresh<D, NZ>(mx0, mx1, vmax, st);
    const float p0 = ex2(s[0] - st.m[0]), p1 = ex2(s[1] - st.m[1]), p2 = ex2(s[2] - st.m[0]), p3 = ex2(s[3] - st.m[1]);
    st.l[0] += p0 + p2;
    st.l[1] += p1 + p3;
    pr[0] = p0 * st.vsc; pr[1] = p1 * st.vsc; pr[2] = p2 * st.vsc; pr[3] = p3 * st.vsc;
}

// A stage of a warp's ring holds a tile's scalars (n_sc 16-byte chunks), then its key rows (first part, second part) and value rows, back
// to back (16 rows of w bytes are w chunks).  Array that chunk c comes from, c made relative to the array's tile, bytes of its rows.
__device__ __forceinline__ const unsigned char* chunk_source(const DecodeParams& p, int& c, int n_sc, int kwh, int kwl, int vwh, int& rb) {
    if (c < n_sc) {
        const int arr = c >> 2;
        rb = 4; c &= 3;
        return reinterpret_cast<const unsigned char*>(arr == 0 ? static_cast<const void*>(p.k_norms) : arr == 1 ? static_cast<const void*>(p.v_norms)
                                                      : arr == 2 ? static_cast<const void*>(p.k_qbits) : arr == 3 ? static_cast<const void*>(p.k_qgamma)
                                                      : arr == 4 ? static_cast<const void*>(p.v_qbits) : static_cast<const void*>(p.v_qgamma));
    }
    c -= n_sc; rb = kwh;
    if (c < kwh) return p.k_hi;
    c -= kwh; rb = kwl;
    if (c < kwl) return p.k_lo;
    c -= kwl; rb = vwh;
    if (c < vwh) return p.v_hi;
    c -= vwh; rb = p.vb_lo ? packed_bytes(p.D / 2, p.vb_lo) : 0;
    return p.v_lo;
}

// Where a lane's share of a tile's arrays starts in a stage of its ring: scalars, key rows (first part, second part), value rows.
struct TileLayout {
    uint32_t tok;                              // scalars of the token in MMA row g
    uint32_t k0, k1, v0, v1, ksh0, ksh1, vsh0, vsh1;      // byte offset of the word and the bit shift inside it
    int kwh, kwl, vwh, vwl, kf, vf;            // bytes of a key row's parts, of a value row's; formats
};
template <typename P, int D> __device__ __forceinline__ TileLayout tile_layout(const DecodeParams& p, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const int kwh = packed_bytes(p.kb_lo ? D / 2 : D, p.kb_hi), kwl = p.kb_lo ? packed_bytes(D / 2, p.kb_lo) : 0;
    const int vwh = packed_bytes(p.vb_lo ? D / 2 : D, p.vb_hi), vwl = p.vb_lo ? packed_bytes(D / 2, p.vb_lo) : 0;
    const int tokA = tok_of_slot(g);           // tokens of MMA rows g and g + 8: tokA, tokA + 8
    TileLayout f;
    f.kf = fmt_of(p.kb_hi, p.kb_lo); f.vf = fmt_of(p.vb_hi, p.vb_lo);
    f.tok = 4u * tokA;
    f.kwh = kwh; f.kwl = kwl; f.vwh = vwh; f.vwl = vwl;
    // key rows tokA of the first / second part (a lane's share: a quarter of the coordinates), value rows t (its share: an eighth)
    auto word_at = [](uint32_t bit, uint32_t base, uint32_t& sh) -> uint32_t { sh = bit & 31u; return base + (bit >> 5) * 4u; };
    const uint32_t o_k = P::SC, o_kl = o_k + 16u * kwh, o_v = o_kl + 16u * kwl, o_vl = o_v + 16u * vwh;
    f.k0 = word_at(8u * (tokA * kwh) + 2u * kwh * t, o_k, f.ksh0);
    f.k1 = word_at(8u * (tokA * kwl) + 2u * kwl * t, o_kl, f.ksh1);
    f.v0 = word_at(8u * (t * vwh) + uint32_t(vwh * g), o_v, f.vsh0);
    f.v1 = word_at(8u * (t * vwl) + uint32_t(vwl * g), o_vl, f.vsh1);
    return f;
}

// One packed tile in the stage at `sa`: scores, softmax, values (and sketches).  Only `left` of its tokens are in the cache.
template <typename T, typename P, int D, bool QJL, int NZ = QJL ? QM / 16 : 0>
__device__ __forceinline__ void packed_tile(uint32_t sa, const TileLayout& f, const uint32_t (&bq)[D / 16][2], const uint32_t (&bu)[QM / 16][2], const Copies& cpy,
                                            int left, WarpAcc<D, NZ>& st, int lane) {
    const int g = lane >> 2, t = lane & 3, tokA = tok_of_slot(g);
    // ---- scores: S[token][head] = K . q^T ----
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    if (f.kf == F4) key_part<T, 4, D / 16>(s, sa + f.k0, 8u * f.kwh, f.ksh0, bq, cpy);
    else if (f.kf == F3) key_part<T, 3, D / 16>(s, sa + f.k0, 8u * f.kwh, f.ksh0, bq, cpy);
    else if (f.kf == F2) key_part<T, 2, D / 16>(s, sa + f.k0, 8u * f.kwh, f.ksh0, bq, cpy);
    else {
        if (f.kf == F43) key_part<T, 4, D / 32>(s, sa + f.k0, 8u * f.kwh, f.ksh0, bq, cpy);
        else key_part<T, 2, D / 32>(s, sa + f.k1, 8u * f.kwl, f.ksh1, bq + D / 32, cpy);
        if (f.kf == F43) key_part<T, 3, D / 32>(s, sa + f.k1, 8u * f.kwl, f.ksh1, bq + D / 32, cpy);
        else key_part<T, 3, D / 32>(s, sa + f.k0, 8u * f.kwh, f.ksh0, bq, cpy);
    }
    const uint32_t aa = sa + f.tok;
    const float kn0 = ring_f32o<P::O_KN>(aa), kn1 = ring_f32o<P::O_KN + 32>(aa);
    float vn0 = ring_f32o<P::O_VN>(aa), vn1 = ring_f32o<P::O_VN + 32>(aa);
    float gv0 = 0.f, gv1 = 0.f;
    if (QJL) {
        // sketch term: (c/d) gamma_k * sum_p sign_p (S q)[p]; signs of rows 4t + q (+ 16) sit at bits 12 + q, 28 + q after one shift
        const uint32_t zs0 = ring32o<P::O_KB>(aa) << (12 - 4 * t), zs1 = ring32o<P::O_KB + 32>(aa) << (12 - 4 * t);
        float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < QM / 16; ++ks)
            mma16816(sq, sign_pair16(zs0 << (3 - 2 * ks)), sign_pair16(zs1 << (3 - 2 * ks)), sign_pair16(zs0 << (2 - 2 * ks)),
                     sign_pair16(zs1 << (2 - 2 * ks)), bu[ks][0], bu[ks][1]);
        const float gk0 = ring_f32o<P::O_KG>(aa) * (QJL_C / D), gk1 = ring_f32o<P::O_KG + 32>(aa) * (QJL_C / D);
        s[0] = fmaf(s[0], kn0, sq[0] * gk0); s[1] = fmaf(s[1], kn0, sq[1] * gk0);
        s[2] = fmaf(s[2], kn1, sq[2] * gk1); s[3] = fmaf(s[3], kn1, sq[3] * gk1);
        gv0 = ring_f32o<P::O_VG>(aa); gv1 = ring_f32o<P::O_VG + 32>(aa);
    } else {
        s[0] *= kn0; s[1] *= kn0; s[2] *= kn1; s[3] *= kn1;
    }
    if (left < TILE) {
        // the last tile of a lane reaches past the end of the cache: its missing tokens (arbitrary bytes) get no weight
        __syncwarp();
        const bool ok0 = tokA < left, ok1 = tokA + 8 < left;
        vn0 = ok0 ? vn0 : 0.f; vn1 = ok1 ? vn1 : 0.f; gv0 = ok0 ? gv0 : 0.f; gv1 = ok1 ? gv1 : 0.f;
        s[0] = ok0 ? s[0] : -INFINITY; s[1] = ok0 ? s[1] : -INFINITY;
        s[2] = ok1 ? s[2] : -INFINITY; s[3] = ok1 ? s[3] : -INFINITY;
    }
    float pr[4];
    softmax_scores<D, NZ>(s, vn0, vn1, fmaxf(gv0, gv1), st, pr);
    uint32_t bp[2];
    bp[0] = movm_t(pack_h2(pr[0] * vn0, pr[1] * vn0));
    bp[1] = movm_t(pack_h2(pr[2] * vn1, pr[3] * vn1));

    // ---- values: O^T[coordinate][head] += V^T . P^T ----
    if (f.vf == F4) value_part<T, 4, D / 16>(st.o, sa + f.v0, 4u * f.vwh, f.vsh0, bp, cpy);
    else if (f.vf == F3) value_part<T, 3, D / 16>(st.o, sa + f.v0, 4u * f.vwh, f.vsh0, bp, cpy);
    else if (f.vf == F2) value_part<T, 2, D / 16>(st.o, sa + f.v0, 4u * f.vwh, f.vsh0, bp, cpy);
    else if (f.vf == F43) {
        value_part<T, 4, D / 32>(st.o, sa + f.v0, 4u * f.vwh, f.vsh0, bp, cpy);
        value_part<T, 3, D / 32>(st.o + D / 32, sa + f.v1, 4u * f.vwl, f.vsh1, bp, cpy);
    } else {
        value_part<T, 3, D / 32>(st.o, sa + f.v0, 4u * f.vwh, f.vsh0, bp, cpy);
        value_part<T, 2, D / 32>(st.o + D / 32, sa + f.v1, 4u * f.vwl, f.vsh1, bp, cpy);
    }
    if (QJL) {
        // sketch rows of the output: z[row][head] += sum_t sign_row(t) * (p_t * gamma_v[t])
        const uint32_t bz0 = movm_t(pack_h2(pr[0] * gv0, pr[1] * gv0));
        const uint32_t bz1 = movm_t(pack_h2(pr[2] * gv1, pr[3] * gv1));
        const uint32_t pa = sa + 4u * t;           // tokens t, t + 4, t + 8, t + 12: k slots 2t, 2t + 1, 2t + 8, 2t + 9
        const uint32_t zv0 = ring32o<P::O_VB>(pa), zv1 = ring32o<P::O_VB + 16>(pa), zv2 = ring32o<P::O_VB + 32>(pa), zv3 = ring32o<P::O_VB + 48>(pa);
        // put the two tokens' half-words side by side (row r of the first at bit r, of the second at bit r + 16)
        const uint32_t x01 = __byte_perm(zv0, zv1, 0x5410) << (7 - g), y01 = __byte_perm(zv0, zv1, 0x7632) << (7 - g);
        const uint32_t x23 = __byte_perm(zv2, zv3, 0x5410) << (7 - g), y23 = __byte_perm(zv2, zv3, 0x7632) << (7 - g);
        mma16816(st.z[0], sign_pair16(x01 << 8), sign_pair16(x01), sign_pair16(x23 << 8), sign_pair16(x23), bz0, bz1);
        mma16816(st.z[NZ ? 1 : 0], sign_pair16(y01 << 8), sign_pair16(y01), sign_pair16(y23 << 8), sign_pair16(y23), bz0, bz1);
    }
}

// ---- the queries ----------------------------------------------------------------------------------------
// q_rot[h][j] = sum_k q[h][k] R[j][k] (rotation.py:81-110), u[h][p] = sum_k q[h][k] S[p][k] (qjl.py:70-94), both times
// scale * log2(e), fp16.  A warp owns a slab of 16 rows of R (or S) as the A operand and eight query heads as the B operand; both
// are split into fp16 high and 2^-11 low parts (the product of the low parts is below float32 resolution).
__device__ __forceinline__ void split_h2(float2 x, uint32_t& h, uint32_t& l) {
    const __half2 a = __floats2half2_rn(x.x, x.y);
    const float2 af = __half22float2(a);
    h = *reinterpret_cast<const uint32_t*>(&a);
    l = pack_h2((x.x - af.x) * 2048.f, (x.y - af.y) * 2048.f);
}
template <int D> __device__ __forceinline__ void load_rows(const DecodeParams& p, int slab, int g, int t, float2 (&rr)[D / 16][4]) {
    const float* row = slab >= D / 16 ? p.qjl_proj + int64_t(slab - D / 16) * 16 * D : p.rot + int64_t(slab) * 16 * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int r = 0; r < 4; ++r) rr[ks][r] = __ldg(reinterpret_cast<const float2*>(row + (g + (r & 1) * 8) * D + ks * 16 + 2 * t + (r >> 1) * 8));
}
// y: rows g, g + 8 of the slab x heads q0 + 2t, + 1
template <int D>
__device__ __forceinline__ void rotate_rows(const DecodeParams& p, int64_t q0, int64_t heads, int g, int t, const float2 (&rr)[D / 16][4], float (&y)[4]) {
    float2 x[D / 16][2];                                  // head q0 + g: coordinates 16 ks + 2 t, + 1 and the same + 8
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int u = 0; u < 2; ++u) x[ks][u] = g < heads ? q_pair(p, q0 + g, ks * 16 + 2 * t + 8 * u) : make_float2(0.f, 0.f);
    float ym[4] = {0.f, 0.f, 0.f, 0.f}, ya[4] = {0.f, 0.f, 0.f, 0.f}, yb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t bh[2], bl[2], ah[4], al[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) split_h2(x[ks][u], bh[u], bl[u]);
#pragma unroll
        for (int r = 0; r < 4; ++r) split_h2(rr[ks][r], ah[r], al[r]);
        mma16816(ym, ah[0], ah[1], ah[2], ah[3], bh[0], bh[1]);
        mma16816(ya, al[0], al[1], al[2], al[3], bh[0], bh[1]);
        mma16816(yb, ah[0], ah[1], ah[2], ah[3], bl[0], bl[1]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) y[r] = ym[r] + (ya[r] + yb[r]) * (1.f / 2048.f);
}

// Fills the tables of the call's widths; gp(address) is the generic pointer of a shared-window address.
template <typename T, int NT, typename GP> __device__ __forceinline__ void fill_tables(const DecodeParams& p, int tid, const GP& gp) {
    auto cent = [&](const float* c, int i, float sc) -> uint32_t { return uint32_t(__half_as_ushort(__float2half_rn(__ldg(c + i) * sc))); };
    const float* ck[2] = {p.kc_hi, p.kc_lo};
    const float* cv[2] = {p.vc_hi, p.vc_lo};
    const int kb[2] = {p.kb_hi, p.kb_lo}, vb[2] = {p.vb_hi, p.vb_lo};
    for (int side = 0; side < 2; ++side) {
        const float* const* cc = side ? cv : ck;
        const int* bb = side ? vb : kb;
        for (int part = 0; part < 2; ++part) {
            const float* c = cc[part];
            const int b = bb[part];
            const float sc = side == 0 ? 1.f : part ? p.v_scale_lo : p.v_scale_hi;
            if (b == 3) {
                for (int i = tid; i < 64 * 8; i += NT) {               // 64 entries of eight 16-byte pieces
                    const int e = i >> 3;
                    const uint32_t x = cent(c, e & 7, sc) | (cent(c, e >> 3, sc) << 16);
                    *reinterpret_cast<uint4*>(gp((side ? T::V3 : T::K3) + uint32_t(i) * 16u)) = make_uint4(x, x, x, x);
                }
            } else if (b == 4) {
                for (int i = tid; i < 256 * 8; i += NT) {
                    const int e = i >> 3;
                    const uint32_t x = cent(c, e & 15, sc) | (cent(c, e >> 4, sc) << 16);
                    *reinterpret_cast<uint4*>(gp(T::B + uint32_t(e) * 256u + (side ? 128u : 0u) + uint32_t(i & 7) * 16u)) = make_uint4(x, x, x, x);
                }
            } else if (b == 2) {
                for (int i = tid; i < 256 * 8; i += NT) {
                    const int e = i >> 3;
                    // keys: four coordinates in a row; values: low nibble = two coordinates of the first token, high nibble of the second
                    const int i0 = e & 3, i1 = (e >> 2) & 3, i2 = (e >> 4) & 3, i3 = e >> 6;
                    const uint32_t x = cent(c, i0, sc) | (cent(c, side ? i2 : i1, sc) << 16), y = cent(c, side ? i1 : i2, sc) | (cent(c, i3, sc) << 16);
                    *reinterpret_cast<uint4*>(gp(T::B + uint32_t(e) * 256u + (side ? 128u : 0u) + uint32_t(i & 7) * 16u)) = make_uint4(x, y, x, y);
                }
            }
        }
    }
}

}  // namespace lut
}  // namespace tq
