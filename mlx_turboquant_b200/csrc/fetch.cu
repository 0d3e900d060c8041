// Dense keys and values for a caller with its own attention (update_and_fetch, cache.py:620-706): the uncompressed regions
// [sink | ... | recent] and, where it is kept expanded, the middle, copied into the results with their conversion in one
// launch; the packed middle dequantized straight to its place between them (tq_dequantize_pair).
//
// The copy is bound by memory: a thread moves eight elements at a time (16 or 32 bytes each way), four in flight.  (torch.cat
// over mixed types: a conversion pass per part, then 1.7 TB/s: 78 us for 8 lanes x 8192 tokens at head_dim 128; direct: 21 us.)
#include <algorithm>

#include "common.cuh"

namespace tq {

struct CopyPart { const void* k; const void* v; int dtype; uint32_t rows; int64_t lane_stride; uint32_t dst_row; };   // rows per lane, lane stride in rows
struct CopyParams {
    CopyPart part[3];
    uint32_t n_rows, chunks;              // rows copied per lane, eight-element chunks per row
    uint32_t blocks_per_lane;
    int d, out_dtype;
    int64_t lanes, out_rows;              // rows per lane of the results
    void *k_out, *v_out;
};

struct Eight { uint4 a, b; };             // eight elements: 16-bit in a, float32 in a and b

__device__ __forceinline__ Eight load8(const void* p, int dtype, int64_t e) {
    Eight x;
    if (dtype == TQ_F32) {
        const uint4* s = reinterpret_cast<const uint4*>(static_cast<const float*>(p) + e);
        x.a = __ldg(s); x.b = __ldg(s + 1);
    } else {
        x.a = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p) + e));
        x.b = make_uint4(0u, 0u, 0u, 0u);
    }
    return x;
}

__device__ __forceinline__ void store8(void* p, int out_dtype, int64_t e, const Eight& x, int dtype) {
    if (out_dtype != TQ_F32) {            // (16-bit results: the parts have the same type)
        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p) + e) = x.a;
        return;
    }
    uint4* dst = reinterpret_cast<uint4*>(static_cast<float*>(p) + e);
    if (dtype == TQ_F32) { dst[0] = x.a; dst[1] = x.b; return; }
    const uint32_t w[4] = {x.a.x, x.a.y, x.a.z, x.a.w};
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (dtype == TQ_BF16) { o[2 * i] = w[i] << 16; o[2 * i + 1] = w[i] & 0xffff0000u; }
        else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            o[2 * i] = __float_as_uint(f.x); o[2 * i + 1] = __float_as_uint(f.y);
        }
    }
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

constexpr int COPY_T = 256, COPY_U = 4;

__global__ void __launch_bounds__(COPY_T) copy_parts_kernel(const __grid_constant__ CopyParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");       // (the dequantize that follows sets itself up meanwhile)
    const uint32_t lane2 = blockIdx.x / p.blocks_per_lane, blk = blockIdx.x - lane2 * p.blocks_per_lane;
    const bool is_v = lane2 >= uint32_t(p.lanes);
    const int64_t lane = is_v ? lane2 - uint32_t(p.lanes) : lane2;
    const uint32_t n = p.n_rows * p.chunks;
    void* out = is_v ? p.v_out : p.k_out;
    Eight x[COPY_U];
    int64_t dst[COPY_U];
    int dt[COPY_U];
#pragma unroll
    for (int u = 0; u < COPY_U; ++u) {
        const uint32_t i = (blk * COPY_U + u) * COPY_T + threadIdx.x;
        dst[u] = -1;
        if (i >= n) continue;
        uint32_t row = i / p.chunks;
        const uint32_t c = (i - row * p.chunks) * 8u;
        int s = 0;
        if (row >= p.part[0].rows) { row -= p.part[0].rows; s = 1; if (row >= p.part[1].rows) { row -= p.part[1].rows; s = 2; } }
        const CopyPart& q = p.part[s];
        dt[u] = q.dtype;
        dst[u] = (lane * p.out_rows + q.dst_row + row) * p.d + c;
        x[u] = load8(is_v ? q.v : q.k, q.dtype, (lane * q.lane_stride + row) * p.d + c);
    }
#pragma unroll
    for (int u = 0; u < COPY_U; ++u)
        if (dst[u] >= 0) store8(out, p.out_dtype, dst[u], x[u], dt[u]);
}

}  // namespace tq

extern "C" int tq_fetch_dense(const tq_fetch_args* a, const tq_dequantize_args* k, const tq_dequantize_args* v, void* stream) {
    using namespace tq;
    if (!a) return fail(TQ_ERR_INVALID, "tq_fetch_dense: null args");
    if (a->d <= 0 || a->d % 8 || a->lanes < 0 || a->out_rows < 0 || !dtype_ok(a->out_dtype)) return fail(TQ_ERR_INVALID, "tq_fetch_dense: bad sizes");
    CopyParams p{};
    p.d = a->d; p.out_dtype = a->out_dtype; p.lanes = a->lanes; p.out_rows = a->out_rows; p.k_out = a->k_out; p.v_out = a->v_out;
    p.chunks = uint32_t(a->d / 8);
    int64_t rows = 0;
    int n = 0;
    for (int i = 0; i < 3; ++i) {
        const tq_fetch_part& s = a->part[i];
        if (s.rows == 0) continue;
        if (s.rows < 0 || s.dst_row < 0 || s.dst_row + s.rows > a->out_rows || s.lane_stride < s.rows || !dtype_ok(s.dtype) || !s.k || !s.v)
            return fail(TQ_ERR_INVALID, "tq_fetch_dense: bad part");
        if ((a->out_dtype != TQ_F32 && s.dtype != a->out_dtype) || !aligned(s.k, 16) || !aligned(s.v, 16))
            return fail(TQ_ERR_UNSUPPORTED, "tq_fetch_dense: parts must be 16-byte aligned, of the results' type or for float32 results");
        p.part[n++] = CopyPart{s.k, s.v, s.dtype, uint32_t(s.rows), s.lane_stride, uint32_t(s.dst_row)};
        rows += s.rows;
    }
    if (a->lanes > 0 && a->out_rows > 0 && (!a->k_out || !a->v_out || !aligned(a->k_out, 16) || !aligned(a->v_out, 16)))
        return fail(TQ_ERR_UNSUPPORTED, "tq_fetch_dense: results must be 16-byte aligned");
    if (a->out_rows * p.chunks >= (int64_t(1) << 31)) return fail(TQ_ERR_UNSUPPORTED, "tq_fetch_dense: too many rows per lane");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (rows > 0 && a->lanes > 0) {
        p.n_rows = uint32_t(rows);
        p.blocks_per_lane = uint32_t((rows * p.chunks + COPY_T * COPY_U - 1) / (COPY_T * COPY_U));
        const int64_t blocks = int64_t(p.blocks_per_lane) * 2 * a->lanes;
        if (blocks >= (int64_t(1) << 31)) return fail(TQ_ERR_UNSUPPORTED, "tq_fetch_dense: too many rows");
        copy_parts_kernel<<<unsigned(blocks), COPY_T, 0, s>>>(p);
        if (int rc = check_launch("tq_fetch_dense")) return rc;
    }
    if (k && v) return tq_dequantize_pair(k, v, stream);
    return TQ_OK;
}
