// Host side of the tensor-core dequantize kernels (dequantize_tc.cuh): argument checks, choice of the kernel, launch.
#include <algorithm>
#include <atomic>

#include "dequantize_tc.cuh"

namespace tq {
namespace dqtc {
template <> Kernel kernel_of<64>(int, int, bool);
template <> Kernel kernel_of<96>(int, int, bool);
template <> Kernel kernel_of<128>(int, int, bool);
template <> Kernel kernel_of<256>(int, int, bool);
}  // namespace dqtc

// One or two jobs that share head_dim, rotation and result type (keys and values of a cache), on the tensor cores when
// every job's layout allows; *handled = false leaves the call to the row kernel.  The second job's launch does not wait for the first: its
// CTAs take the SMs that the first one's last tiles leave idle.
int tq_dequantize_tc(const tq_dequantize_args* q, int n_jobs, cudaStream_t s, bool* handled) {
    *handled = false;
    const int d = q[0].d;
    if ((d != 64 && d != 96 && d != 128 && d != 256) || n_jobs < 1 || n_jobs > 2) return TQ_OK;
    dqtc::Params p[2] = {};
    dqtc::Kernel k[2];
    int* status = decode_status_ptr();
    if (!status) return fail(TQ_ERR_LAUNCH, "tq_dequantize: cannot locate the status word");
    for (int i = 0; i < n_jobs; ++i) {
        const tq_dequantize_args& a = q[i];
        dqtc::Params& j = p[i];
        if (a.d != d || !aligned(a.rot, 16)) return TQ_OK;
        if (a.bits_lo && a.bits_lo != a.bits_hi - 1) return TQ_OK;              // the reference's fractional widths are (b, b - 1)
        const int half = a.bits_lo ? d / 2 : d;
        const int es = a.out_dtype == TQ_F32 ? 4 : 2;
        if (!aligned(a.out, 2 * es) || a.out_lane_stride % 8 || a.out_row_stride % 8 || a.out_row_stride < d) return TQ_OK;
        if (((a.n_lanes - 1) * a.out_lane_stride + a.n_rows * a.out_row_stride) / 8 >= 0xffffffffll) return TQ_OK;   // offsets are kept as 32-bit multiples of eight
        // packed rows are read as 4-byte words (4 bits), 2-byte words (2 bits) or bytes
        const int w_hi = half * a.bits_hi / 8, w_lo = a.bits_lo ? (d - half) * a.bits_lo / 8 : 0;
        auto words_ok = [](const void* ptr, int bits, int w) {
            const size_t n = bits == 4 ? 4 : bits == 2 ? 2 : 1;
            return aligned(ptr, n) && w % int(n) == 0;
        };
        if (!words_ok(a.packed_hi, a.bits_hi, w_hi) || (a.bits_lo && !words_ok(a.packed_lo, a.bits_lo, w_lo))) return TQ_OK;
        const int64_t total = a.n_lanes * a.n_rows;
        if (total >= (int64_t(1) << 31) || a.n_lanes * a.in_lane_stride >= (int64_t(1) << 31)) return TQ_OK;
        j.packed_hi = a.packed_hi; j.packed_lo = a.packed_lo; j.norms = a.norms;
        j.n_rows = uint32_t(a.n_rows); j.total = uint32_t(total); j.in_lane_stride = a.in_lane_stride;
        j.half = half; j.bits_hi = a.bits_hi; j.bits_lo = a.bits_lo; j.w_hi = w_hi; j.w_lo = w_lo;
        j.cent_hi = a.cent_hi; j.cent_lo = a.cent_lo; j.rot = a.rot;
        j.qjl_proj = a.qjl_proj; j.qjl_bits = a.qjl_bits; j.qjl_gamma = a.qjl_gamma;
        j.out = a.out; j.out_dtype = a.out_dtype; j.out_lane_stride = a.out_lane_stride; j.out_row_stride = a.out_row_stride;
        j.n_tiles = int((total + dqtc::TM - 1) / dqtc::TM);
        j.follows = i; j.status = status;
        k[i] = d == 64 ? dqtc::kernel_of<64>(a.bits_hi, a.bits_lo, a.qjl_bits != nullptr) : d == 96 ? dqtc::kernel_of<96>(a.bits_hi, a.bits_lo, a.qjl_bits != nullptr)
             : d == 128 ? dqtc::kernel_of<128>(a.bits_hi, a.bits_lo, a.qjl_bits != nullptr) : dqtc::kernel_of<256>(a.bits_hi, a.bits_lo, a.qjl_bits != nullptr);
        if (!k[i]) return TQ_OK;
    }
    const size_t smem = d == 64 ? dqtc::Plan<64>::SMEM : d == 96 ? dqtc::Plan<96>::SMEM : d == 128 ? dqtc::Plan<128>::SMEM : dqtc::Plan<256>::SMEM;
    static std::atomic<uint64_t> set[64][4];             // bit = width pair whose shared-memory limit is raised
    static std::atomic<int> sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TQ_OK;
    int n_sms = sms[dev].load();
    if (!n_sms) {
        if (cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n_sms <= 0) n_sms = 148;
        sms[dev].store(n_sms);
    }
    static PFN_cuTensorMapEncodeTiled encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) fn = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }();
    if (!encode) return TQ_OK;
    CUtensorMap maps[2] = {};
    for (int i = 0; i < n_jobs; ++i) {
        // the result as (column, row, cache lane), boxes of 64 bytes x 32 rows
        const tq_dequantize_args& a = q[i];
        const int es = a.out_dtype == TQ_F32 ? 4 : 2;
        const cuuint64_t dims[3] = {cuuint64_t(d), cuuint64_t(a.n_rows), cuuint64_t(a.n_lanes)};
        const cuuint64_t strides[2] = {cuuint64_t(a.out_row_stride) * es, cuuint64_t(a.n_lanes > 1 ? a.out_lane_stride : a.out_row_stride * a.n_rows) * es};
        const cuuint32_t box[3] = {cuuint32_t(64 / es), 32, 1}, est[3] = {1, 1, 1};
        if (strides[1] == 0 || strides[1] >= (cuuint64_t(1) << 40) || !aligned(a.out, 16)) return TQ_OK;
        if (encode(&maps[i], es == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, a.out, dims, strides, box, est,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return TQ_OK;
    }
    *handled = true;
    // Two jobs of few tiles run side by side on half the SMs each: a CTA's set-up (R as operand tiles, 8 us) is then paid once
    // (65,536 rows a side at d = 128: 39 us one after the other, 27 side by side); long ones balance better one after the other.
    const bool share = n_jobs == 2 && std::max(p[0].n_tiles, p[1].n_tiles) <= 16 * n_sms;
    for (int i = 0; i < n_jobs; ++i) {
        std::atomic<uint64_t>& bits = set[dev][d == 64 ? 0 : d == 96 ? 1 : d == 128 ? 2 : 3];
        const uint64_t bit = uint64_t(1) << (p[i].bits_hi * 8 + p[i].bits_lo - 8 + (p[i].qjl_bits ? 32 : 0));
        if (!(bits.load(std::memory_order_acquire) & bit)) {
            cudaError_t e = cudaFuncSetAttribute(k[i], cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_dequantize: shared memory %zu B: %s", smem, cudaGetErrorString(e));
            bits.fetch_or(bit, std::memory_order_release);
        }
        cudaLaunchConfig_t cfg{};
        const int ctas = share ? n_sms / 2 : n_sms;
        cfg.gridDim = dim3(unsigned(d == 256 ? 2 * std::min(p[i].n_tiles, ctas / 2) : std::min(p[i].n_tiles, ctas)));
        cfg.blockDim = dim3(dqtc::NT);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k[i], p[i], maps[i]);
        if (e != cudaSuccess) return fail(TQ_ERR_LAUNCH, "tq_dequantize: %s", cudaGetErrorString(e));
    }
    return TQ_OK;
}

}  // namespace tq
