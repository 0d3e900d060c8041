"""Dense results written in one call: every combination of regions, ragged lengths, storage types, the widths and head dims
whose middle is dequantized in place and those whose middle is kept expanded.  Reference: the regions put together one by one."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,kb,vb,qjl", ((64, 4, 2, False), (96, 3, 4, False), (128, 3.5, 2.5, False), (128, 4, 2, True), (256, 4, 3, False), (48, 4, 2, False)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16, torch.float32))
@pytest.mark.parametrize("sink,rw,steps", ((0, 16, (101, 1)), (7, 16, (5,)), (7, 16, (12, 3)), (5, 0, (77, 9)), (128, 32, (700, 1, 1, 90)), (0, 0, (1, 333))))
def test_regions_side_by_side(d, kb, vb, qjl, dtype, sink, rw, steps):
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib, kernels
    g = torch.Generator(device="cuda").manual_seed(d + sink)
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=3, key_bits=kb, value_bits=vb, residual_window=rw, fp16_sink_size=sink, qjl_correction=qjl)
    for t in steps:
        got = c.update_and_fetch(*(torch.randn(2, 3, t, d, device="cuda", generator=g).to(dtype) for _ in range(2)))
        for out, side, s_buf, r_buf in ((got[0], c._k, c.sink_keys, c.keys), (got[1], c._v, c.sink_values, c.values)):
            parts = []
            if c._sink_len:
                parts.append(s_buf[:, :, :c._sink_len])
            if c._compressed_len:
                parts.append(kernels.dequantize_rows(side.hi, side.lo, side.norms, c.rotation, side.cent_hi, side.bits_hi, side.cent_lo, side.bits_lo, d,
                                                     n_rows=c._compressed_len, qjl=dict(proj=c._qjl_proj, bits=side.qbits, gamma=side.qgamma) if qjl else None))
            if c._fp16_len:
                parts.append(r_buf[:, :, :c._fp16_len])
            want = torch.cat(parts, dim=2)
            assert out.dtype == want.dtype and out.shape == want.shape and out.shape[2] == c.offset
            assert torch.equal(out, want)
    assert _lib.lib().tq_device_status() == 0
