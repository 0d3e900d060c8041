"""The tensor-core dequantize kernel where its tiles, lanes and widths can go wrong: a single row, rows that straddle cache
lanes and 128-row tiles, head_dim 256 (two CTAs share a tile's columns), fractional splits, the sketch correction, 16-bit
results at an offset of a larger buffer.  Reference: the float32 formula on the same codes."""

import numpy as np
import pytest
import torch

from gpu_util import cu, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("hi,lo", ((1, 0), (2, 0), (3, 0), (4, 0), (3, 2), (4, 3)))
@pytest.mark.parametrize("qjl", (False, True))
@pytest.mark.parametrize("lanes,rows,dtype", ((1, 1, torch.float32), (5, 37, torch.bfloat16), (3, 333, torch.float32), (2, 16500, torch.float16)))
def test_tiles_lanes_widths(oracle, tables, d, hi, lo, qjl, lanes, rows, dtype):
    from mlx_turboquant_b200 import _lib, kernels
    from mlx_turboquant_b200.codebook import get_codebook
    from mlx_turboquant_b200.qjl import get_projection_matrix
    from mlx_turboquant_b200.rotation import get_rotation_matrix
    from oracle import tq_oracle as orc
    rs = np.random.RandomState(d + 10 * hi + lo + rows)
    half = d // 2 if lo else d
    ih, il = rs.randint(0, 1 << hi, size=(lanes, rows + 3, half)).astype(np.uint8), rs.randint(0, 1 << max(lo, 1), size=(lanes, rows + 3, d - half)).astype(np.uint8)
    norms = np.exp(rs.randn(lanes, rows + 3)).astype(np.float32)
    bits = rs.randint(0, 1 << 32, size=(lanes, rows + 3), dtype=np.uint64).astype(np.uint32)
    gamma = rs.rand(lanes, rows + 3).astype(np.float32)
    sketch = dict(proj=get_projection_matrix(d, 32), bits=cu(bits.view(np.int32)), gamma=cu(gamma)) if qjl else None
    ch, cl = get_codebook(d, hi)[0], get_codebook(d, lo)[0] if lo else None
    out = torch.full((lanes, rows + 9, d), 7.0, dtype=dtype, device="cuda")
    kernels.dequantize_rows(cu(orc.pack(ih, hi)), cu(orc.pack(il, lo)) if lo else None, cu(norms), get_rotation_matrix(d), ch, hi, cl, lo, d,
                            n_rows=rows, in_offset=2, out=out, out_offset=4, qjl=sketch)
    y = np.concatenate([host(ch)[ih], host(cl)[il]], -1) if lo else host(ch)[ih]
    ref = (y[:, 2:2 + rows].astype(np.float64) @ host(get_rotation_matrix(d)).astype(np.float64)) * norms[:, 2:2 + rows, None]
    if qjl:
        signs = ((bits[:, 2:2 + rows, None] >> np.arange(32, dtype=np.uint32)) & 1) * 2.0 - 1.0
        ref = ref + np.sqrt(np.pi / 2) / d * gamma[:, 2:2 + rows, None] * (signs @ host(sketch["proj"]).astype(np.float64))
    got = host(out.float())
    tol = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    assert np.all(got[:, :4] == 7.0) and np.all(got[:, 4 + rows:] == 7.0)
    np.testing.assert_allclose(got[:, 4:4 + rows], ref, rtol=tol, atol=(2e-6 + tol) * np.abs(ref).max())
    assert _lib.lib().tq_device_status() == 0
