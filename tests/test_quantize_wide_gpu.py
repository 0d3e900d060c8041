"""The tensor-core quantize kernel at head_dim 256, where four CTAs share a tile: every width and split, both 16-bit types, ragged
lanes, rows at an offset of larger storage, zero rows.  Reference: the float32 row kernel on the same values; a code may differ
only where the rotated value lies within float32 rounding of a boundary."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("bits", (1, 2, 3, 4, 1.5, 2.5, 3.5))
@pytest.mark.parametrize("lanes,rows", ((1, 512), (3, 301), (5, 128), (2, 6000)))
def test_slices_equal_the_row_kernel(dtype, bits, lanes, rows):
    from mlx_turboquant_b200 import _lib, kernels
    from mlx_turboquant_b200.codebook import get_codebook
    from mlx_turboquant_b200.rotation import get_rotation_matrix
    d = 256
    hi, lo = kernels.split_bits(bits)
    g = torch.Generator(device="cuda").manual_seed(rows + hi)
    x = (torch.randn(lanes, rows + 5, d, device="cuda", generator=g) * torch.exp(2 * torch.randn(lanes, rows + 5, 1, device="cuda", generator=g))).to(dtype)[:, 3:3 + rows]
    x[:, 7] = 0
    w_hi, w_lo = kernels.packed_widths(d, hi, lo)
    b_hi, b_lo = get_codebook(d, hi)[1], get_codebook(d, lo)[1] if lo else None
    res = []
    for v in (x, x.float()):
        out = [torch.full((lanes, rows + 32, w), 0xA5, dtype=torch.uint8, device="cuda") for w in (w_hi, max(w_lo, 1))]
        norms = torch.full((lanes, rows + 32), -1.0, device="cuda")
        kernels.quantize_pack(v, get_rotation_matrix(d), b_hi, hi, b_lo, lo, out_hi=out[0], out_lo=out[1] if lo else None, out_norms=norms, out_offset=16)
        res.append((*out, norms))
    for a, b in zip(res[0][:2], res[1][:2]):
        assert (a != b).float().mean() < 2e-4
        assert (a[:, :16] == 0xA5).all() and (a[:, 16 + rows:] == 0xA5).all()
    torch.testing.assert_close(res[0][2], res[1][2], rtol=1e-6, atol=0)
    assert _lib.lib().tq_device_status() == 0
