"""Sign sketches of the tensor-core quantize kernel against float64, from the codes it wrote itself.

The kernel's rotated rows are within 2e-6 of |x| (the bound of the rotation tests) and its projections carry a relative 2^-20 of the residual
(fp16 high and low parts on both sides, the product of the low parts left out): a sign may differ only where the float64 projection is
below |s| (2e-6 + 2^-20 |e|) in size, |s| the projection row's norm; the residual's norm differs by 2e-6 |x| at most, and d / 2 roundings."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bits", ((64, 3), (96, 4), (128, 2), (128, 3.5), (96, 1.5), (128, 1)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("h,n", ((1, 1), (3, 129), (2, 1000), (1, 148 * 128 * 3 + 1), (150, 500)))
def test_sketch(d, bits, dtype, h, n):
    """A row; a ragged tile; CTAs of four tiles (every stage used again) beside CTAs of three; as many ragged lanes as CTAs and more."""
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib, kernels
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device="cuda").manual_seed(n + d)
    x = (torch.randn(1, h, n, d, device=dev, generator=g) * torch.exp(torch.randn(1, h, n, 1, device=dev, generator=g))).to(dtype)
    x[0, 0, n // 2] = 0
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=h, key_bits=bits, value_bits=bits, fp16_sink_size=0, residual_window=16, qjl_correction=True)
    c._bind(dev)
    s = c._k
    s.reserve(1, h, d, n, 0, dev, True)
    job = _lib.QuantizeArgs()
    s.quantize_job(job, x, 0)
    _lib.check(_lib.launch(dev, "tq_quantize_pack", job, _lib.stream_ptr(dev)))
    assert _lib.lib().tq_device_status() == 0
    bh, bl = kernels.split_bits(bits)
    half = d // 2 if bl else d
    shift = torch.arange(8, device=dev)

    def centroids(packed, cent, b, w):
        flat = ((packed[:, :, :n].long()[..., None] >> shift) & 1).flatten(-2)[..., :w * b].unflatten(-1, (w, b))
        return cent.double()[(flat << torch.arange(b, device=dev)).sum(-1)]

    q = centroids(s.hi, s.cent_hi, bh, half)
    if bl:
        q = torch.cat([q, centroids(s.lo, s.cent_lo, bl, d - half)], -1)
    norm = x.double().norm(dim=-1, keepdim=True)
    e = (x.double() @ c._rotation.double().T) / norm.clamp_min(1e-10) - q
    size = e.norm(dim=-1, keepdim=True)
    p = c._qjl_proj_rot.double()
    proj = e @ p.T
    got = (s.qbits[:, :, :n].long()[..., None] >> torch.arange(32, device=dev)) & 1
    zero = norm[..., 0] == 0
    assert bool((got[zero] == 1).all())
    clear = proj.abs() > p.norm(dim=-1) * (2e-6 + 2.0 ** -20 * size)
    assert torch.equal((got == 1)[clear & ~zero[..., None]], (proj >= 0)[clear & ~zero[..., None]])
    want = norm * size
    assert bool(((s.qgamma[:, :, :n, None] - want).abs() <= norm * 2e-6 + want * (d / 2 + 8) * 2.0 ** -24).all())
