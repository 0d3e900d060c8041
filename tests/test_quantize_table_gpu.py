"""The 4-bit boundary search by table, for codebooks whose boundaries leave the table's range or crowd into one bin.

A rotated value is within 2e-6 of float64 (the bound of the rotation tests, rows of norm one), so a code has to be the count of smaller
boundaries wherever no boundary is nearer than that."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,qjl", ((64, False), (96, True), (128, False), (128, True), (256, False)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("kind", ("wide", "outside", "one_bin", "edges"))
def test_codebooks(d, qjl, dtype, kind):
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib
    dev = torch.device("cuda", torch.cuda.current_device())
    bnd = {"wide": torch.linspace(-0.95, 0.95, 15), "outside": torch.cat([torch.linspace(-0.99, -0.52, 8), torch.linspace(0.51, 0.98, 7)]),
           "one_bin": 0.0501 + torch.arange(15) * 1e-4, "edges": torch.tensor([-0.51, -0.505, -0.5, -0.499, -0.495, -0.3, -0.1, 0, 0.1, 0.3, 0.495, 0.499, 0.5, 0.505, 0.51])}[kind]
    bnd = bnd.float().to(dev)
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=2, key_bits=4, value_bits=4, fp16_sink_size=0, residual_window=16, qjl_correction=qjl)
    c._bind(dev)
    r = c._rotation
    g = torch.Generator(device="cuda").manual_seed(d)
    a, b = (torch.randn(2000, 1, device=dev, generator=g) for _ in range(2))
    x = torch.cat([r, -r, a * r[:1] + b * r[1:2], torch.randn(500, d, device=dev, generator=g)])      # |y| = 1; two coordinates of any size; dense rows
    x = x.to(dtype)[None, None].repeat(1, 2, 1, 1)
    n, s, job = x.shape[2], c._k, _lib.QuantizeArgs()
    s.reserve(1, 2, d, n, 0, dev, qjl)
    s.quantize_job(job, x, 0)
    job.bnd_hi = bnd.data_ptr()
    _lib.check(_lib.launch(dev, "tq_quantize_pack", job, _lib.stream_ptr(dev)))
    y = x.double() @ r.double().T
    y = y / y.norm(dim=-1, keepdim=True)
    packed = s.hi[:, :, :n].long()
    got = torch.stack([packed & 15, packed >> 4], -1).flatten(-2)
    far = (y[..., None] - bnd.double()).abs().amin(-1) > 2e-6
    assert torch.equal(got[far], (y[..., None] > bnd.double()).sum(-1)[far])
    # (the other coordinates of a two-coordinate row are rounding noise around zero, a boundary of two of the codebooks: not compared)
    assert float(far.float().mean()) > 0.5 and int(got.max()) == 15 and int(got.min()) == 0
