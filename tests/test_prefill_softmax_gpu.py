"""The running reference of the several-token kernel's softmax, which is looked at through the sums of weights: scores that climb, fall, stay,
sit far below zero, or add up past the limit without one weight that exceeds it, in every head_dim and with rows that see part of a tile."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _scores(kind, n):
    t = torch.arange(n, dtype=torch.float64)
    if kind == "climb":
        return -300.0 + 600.0 * t / n
    if kind == "fall":
        return 300.0 - 600.0 * t / n
    if kind == "low":                                    # below the smallest exponential: the first token of a row decides
        return -250.0 - 3.0 * torch.sin(t)
    if kind == "steps":                                  # 3 bits above the reference at a time: sums pass 2^6, no weight does
        return torch.floor(t / 64) * 2.0
    return torch.sin(t) * 4.0


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("kind", ("climb", "fall", "low", "steps", "flat"))
def test_references(d, kind):
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib
    n, tq, hkv, g = 700, 150, 2, 4
    gen = torch.Generator().manual_seed(d)
    u = torch.nn.functional.normalize(torch.randn(d, dtype=torch.float64, generator=gen), dim=0)
    k = (_scores(kind, n)[:, None] * u).expand(1, hkv, n, d).half()
    v = torch.randn(1, hkv, n, d, dtype=torch.float64, generator=gen).half()
    q = (u * (1 + 0.1 * torch.arange(g * hkv, dtype=torch.float64)[:, None])).view(1, g * hkv, 1, d).expand(1, g * hkv, tq, d).half().contiguous()
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=hkv, residual_window=1024, fp16_sink_size=64)
    c.update(k.cuda(), v.cuda())
    out = c.attend(q.cuda(), scale=1.0, out_dtype=torch.float32).cpu().double()
    s = torch.einsum("bhrtd,bhnd->bhrtn", q.double().view(1, hkv, g, tq, d), k.double())
    s = s.masked_fill(torch.arange(n) > (n - tq + torch.arange(tq))[:, None], float("-inf"))
    ref = torch.einsum("bhrtn,bhnd->bhrtd", torch.softmax(s, -1), v.double()).reshape(1, g * hkv, tq, d)
    # The scaled query is rounded to fp16 (2^-11), which scales a row's scores by 1 + 2^-11 at most, the keys being multiples of one vector:
    # weights of scores within 20 of the row's largest are off by 20 x 2^-11, the others do not count.
    tol = 1e-2
    assert torch.isfinite(out).all() and (out - ref).abs().max() < tol * ref.abs().max()
    assert _lib.lib().tq_device_status() == 0
