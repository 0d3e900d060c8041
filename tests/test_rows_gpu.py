"""Token buffers filled in one launch, and the native host path against the same steps in torch: layouts it takes and layouts it hands back."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(g, *shape, dtype=torch.float16):
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


@pytest.mark.parametrize("b,h,d,n,cap,kept", ((1, 1, 64, 1, 1, 0), (1, 3, 96, 5, 300, 0), (2, 4, 128, 255, 512, 130), (3, 2, 256, 0, 65, 64), (1, 8, 128, 1000, 1300, 7), (2, 1, 64, 3, 3, 0)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16, torch.float32))
@pytest.mark.parametrize("layout", ("plain", "projection"))
def test_buffers(b, h, d, n, cap, kept, dtype, layout):
    """Kept rows, new rows, zeros; new rows that begin inside a longer tensor; and (B, T, H, D) memory, whose rows are not side by side: handed back."""
    from mlx_turboquant_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(n + cap)
    x = [_rows(g, b, h, n + 9, d, dtype=dtype) if layout == "plain" else _rows(g, b, n + 9, h, d, dtype=dtype).transpose(1, 2) for _ in range(2)]
    old = [_rows(g, b, h, kept + 20, d, dtype=dtype) for _ in range(2)]
    got = _lib.host().buffers(x[0], x[1], 4, n, cap, old[0], old[1], 11, kept)
    if layout == "projection" and h > 1:
        assert got is None
        return
    for y, src, o in zip(got, x, old):
        want = torch.zeros(b, h, cap, d, device="cuda", dtype=dtype)
        want[:, :, :kept], want[:, :, kept:kept + n] = o[:, :, 11:11 + kept], src[:, :, 4:4 + n]
        assert torch.equal(y, want)
    if n > 0 and kept + n <= cap:
        bufs = [t.clone() for t in got]
        assert _lib.host().append(bufs[0], bufs[1], x[0], x[1], 2, n, cap - n) == 0
        for y, src, w in zip(bufs, x, got):
            w[:, :, cap - n:] = src[:, :, 2:2 + n]
            assert torch.equal(y, w)


def test_what_is_handed_back():
    from mlx_turboquant_b200 import _lib
    host = _lib.host()
    x = torch.zeros(2, 2, 8, 64, device="cuda", dtype=torch.float16)
    cpu, other, wide = x.cpu(), x.bfloat16(), torch.zeros(2, 2, 8, 60, device="cuda", dtype=torch.float16)
    windows = x.flatten().as_strided((2, 2, 8, 64), (128, 64, 64, 1))
    for k, v in ((cpu, cpu), (x, other), (wide, wide), (windows, windows), (x.expand(2, 2, 8, 64)[:, :1].expand(2, 2, 8, 64),) * 2):
        assert host.buffers(k, v, 0, 8, 8, None, None, 0, 0) is None
    assert host.append(x, x, x, x, 0, 8, 1) is None                 # no room
    assert host.codec_quantize(b"", 4, x, x) is None


@pytest.mark.parametrize("kb,vb,qjl,d", ((4, 2, False, 128), (3.5, 3.5, False, 128), (4, 2, True, 96), (4, 2, False, 256)))
def test_prompt_in_any_layout(kb, vb, qjl, d):
    """A prompt whose rows the native path takes, and the same values in a layout that it hands back, leave the same cache and dense result."""
    from mlx_turboquant_b200 import TurboQuantKVCache
    g = torch.Generator(device="cuda").manual_seed(5)
    k, v = (_rows(g, 2, 4, 700, d, dtype=torch.bfloat16) for _ in range(2))
    mk = lambda: TurboQuantKVCache(head_dim=d, num_kv_heads=4, key_bits=kb, value_bits=vb, fp16_sink_size=100, residual_window=64, qjl_correction=qjl)  # noqa: E731
    a, b = mk(), mk()
    odd = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)  # noqa: E731
    for n0, n1 in ((0, 40), (40, 500), (500, 501), (501, 700)):
        ra = a.update_and_fetch(k[:, :, n0:n1].contiguous(), v[:, :, n0:n1].contiguous())
        rb = b.update_and_fetch(odd(k[:, :, n0:n1]), odd(v[:, :, n0:n1]))
        assert torch.equal(ra[0], rb[0]) and torch.equal(ra[1], rb[1])
    assert a.meta_state == b.meta_state and a.empty() is False
    for x, y in zip(a.state, b.state):
        assert (x is None) == (y is None) and (x is None or torch.equal(x, y))


@pytest.mark.parametrize("qjl", (False, True))
@pytest.mark.parametrize("kb,vb", ((4, 2), (3.5, 3)))
def test_the_python_steps_do_the_same(monkeypatch, kb, vb, qjl):
    """Without the native module: the same bytes in every array, the same dense results, the same codec."""
    from mlx_turboquant_b200 import TurboQuantKVCache, TurboQuantMSE, _lib

    def run():
        g = torch.Generator(device="cuda").manual_seed(5)
        c = TurboQuantKVCache(head_dim=96, num_kv_heads=3, key_bits=kb, value_bits=vb, residual_window=32, fp16_sink_size=8, qjl_correction=qjl)
        out = [c.update_and_fetch(_rows(g, 2, 3, n, 96), _rows(g, 2, 3, n, 96)) for n in (300, 1, 5, 90)]
        m = TurboQuantMSE(96, 4)
        z = m.quantize(_rows(g, 50, 96))
        n = c._compressed_len
        sides = [x[:, :, :n].clone() for s in (c._k, c._v) for x in (s.hi, s.lo, s.norms, s.qbits, s.qgamma) if x is not None]
        return [x for kv in out for x in kv] + sides + [z.packed_indices, z.norms, m.dequantize(z)]

    native = run()
    monkeypatch.setattr(_lib, "_host", _lib._NoHost())
    assert all(torch.equal(a, b) for a, b in zip(run(), native, strict=True))
