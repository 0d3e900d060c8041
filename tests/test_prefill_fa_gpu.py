"""The two-step attention for several query tokens where its tiles can go wrong: key counts around multiples of 64 and 128, query
counts around a block's rows, key ranges split over CTAs, every head_dim, lanes done in rounds for want of workspace.  Reference:
float32 attention over the cache's dense rows."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(d, b, hq, hkv, t, tq, dtype, kb=3.5, vb=4):
    from mlx_turboquant_b200 import TurboQuantKVCache
    g = torch.Generator(device="cuda").manual_seed(d + t + tq)
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=hkv, key_bits=kb, value_bits=vb, residual_window=16, fp16_sink_size=5)
    k, v = (torch.randn(b, hkv, t, d, device="cuda", generator=g) for _ in range(2))
    k, v = k.to(dtype), (v * torch.exp(torch.randn(b, hkv, t, 1, device="cuda", generator=g))).to(dtype)
    q = (torch.randn(b, hq, tq, d, device="cuda", generator=g) / d ** 0.5).to(dtype)
    dk, dv = (x.float().repeat_interleave(hq // hkv, 1) for x in c.update_and_fetch(k, v))
    s = (q.float() @ dk.transpose(-1, -2)) * d ** -0.5
    pos = torch.arange(t, device="cuda")
    s = s.masked_fill(pos[None, :] > (t - tq + torch.arange(tq, device="cuda"))[:, None], float("-inf"))
    return c, q, torch.softmax(s, -1) @ dv


def _check(out, ref):
    from mlx_turboquant_b200 import _lib
    err = float((out.float() - ref).abs().max() / ref.abs().max())
    assert err < 1e-3, err
    assert _lib.lib().tq_device_status() == 0


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("b,hq,hkv,t,tq", ((1, 4, 4, 64, 2), (2, 4, 2, 65, 65), (1, 8, 1, 127, 33), (1, 8, 2, 129, 64), (2, 16, 1, 1500, 3), (1, 4, 4, 3001, 257),
                                            (3, 12, 4, 640, 129)))
def test_tile_and_block_edges(d, dtype, b, hq, hkv, t, tq):
    c, q, ref = _case(d, b, hq, hkv, t, tq, dtype)
    _check(c.attend(q, out_dtype=torch.float32), ref)


@pytest.mark.parametrize("d", (64, 128, 256))
@pytest.mark.parametrize("b,hkv,lent", ((3, 4, 1), (5, 2, 3)))              # one lane at a time; three at a time, the last round has one
def test_lanes_in_rounds(d, b, hkv, lent):
    from mlx_turboquant_b200 import _lib
    c, q, ref = _case(d, b, 2 * hkv, hkv, 700, 40, torch.float16, 4, 2)
    out = torch.empty(b, 2 * hkv, 40, d, device="cuda")
    a = c._fill_decode_args(b, 2 * hkv, q.dtype, out.dtype, None)
    a.q, a.out, a.c_len, a.sink_len, a.res_len = q.data_ptr(), out.data_ptr(), c._compressed_len, c._sink_len, c._fp16_len
    need = _lib.lib().tq_prefill_workspace_bytes(lent, 2, 1, d, 700, 40)
    assert need < _lib.lib().tq_prefill_workspace_bytes(b, 2 * hkv, hkv, d, 700, 40)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    _lib.check(_lib.lib().tq_prefill_attn(C.byref(a), 40, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    _check(out, ref)


@pytest.mark.parametrize("d,kb,vb", ((128, 4, 2), (128, 3.5, 3.5), (64, 4, 4), (256, 4, 2)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("room", ("one lane", "none"))
def test_a_card_without_room_for_the_scratch(monkeypatch, d, kb, vb, dtype, room):
    from mlx_turboquant_b200 import kernels
    c, q, ref = _case(d, 2, 8, 2, 900, 80, dtype, kb, vb)
    full = kernels.scratch
    monkeypatch.setattr(kernels, "scratch", lambda dev, *sizes: full(dev, sizes[-1]) if room == "one lane" else None)
    _check(c.attend(q, out_dtype=torch.float32), ref)


def test_float32_queries_need_no_scratch(monkeypatch):
    from mlx_turboquant_b200 import kernels
    c, q, ref = _case(128, 1, 8, 2, 500, 70, torch.float32, 4, 2)
    monkeypatch.setattr(kernels, "scratch", lambda *a: pytest.fail("scratch asked for"))
    _check(c.attend(q), ref)


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("kb,vb", ((4, 2), (3.5, 3.5), (2, 4)))
@pytest.mark.parametrize("loud", (1.0, 8.0))
def test_as_close_to_64_bits_as_the_kernel_that_unpacks_as_it_goes(d, kb, vb, loud):
    """The same operands rounded to fp16 (rotated queries, centroids, weights) and float32 sums: no further off, up to the scatter of
    some 10,000 outputs' root mean square."""
    from mlx_turboquant_b200 import TurboQuantKVCache, kernels
    g = torch.Generator(device="cuda").manual_seed(7)
    t, tq, h = 2500, 60, 2
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=h, key_bits=kb, value_bits=vb, residual_window=64, fp16_sink_size=10)
    k, v = ((torch.randn(1, h, t, d, device="cuda", generator=g) * torch.exp(0.5 * torch.randn(1, h, t, 1, device="cuda", generator=g))).half() for _ in range(2))
    q = (torch.randn(1, 4 * h, tq, d, device="cuda", generator=g) * loud / d ** 0.5).half()
    dk, dv = (x.double().repeat_interleave(4, 1) for x in c.update_and_fetch(k, v))
    s = (q.double() @ dk.transpose(-1, -2)) * d ** -0.5
    s = s.masked_fill(torch.arange(t, device="cuda")[None, :] > (t - tq + torch.arange(tq, device="cuda"))[:, None], float("-inf"))
    ref = torch.softmax(s, -1) @ dv
    err = []
    for tc in (1, 0):
        kernels.set_tuning("prefill_tc", tc)
        err.append(float((c.attend(q, out_dtype=torch.float32) - ref).norm() / ref.norm()))
    kernels.set_tuning("prefill_tc", 1)
    assert err[0] < 1.1 * err[1], err


@pytest.mark.parametrize("b,tq,unpacks", ((16, 16, True), (16, 33, False), (8, 16, False)))
def test_a_block_of_query_rows_over_many_long_lanes_unpacks_as_it_goes(monkeypatch, b, tq, unpacks):
    """128 query rows per lane: where waves of one CTA per lane are the faster way, the result is that kernel's, bit for bit (it is what
    runs without scratch); other calls take the expansion."""
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib, kernels
    g = torch.Generator(device="cuda").manual_seed(2)
    c = TurboQuantKVCache(head_dim=128, num_kv_heads=8, key_bits=4, value_bits=2, fp16_sink_size=128)
    x = torch.randn(b, 8, 8192, 128, device="cuda", generator=g).half()
    c.update(x, x)
    q = torch.randn(b, 32, tq, 128, device="cuda", generator=g).half() / 11
    got = c.attend(q, out_dtype=torch.float32)
    monkeypatch.setattr(kernels, "scratch", lambda *a: None)
    want = c.attend(q, out_dtype=torch.float32)
    assert torch.equal(got, want) == unpacks and (got - want).abs().max() < 1e-3 * want.abs().max()
    assert _lib.lib().tq_device_status() == 0


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("hq,hkv,tq", ((2, 2, 17), (8, 2, 4), (8, 2, 5), (6, 2, 33), (16, 2, 2), (16, 2, 34), (4, 4, 129)))
@pytest.mark.parametrize("t", (140, 2000))                                  # one key range; several, merged from float32 partials
def test_rows_of_16_and_result_types(d, dtype, hq, hkv, tq, t):
    """Query rows that fill some of the sixteen-row shares of a block: the others take no part.  A 16-bit result is the float32 one, rounded."""
    c, q, ref = _case(d, 1, hq, hkv, t, tq, dtype)
    out = c.attend(q, out_dtype=torch.float32)
    _check(out, ref)
    for out_dtype in (torch.float16, torch.bfloat16):
        assert torch.equal(c.attend(q, out_dtype=out_dtype), out.to(out_dtype))
