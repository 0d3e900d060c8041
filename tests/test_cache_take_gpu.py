"""Tokens that leave the recent-token buffer at once are quantized from the caller's tensors: every way the split between
buffer and newcomers can fall, against the reference's state machine (the oracle), and odd layouts of the newcomers."""

import numpy as np
import pytest
import torch

from gpu_util import cu, host, host_tables, kv_like

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rw,chunk,sink,steps", (
    (16, 0, 0, (300,)),                       # a fresh cache: nothing in the buffer
    (16, 0, 4, (2, 5, 300)),                  # the last call straddles sink, buffer and newcomers
    (16, 0, 0, (30, 1, 1, 1, 1)),             # the due tokens all sit in the buffer
    (16, 0, 0, (20, 200, 33, 1, 40)),         # buffer and newcomers
    (32, 8, 4, (38, 3, 70, 1, 9, 600)),       # chunks shorter than the buffer: part of the buffer stays
    (0, 0, 0, (1, 7, 300)),                   # nothing stays
))
@pytest.mark.parametrize("strided", (False, True))
def test_compressed_tokens_and_buffers_match_the_state_machine(rw, chunk, sink, steps, strided):
    from mlx_turboquant_b200 import TurboQuantKVCache
    from oracle import tq_oracle as orc
    d, h, b = 64, 3, 2
    rs = np.random.RandomState(11)
    n = sum(steps)
    k, v = kv_like(rs, (b, h, n, d)), kv_like(rs, (b, h, n, d))
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=h, residual_window=rw, chunk_size=chunk, fp16_sink_size=sink)
    ref = orc.KVCacheOracle(d, host_tables(d), 4, 2, rw, fp16_sink_size=sink, chunk_size=chunk)
    at = 0
    for t in steps:
        kt, vt = cu(k[:, :, at:at + t]), cu(v[:, :, at:at + t])
        if strided:                           # (B, T, H, D) storage seen as (B, H, T, D): a projection's output
            kt, vt = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (kt, vt))
        c.update(kt, vt)
        ref.update_and_fetch(k[:, :, at:at + t], v[:, :, at:at + t])
        at += t
        assert (c._compressed_len, c._fp16_len) == (ref.comp_len, ref.fp_len)
    assert np.array_equal(host(c.keys[:, :, :c._fp16_len]), ref.k[:, :, :ref.fp_len])
    assert np.array_equal(host(c.values[:, :, :c._fp16_len]), ref.v[:, :, :ref.fp_len])
    if sink:
        assert np.array_equal(host(c.sink_keys), k[:, :, :sink])
    if c._compressed_len:
        assert (host(c._compressed_keys) == ref.comp["k"][0][:, :, :ref.comp_len]).mean() > 0.999
        assert (host(c._compressed_values) == ref.comp["v"][0][:, :, :ref.comp_len]).mean() > 0.999


def test_newcomers_of_another_dtype_take_the_buffers():
    from mlx_turboquant_b200 import TurboQuantKVCache
    x = torch.randn(1, 2, 200, 64, device="cuda")
    c = TurboQuantKVCache(head_dim=64, num_kv_heads=2, residual_window=16)
    c.update(x[:, :, :10].half(), x[:, :, :10].half())
    c.update(x[:, :, 10:60], x[:, :, 10:60])
    assert c.keys.dtype == torch.float16 and torch.equal(c.keys[:, :, :c._fp16_len], x[:, :, 44:60].half())


@pytest.mark.parametrize("d", (64, 128, 256))
@pytest.mark.parametrize("axis", (0, 1))
def test_expanded_newcomers_equal_their_copies(d, axis):
    from mlx_turboquant_b200 import TurboQuantKVCache, kernels
    shape, full = ((1, 1, 300, d), (3, 1, 300, d) if axis == 0 else (1, 3, 300, d))
    k, v = (torch.randn(*shape, device="cuda").half() for _ in range(2))
    cs = [TurboQuantKVCache(head_dim=d, num_kv_heads=full[1], residual_window=16, fp16_sink_size=4) for _ in range(2)]
    cs[0].update(k.expand(full), v.expand(full))
    cs[1].update(k.expand(full).contiguous(), v.expand(full).contiguous())
    assert all(x is y is None or torch.equal(x, y) for x, y in zip(cs[0].state, cs[1].state))
    c = cs[1]
    got, want = (kernels.quantize_pack(x, c._rotation, c._k.bnd_hi, 4) for x in (k.expand(full), k.expand(full).contiguous()))
    assert (got[0] == want[0]).float().mean() > 0.999 and torch.allclose(got[2], want[2], rtol=1e-5)     # (the row kernel takes the expanded one)


@pytest.mark.parametrize("d,qjl", ((256, False), (64, True), (64, False)))
def test_a_second_continuation_does_not_see_the_first_one(d, qjl):
    from mlx_turboquant_b200 import TurboQuantKVCache
    x = [torch.randn(1, 2, 40, d, device="cuda").half() for _ in range(3)]
    make = lambda: TurboQuantKVCache(head_dim=d, num_kv_heads=2, residual_window=0, qjl_correction=qjl)   # noqa: E731
    c, ref = make(), make()
    c.update_and_fetch(x[0], x[0])
    mark = c.meta_state
    c.update_and_fetch(x[1], x[1])
    c.meta_state = mark
    ref.update(x[0], x[0])
    got, want = c.update_and_fetch(x[2], x[2]), ref.update_and_fetch(x[2], x[2])
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
