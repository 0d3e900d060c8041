"""The one-launch decode kernel (a cluster of CTAs per cache lane) against the oracle: every code format and head_dim, every cluster size,
tiles that do and do not fill the warps, head groups, regions, appends, and that the rule for it leaves long contexts alone."""

import ctypes as C

import numpy as np
import pytest
import torch

import test_decode_gpu as general
import test_decode_lut_gpu as lookup
from test_decode_gpu import _case, _check

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lane():
    """lane(ctas): the kernel for every call that it can run, with so many CTAs per lane (0: its own choice)."""
    from mlx_turboquant_b200.kernels import set_tuning

    def force(ctas):
        set_tuning("decode_lane", 2)
        set_tuning("decode_lane_ctas", ctas)
    yield force
    set_tuning("decode_lane", 1)
    set_tuning("decode_lane_ctas", 0)


def _taken(c):
    from mlx_turboquant_b200 import _lib
    return _lib.lib().tq_decode_one_launch(C.byref(c._dargs))


def _choice(c):
    from mlx_turboquant_b200 import _lib
    return _lib.lib().tq_decode_kernel_choice(C.byref(c._dargs))


def _run(c, q, ref, ctas=0):
    from mlx_turboquant_b200 import _lib
    out = c.attend(q, out_dtype=torch.float32)
    got = _taken(c)
    assert got == ctas if ctas else got > 0
    assert _choice(c) == 4
    _check(out, ref)
    assert _lib.lib().tq_device_status() == 0


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("kb,vb", ((4, 2), (4, 4), (3, 2), (2, 3), (3.5, 2.5), (2.5, 3.5), (2, 2)))
@pytest.mark.parametrize("qjl", (False, True))
def test_every_format(oracle, lane, d, kb, vb, qjl):
    rs = np.random.RandomState(d + int(10 * kb + vb))
    c, q, ref = _case(oracle, rs, 2, 8, 4, 333, d, kb, vb, 32, 8, qjl=qjl, bf16=qjl)
    lane(0)
    _run(c, q, ref)


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("ctas", (1, 2, 3, 4, 5, 6, 8, 12, 16))
def test_every_cluster_size(oracle, lane, d, ctas):
    """More warps than tiles, and a few tiles per warp; d / ctas columns per CTA with remainders."""
    rs = np.random.RandomState(d + ctas)
    lane(ctas)
    for t in (100, 900):
        c, q, ref = _case(oracle, rs, 1, 12, 2, t, d, 3, 4, 16, 4, bf16=ctas % 2 == 0, qjl=d != 128)
        _run(c, q, ref, ctas)


@pytest.mark.parametrize("b,hq,hkv,t,rw,sink", ((1, 8, 8, 49, 16, 4), (3, 48, 3, 700, 16, 4), (70, 16, 16, 90, 16, 4), (1, 4, 1, 33, 0, 0), (2, 8, 2, 400, 0, 8),
                                                  (2, 8, 2, 400, 150, 0), (1, 8, 1, 1000, 128, 128)))
@pytest.mark.parametrize("bf16", (False, True))
def test_heads_lanes_and_regions(oracle, lane, b, hq, hkv, t, rw, sink, bf16):
    rs = np.random.RandomState(b + t)
    c, q, ref = _case(oracle, rs, b, hq, hkv, t, 128, 4, 2, rw, sink, bf16=bf16)
    lane(0)
    _run(c, q, ref)


@pytest.mark.parametrize("v_scale", (1e5, 1e-6))
def test_value_norms_far_outside_the_fp16_range(oracle, lane, v_scale):
    rs = np.random.RandomState(13)
    c, q, ref = _case(oracle, rs, 2, 8, 8, 600, 128, 3, 3, 32, 16, dtype=np.float32, v_scale=v_scale, bf16=True, qjl=True)
    lane(3)
    _run(c, q, ref, 3)


def test_steps_append(lane):
    """The appended token counts, and its rows are in the buffer: steps equal update followed by attend; across a drain too."""
    from mlx_turboquant_b200 import TurboQuantKVCache
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda n, h=4: torch.randn(2, h, n, 96, device="cuda", generator=g).bfloat16()  # noqa: E731
    cs = [TurboQuantKVCache(head_dim=96, num_kv_heads=4, key_bits=3.5, value_bits=3, residual_window=32, fp16_sink_size=16) for _ in range(2)]
    k, v = r(300), r(300)
    for c in cs:
        c.update(k, v)
    lane(4)
    for _ in range(40):
        kn, vn, q = r(1), r(1), r(1, 16) / 96 ** 0.5
        o = cs[0].decode_step(q, kn, vn)
        cs[1].update(kn, vn)
        assert torch.equal(o, cs[1].attend(q))
    n = cs[0]._fp16_len
    assert n == cs[1]._fp16_len and torch.equal(cs[0].keys[:, :, :n], cs[1].keys[:, :, :n]) and torch.equal(cs[0].values[:, :, :n], cs[1].values[:, :, :n])


def test_what_it_leaves_to_the_others(oracle, lane):
    """float32 rows, caches without packed tokens and, by its rule, long contexts of many lanes."""
    from mlx_turboquant_b200 import _lib
    from mlx_turboquant_b200.kernels import set_tuning
    lane(0)
    takes = lambda c: _lib.lib().tq_decode_one_launch(C.byref(c._dargs))  # noqa: E731
    for t, dtype in ((300, np.float32), (20, np.float16)):
        c, q, ref = _case(oracle, np.random.RandomState(t), 2, 8, 2, t, 128, 4, 2, 32, 8, dtype=dtype)
        _check(c.attend(q, out_dtype=torch.float32), ref)
        assert takes(c) == 0 and _choice(c) != 4
    set_tuning("decode_lane", 1)
    from mlx_turboquant_b200 import TurboQuantKVCache
    for b, t, want in ((8, 16384, False), (1, 600, True)):
        c = TurboQuantKVCache(head_dim=128, num_kv_heads=8, key_bits=4, value_bits=2, residual_window=128, fp16_sink_size=128)
        x = torch.randn(b, 8, t, 128, device="cuda").half()
        c.update(x, x)
        c.attend(torch.zeros(b, 32, 1, 128, device="cuda").half())
        assert (takes(c) > 0) == want == (_choice(c) == 4)


def test_a_split_count_that_is_asked_for(oracle):
    """goes to the kernels that split, whatever the rule says of the call."""
    from mlx_turboquant_b200.kernels import set_tuning
    c, q, ref = _case(oracle, np.random.RandomState(7), 1, 8, 2, 700, 128, 4, 2, 32, 16)
    try:
        for splits, want in ((0, 4), (3, 1), (0, 4)):
            set_tuning("decode_splits", splits)
            _check(c.attend(q, out_dtype=torch.float32), ref)
            assert _choice(c) == want
    finally:
        set_tuning("decode_splits", 0)


@pytest.fixture()
def off():
    from mlx_turboquant_b200.kernels import set_tuning
    set_tuning("decode_lane", 0)
    yield
    set_tuning("decode_lane", 1)


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("kb,vb", ((4, 4), (3, 2), (2, 3), (3.5, 2.5), (2.5, 3.5), (2, 2)))
@pytest.mark.parametrize("qjl", (False, True))
def test_the_lookup_kernel_where_this_one_would_take_the_call(oracle, off, d, kb, vb, qjl):
    lookup.test_every_format(oracle, d, kb, vb, qjl)


@pytest.mark.parametrize("b,hq,hkv,t", ((1, 8, 1, 2500), (3, 48, 3, 700), (70, 16, 16, 90), (2, 12, 4, 130)))
def test_lookup_kernel_lanes_and_folds(oracle, off, b, hq, hkv, t):
    lookup.test_lanes_runs_and_folds(oracle, b, hq, hkv, t, True)


@pytest.mark.parametrize("t", (129, 300, 2500))
def test_the_table_lookup_kernel(oracle, off, t):
    general.test_k4v2_direct_path_lengths(oracle, t)


@pytest.mark.parametrize("ctas", (1, 4))
@pytest.mark.parametrize("d,kb,vb,dtype", ((128, 4, 2, torch.float16), (96, 3.5, 3, torch.bfloat16), (64, 3, 4, torch.bfloat16), (256, 4, 4, torch.float16)))
@pytest.mark.parametrize("where", ("new key", "packed norms", "value without weight"))
def test_nan_reaches_the_result(lane, ctas, d, kb, vb, dtype, where):
    """A warp whose every score is NaN, or whose weight is 0 and a value NaN: float arithmetic gives NaN for the query heads of that KV head
    (0 x NaN is NaN, in the softmax sum and in the values), as the other decode kernels do, and leaves the other KV head's alone."""
    from mlx_turboquant_b200 import TurboQuantKVCache
    g = torch.Generator(device="cuda").manual_seed(d)
    r = lambda n, h=2: torch.randn(1, h, n, d, device="cuda", generator=g).to(dtype)  # noqa: E731
    c = TurboQuantKVCache(head_dim=d, num_kv_heads=2, key_bits=kb, value_bits=vb, residual_window=32, fp16_sink_size=16)
    c.update(r(300), r(300))
    while (c._sink_len + c._fp16_len) % 16:
        c.update(r(1), r(1))
    q, k, v = r(1, 8) / d ** 0.5, r(1), r(1)
    columns = slice(None)
    if where == "new key":                  # alone in the last uncompressed tile
        k[0, 0] = float("nan")
    elif where == "packed norms":           # a whole packed tile
        c._k.norms[0, 0, 32:48] = float("nan")
    else:                                   # scores of 300 and more: exp leaves nothing for the recent tokens
        c.sink_keys[0, 0, 0] = 300 * d ** 0.5 * q[0, :4, 0].sum(0)
        c.values[0, 0, 25, 7] = float("nan")
        columns = 7
    lane(ctas)
    out = c.decode_step(q, k, v)[0, :, 0]
    assert _taken(c) == ctas
    assert out[:4, columns].isnan().all()
    assert out[4:].isfinite().all()


def test_the_rule_and_the_sizes(oracle):
    """A bound turns calls away before their plans are made: none with a plan that the rule would take.  (With a forced size the rule sees that plan
    alone, so it takes the call at some forced size exactly when it takes it at the size of its choice.)"""
    from mlx_turboquant_b200 import _lib
    from mlx_turboquant_b200.kernels import set_tuning
    f = _lib.lib().tq_decode_one_launch
    taken = 0
    for b, h, t, d in ((1, 8, 600, 128), (1, 2, 3000, 128), (4, 8, 2000, 96), (1, 8, 9000, 64), (16, 8, 700, 128), (2, 4, 6000, 256), (1, 1, 20000, 128), (40, 8, 300, 64)):
        a = _lib.DecodeArgs(batch=b, n_q_heads=4 * h, n_kv_heads=h, d=d, c_len=t, c_lane_stride=(t + 15) // 16 * 16, k_bits_hi=3, v_bits_hi=3, sink_len=128, sink_lane_stride=128,
                            res_len=100, res_lane_stride=512, scale=0.1, v_cent_scale_hi=1.0, v_cent_scale_lo=1.0, workspace_bytes=1 << 40)
        for name in ("q", "rot", "k_hi", "v_hi", "k_norms", "v_norms", "k_cent_hi", "v_cent_hi", "sink_k", "sink_v", "res_k", "res_v", "out", "workspace"):
            setattr(a, name, 1 << 40)                                    # (aligned; nothing is launched)
        own = f(C.byref(a))
        forced = set()
        for ctas in (1, 2, 3, 4, 5, 6, 8, 12, 16):
            set_tuning("decode_lane_ctas", ctas)
            forced.add(f(C.byref(a)))
        set_tuning("decode_lane_ctas", 0)
        assert own >= 0 and own in forced and (own > 0) == (max(forced) > 0)
        taken += own > 0
    assert 0 < taken < 8


FIRST_CALL = """
import ctypes as C, torch
from mlx_turboquant_b200 import TurboQuantKVCache, _lib
g = torch.Generator(device="cuda").manual_seed(1)
r = lambda h, n: torch.randn(1, h, n, 128, device="cuda", generator=g).half()
c = TurboQuantKVCache(head_dim=128, num_kv_heads=4, key_bits=3, value_bits=3, residual_window=32, fp16_sink_size=16)
c.update(r(4, 500), r(4, 500))
q = r(16, 1) / 11
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = c.attend(q)
assert _lib.lib().tq_decode_kernel_choice(C.byref(c._dargs)) == 4
out.zero_()
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, c.attend(q)) and out.abs().max() > 0 and _lib.lib().tq_device_status() == 0
"""


def test_the_first_call_of_a_process_under_capture():
    """What the kernel asks the device for once (where its shared memory begins, how many clusters fit) must not end the capture."""
    import subprocess
    import sys
    from pathlib import Path
    run = subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr
