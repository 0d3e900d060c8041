"""The lookup decode kernel for the widths and head dims without a kernel of their own, against the oracle: every code format
of a side, every head_dim, ragged tails, one lane and many, head groups, sketches, 16-bit and float32 uncompressed tokens."""

import ctypes as C

import numpy as np
import pytest
import torch

from gpu_util import host
from test_decode_gpu import _case, _check

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def other_kernels_only():
    """The one-launch kernel (test_decode_lane_gpu.py) would take most of these small calls."""
    from mlx_turboquant_b200.kernels import set_tuning
    set_tuning("decode_lane", 0)
    yield
    set_tuning("decode_lane", 1)


def _choice(c):
    from mlx_turboquant_b200 import _lib
    return _lib.lib().tq_decode_kernel_choice(C.byref(c._dargs))


def _run(c, q, ref, want=3):
    from mlx_turboquant_b200 import _lib
    out = c.attend(q, out_dtype=torch.float32)
    assert _choice(c) == want
    _check(out, ref)
    assert _lib.lib().tq_device_status() == 0
    return out


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("kb,vb", ((4, 4), (3, 2), (2, 3), (3.5, 2.5), (2.5, 3.5), (2, 2)))
@pytest.mark.parametrize("qjl", (False, True))
def test_every_format(oracle, d, kb, vb, qjl):
    rs = np.random.RandomState(d + int(10 * kb + vb))
    c, q, ref = _case(oracle, rs, 2, 8, 4, 333, d, kb, vb, 32, 8, qjl=qjl)
    _run(c, q, ref)


@pytest.mark.parametrize("b,hq,hkv,t", ((1, 8, 1, 2500), (1, 8, 8, 49), (3, 48, 3, 700), (70, 16, 16, 90), (1, 4, 4, 4000), (2, 12, 4, 130)))
@pytest.mark.parametrize("bf16", (False, True))
def test_lanes_runs_and_folds(oracle, b, hq, hkv, t, bf16):
    """Few long lanes (CTAs fold their warps' partials), a single short one, two head groups, more lanes than CTAs."""
    rs = np.random.RandomState(b + t)
    c, q, ref = _case(oracle, rs, b, hq, hkv, t, 128, 3.5, 4, 16, 4, bf16=bf16)
    _run(c, q, ref)


@pytest.mark.parametrize("t,rw,sink", ((600, 0, 0), (600, 16, 0), (600, 0, 8), (20, 64, 16), (300, 100, 128)))
def test_regions(oracle, t, rw, sink):
    rs = np.random.RandomState(t + rw + sink)
    c, q, ref = _case(oracle, rs, 2, 4, 2, t, 64, 4, 4, rw, sink)
    _run(c, q, ref)
    c, q, ref = _case(oracle, rs, 2, 4, 2, t, 96, 3, 4, rw, sink, dtype=np.float32)
    _run(c, q, ref)


@pytest.mark.parametrize("v_scale", (1e5, 1e-6))
@pytest.mark.parametrize("dt", ("fp32", "bf16"))
def test_value_norms_far_outside_the_fp16_range(oracle, v_scale, dt):
    rs = np.random.RandomState(13)
    c, q, ref = _case(oracle, rs, 2, 8, 8, 600, 128, 3, 3, 32, 16, dtype=np.float32, v_scale=v_scale, bf16=dt == "bf16", qjl=True)
    _run(c, q, ref)


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
def test_decode_steps_append_and_attend(dtype):
    from mlx_turboquant_b200 import TurboQuantKVCache
    g = torch.Generator(device="cuda").manual_seed(3)
    b, h, d = 2, 4, 128
    r = lambda n, hh=h: torch.randn(b, hh, n, d, device="cuda", generator=g).to(dtype)  # noqa: E731
    mk = lambda: TurboQuantKVCache(head_dim=d, num_kv_heads=h, key_bits=3, value_bits=4, residual_window=64, fp16_sink_size=16)  # noqa: E731
    c1, c2 = mk(), mk()
    k, v = r(500), r(500)
    c1.update(k, v)
    c2.update(k, v)
    for _ in range(5):
        kn, vn, q = r(1), r(1), r(1, 16) / d ** 0.5
        o1 = c1.decode_step(q, kn, vn)
        assert _choice(c1) == 3
        c2.update(kn, vn)
        assert torch.equal(o1, c2.attend(q))
    assert torch.equal(c1.keys[:, :, :c1._fp16_len], c2.keys[:, :, :c2._fp16_len])
    assert np.isfinite(host(o1.float())).all()


@pytest.mark.parametrize("d,b,hq,hkv,t,qjl,bf16", ((128, 64, 8, 4, 90, False, False), (128, 16, 8, 4, 120, False, True), (96, 2, 8, 4, 300, False, False),
                                                   (256, 1, 8, 2, 300, False, False), (128, 2, 8, 4, 250, True, False), (64, 2, 4, 2, 200, False, True)))
def test_four_and_two_bits_where_this_kernel_is_the_faster_one(oracle, d, b, hq, hkv, t, qjl, bf16):
    rs = np.random.RandomState(d + b)
    c, q, ref = _case(oracle, rs, b, hq, hkv, t, d, 4, 2, 32, 8, qjl=qjl, bf16=bf16)
    _run(c, q, ref)


@pytest.mark.parametrize("d,b,hq,hkv,t,rw,dt,want", ((128, 12, 12, 6, 300, 32, "bf16", 1), (128, 16, 8, 4, 120, 32, "fp32", 1), (128, 32, 16, 8, 60, 16, "fp16", 3),
                                                     (256, 16, 32, 4, 30, 64, "fp16", 0), (256, 4, 8, 1, 200, 128, "fp16", 3), (64, 6, 8, 4, 20, 64, "fp16", 0),
                                                     (96, 6, 8, 4, 20, 64, "fp32", 0), (128, 6, 8, 4, 20, 64, "bf16", 3), (64, 4, 8, 8, 200, 32, "fp32", 3)))
def test_calls_that_other_kernels_do_faster_stay_with_them(oracle, d, b, hq, hkv, t, rw, dt, want):
    """4-bit keys / 2-bit values, and caches without packed tokens: one launch of little code, or a wave of CTAs, is faster than this kernel's two."""
    rs = np.random.RandomState(d + b + t)
    c, q, ref = _case(oracle, rs, b, hq, hkv, t, d, 4, 2, rw, 8, dtype=np.float32 if dt == "fp32" else np.float16, bf16=dt == "bf16")
    _run(c, q, ref, want)
