"""Keys and values in layouts that repeat or overlap rows (an expanded head or batch axis, sliding windows): what the launches are
told about them (no GPU needed)."""

import pytest
import torch


def _side(b, h, cap, d):
    from mlx_turboquant_b200 import _lib
    from mlx_turboquant_b200.cache import _Side
    s = _Side(4)
    s.hi, s.norms = torch.zeros(b, h, cap, d // 2, dtype=torch.uint8), torch.zeros(b, h, cap)
    s.q_block = bytes(_lib.QuantizeArgs())
    return s


T, D = 7, 16


@pytest.mark.parametrize("shape,stride", (
    ((1, 3, T, D), (T * D, 0, D, 1)),            # one head seen as three
    ((4, 1, T, D), (0, T * D, D, 1)),            # one sequence seen as four
    ((4, 3, T, D), (0, 0, D, 1)),
    ((4, 3, T, D), (T * D, 0, D, 1)),
    ((4, 3, T, D), (0, T * D, D, 1)),
    ((2, 3, T, D), (3 * D, D, 0, 1)),            # one token seen as seven
    ((1, 1, T, D), (0, 0, D, 1)),                # a single lane: its stride is not looked at
    ((2, 3, 1, D), (3 * D, D, 0, 1)),            # a single token likewise
    ((1, 3, T, D), (T * 3 * D, D, 3 * D, 1)),    # a projection's output
    ((1, 3, T, D), (T * D, 2 * D, D, 1)),        # sliding windows
))
def test_quantize_job_addresses_every_row(shape, stride):
    from mlx_turboquant_b200 import _lib
    x = torch.as_strided(torch.arange(4096, dtype=torch.float16), shape, stride)
    b, h, t, d = shape
    a = _lib.QuantizeArgs()
    kept = _side(b, h, 16, d).quantize_job(a, x, 0)
    assert (a.n_lanes, a.n_rows) == (b * h, t)
    assert (b * h == 1 or a.x_lane_stride > 0) and (t == 1 or a.x_row_stride > 0)          # what the tensor-core kernel takes
    flat = torch.as_strided(kept, (kept.untyped_storage().nbytes() // 2,), (1,), 0)
    at = kept.storage_offset()
    for lane in range(b * h):
        for r in range(t):
            o = at + lane * a.x_lane_stride + r * a.x_row_stride
            assert torch.equal(flat[o:o + d], x[lane // h, lane % h, r])


@pytest.mark.parametrize("shape,stride,launched", (
    ((3, 1, T, D), (T * D, T * D, D, 1), True),
    ((3, 2, T, D), (2 * T * D, T * D, D, 1), True),
    ((1, 1, T, D), (D, D, D, 1), True),              # a single lane: its stride is not looked at
    ((3, 1, T, D), (D, D, D, 1), False),             # sequences that are windows over one run of tokens
    ((3, 1, T, D), (0, 0, D, 1), False),
    ((3, 2, T, D), (2 * D, D, D, 1), False),
))
def test_append_reads_every_row_where_it_is(monkeypatch, shape, stride, launched):
    from mlx_turboquant_b200 import _lib
    from mlx_turboquant_b200.cache import TurboQuantKVCache
    calls = []
    monkeypatch.setattr(_lib, "require_cuda", lambda *t: torch.device("cpu"))
    monkeypatch.setattr(_lib, "stream_ptr", lambda dev: 0)
    monkeypatch.setattr(_lib, "launch", lambda dev, name, *args: calls.append(args) or 0)
    k, v = (torch.as_strided(torch.randn(1024).half(), shape, stride) for _ in range(2))
    b, h, t, d = shape
    kb, vb = (torch.zeros(b, h, 20, d, dtype=torch.float16) for _ in range(2))
    TurboQuantKVCache._append(kb, vb, k, v, 5)
    assert bool(calls) == launched
    if launched:
        src, lanes, row_bytes, src_rows = calls[0][0], calls[0][4], calls[0][6], calls[0][7]
        assert src == k.data_ptr() and lanes == b * h
        assert b * h == 1 or src_rows * row_bytes == 2 * stride[1]
    else:
        assert torch.equal(kb[:, :, 5:5 + t], k) and torch.equal(vb[:, :, 5:5 + t], v)
