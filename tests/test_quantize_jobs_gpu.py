"""Quantize jobs of one compression that share the SMs, against the same jobs one by one: the same bytes, norms and sketches."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _lanes(dtype, d, h, n, seed):
    return torch.randn(1, h, n, d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("d,kb,vb,qjl", ((64, 4, 4, False), (96, 4, 2, True), (128, 3.5, 3.5, False), (256, 4, 2, False)))
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16, torch.float32))
@pytest.mark.parametrize("h,sizes", ((1, (1, 1)), (3, (129, 128, 1, 300)), (8, (1, 2400)), (37, (512, 512)), (8, (9472, 9472)), (8, (9473, 9472, 100))))
def test_jobs_side_by_side(d, kb, vb, qjl, dtype, h, sizes):
    """One tile a job; jobs of unlike sizes; as many tiles as SMs; the last total that shares them at eight tiles per CTA, and one above it."""
    from mlx_turboquant_b200 import TurboQuantKVCache, _lib
    if d == 256 and h * max(sizes) > 40000:
        sizes = tuple(max(1, n // 4) for n in sizes)
    dev = torch.device("cuda", torch.cuda.current_device())
    total = sum(sizes)

    def run(together):
        c = TurboQuantKVCache(head_dim=d, num_kv_heads=h, key_bits=kb, value_bits=vb, fp16_sink_size=0, residual_window=16, qjl_correction=qjl)
        jobs, alive, at = (_lib.QuantizeArgs * 4)(), [], 0
        c._bind(dev)
        for side in (c._k, c._v):
            side.reserve(1, h, d, total, 0, dev, qjl)
            for t in (side.hi, side.lo, side.norms, side.qbits, side.qgamma):
                if t is not None:
                    t.zero_()
        for i, n in enumerate(sizes):
            alive.append((c._k, c._v)[i % 2].quantize_job(jobs[i], _lanes(dtype, d, h, n, i), at))
            at += n
        if together:
            _lib.check(_lib.launch(dev, "tq_quantize_pack_many", jobs, len(sizes), _lib.stream_ptr(dev)))
        else:
            for i in range(len(sizes)):
                _lib.check(_lib.launch(dev, "tq_quantize_pack", jobs[i], _lib.stream_ptr(dev)))
        torch.cuda.synchronize()
        return [t for s in (c._k, c._v) for t in (s.hi, s.lo, s.norms, s.qbits, s.qgamma) if t is not None]

    for x, y in zip(run(True), run(False)):
        assert torch.equal(x, y)
