"""Cache lanes and query rows of a several-query-token call done in rounds for want of workspace: no round may use more than the
workspace holds, whatever the sizes (host arithmetic; the library's planning for 148 SMs where no device answers)."""

import random

import pytest


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as g
    g.build()
    from mlx_turboquant_b200 import _lib
    return _lib.lib()


# a last round of fewer lanes, planned by itself, chose more key ranges than fit
@pytest.mark.parametrize("b,hq,hkv,d,total,tq", ((13, 32, 8, 128, 120026, 5281), (15, 16, 2, 256, 40000, 2048), (7, 8, 1, 256, 45056, 4096), (50, 32, 8, 128, 65536, 2048)))
@pytest.mark.parametrize("dense", (0, 1, 384, 5000))
def test_uneven_rounds_fit_the_reported_workspace(lib, b, hq, hkv, d, total, tq, dense):
    need = lib.tq_prefill_workspace_bytes(b, hq, hkv, d, total, tq)
    assert 0 < lib.tq_prefill_workspace_used(b, hq, hkv, d, total - dense, dense, tq, need) <= need


def test_every_round_fits_any_workspace_that_is_taken(lib):
    rng = random.Random(5)
    for _ in range(4000):
        d, hkv, g = rng.choice((64, 96, 128, 256)), rng.choice((1, 2, 3, 8)), rng.choice((1, 2, 3, 4, 8, 12))
        b, total = rng.randint(1, 20), int(10 ** rng.uniform(1.5, 5.2))
        tq, dense = min(total, int(10 ** rng.uniform(0.3, 3.8))), rng.choice((0, total, rng.randint(0, total), min(total, rng.randint(1, 400))))
        all_lanes, one = lib.tq_prefill_workspace_bytes(b, hkv * g, hkv, d, total, tq), lib.tq_prefill_workspace_bytes(1, g, 1, d, total, tq)
        for lent in (all_lanes, one, int(one + rng.random() ** 2 * max(0, all_lanes - one))):
            used = lib.tq_prefill_workspace_used(b, hkv * g, hkv, d, total - dense, dense, tq, lent)
            assert 0 < used <= lent, (b, g, hkv, d, total, dense, tq, lent)


def test_partials_stay_small(lib):
    """The rows of a long cache need what they need; the partials of many query rows do not come on top without a limit."""
    rows, queries = 2 * 128 * (1 << 20) * 2, 2 * 8 * 32768 * 128 * 2
    assert lib.tq_prefill_workspace_bytes(1, 8, 1, 128, 1 << 20, 32768) < rows + queries + 2 ** 28
    assert lib.tq_prefill_workspace_bytes(64, 32, 8, 128, 32768, 2048) <= 2 ** 29
