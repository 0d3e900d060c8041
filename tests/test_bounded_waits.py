"""Kernels whose roles wait on one another end those waits after a limit, and a role that gives up goes straight to the teardown.  A hardware
barrier that only part of the CTA takes has no limit: one warp that gave up leaves the others of it waiting for good.  So between roles there
are mbarriers only; hardware barriers are for all threads of a CTA (__syncthreads, barrier 0), before the roles part and after they meet."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mlx_turboquant_b200" / "csrc"
BOUNDED = sorted(p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh") and "mbarrier.try_wait" in p.read_text())


def test_the_kernels_are_found():
    assert {"prefill_fa.cu", "quantize_tc.cu"} <= set(BOUNDED)


@pytest.mark.parametrize("name", BOUNDED)
def test_no_barrier_of_part_of_a_cta(name):
    code = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for m in re.finditer(r"\b(?:barrier(?:\.cta)?\.(?:sync|arrive|red)|bar\.(?:sync|arrive|red))[^;]*;", code):
        assert re.fullmatch(r"barrier\.sync 0;", m.group()), f"{name}: {m.group()}"
