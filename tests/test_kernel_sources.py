"""Rules of the CUDA sources that no run can show without risk to the GPU, checked on their text."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "oasr_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"\btmem_alloc(_pair)?\(", _code(p))))
def test_tensor_memory_is_allocated_before_dependents_may_start(name):
    """A dependent that starts early can allocate tensor memory on the same SM and then wait for this kernel: a kernel that
    triggered before its own allocation could wait for those columns without end."""
    kernel_allocs = 0
    for body in re.split(r"\n(?=(?:template|__global__|__device__))", _code(CSRC / name)):
        alloc = re.search(r"\btmem_alloc(_pair)?\(", body)
        if alloc is None:
            continue
        kernel_allocs += 1
        trigger = body.find("grid_dep_launch()")
        assert trigger < 0 or trigger > body.rfind("tmem_alloc"), f"{name}: grid_dep_launch() before the allocation"
    assert kernel_allocs


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*") if "mbar_test(" in _code(p)))
def test_a_warp_counts_a_barrier_as_complete_only_if_every_lane_has_seen_it(name):
    """mbarrier tests acquire for the lane that sees the phase complete; a vote carries no ordering to the others, and the lane
    that issues the copy or the MMA behind it may be any of them."""
    assert not re.search(r"__(any|ballot)_sync\b", _code(CSRC / name))
