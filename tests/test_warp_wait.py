"""Waits of a whole warp: each lane polls with its own clock, but all lanes get
one answer, because what follows (elect.sync, TMEM loads) needs them all."""
import glob
import os
import re

import pytest

import gatlas_b200 as g

KERNELS = os.path.join(os.path.dirname(os.path.abspath(g.__file__)), "csrc", "kernels")


@pytest.mark.gpu
def test_lanes_that_disagree_leave_together(cuda):
    g.device_faults(clear=True)
    assert g.selftest_warp_wait() == (0, 1)
    assert g.device_faults(clear=True) == g.FAULT_SELFTEST_WAIT


def test_limits_are_checked_before_any_device_work():
    for limit in (0, 5_000_000_000):
        with pytest.raises(g.GatlasError, match="limit"):
            g.selftest_warp_wait(limit_ns=limit)


def test_single_lane_waits_stand_under_a_single_lane():
    """The lane-wise wait is called by one thread only: its call, or the branch
    around it, names lane 0 or thread 0; the pair relay's wait is named for it."""
    calls = 0
    for path in sorted(glob.glob(os.path.join(KERNELS, "*.cu*"))):
        lines = open(path).read().split("\n")
        for i, line in enumerate(lines):
            if not re.search(r"\bwait_timed(_cluster)?\(", line):
                continue
            calls += 1
            depth = len(line) - len(line.lstrip())
            around = [line]
            for above in reversed(lines[:i]):
                if above.strip() and len(above) - len(above.lstrip()) < depth:
                    around.append(above)
                    depth = len(above) - len(above.lstrip())
            assert any(re.search(r"lane == 0|threadIdx\.x == 0|auto wait_lane", a) for a in around), \
                f"{os.path.basename(path)}:{i + 1}: {line.strip()}"
    assert calls > 0


def test_aligned_cluster_barriers_stand_behind_a_converged_warp():
    """barrier.cluster's aligned forms appear once, in the helper that
    converges the warp first."""
    uses = []
    for path in sorted(glob.glob(os.path.join(os.path.dirname(KERNELS), "**", "*.cu*"), recursive=True)):
        text = open(path).read()
        uses += [text[:m.start()] for m in re.finditer(r"barrier\.cluster\.arrive[a-z.]*\.aligned", text)]
    assert len(uses) == 1
    assert re.search(r"void cluster_sync\(\) \{\n    __syncwarp\(\);\n    asm volatile\(\"$", uses[0])
