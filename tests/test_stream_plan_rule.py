"""Which whole systems take k_trsv_stream: those of many short levels, in either precision; not natural-order
bars whose chunks wait for older values or hold a step or two, where k_trsv_task measured sooner."""
import pytest

from vshe import devices as D
from vshe import gpu
import test_local_plan as plans


@pytest.mark.parametrize("make, precision, stream", [
    (D.config1, "mixed", True), (D.config1, "fp64", True),                    # 3 to 4 slices a level
    (lambda: D.config3()[8], "mixed", True), (lambda: D.config3()[8], "fp64", True),
    (lambda: D.config2(50, 20, 60, 1), "mixed", True), (lambda: D.config2(50, 20, 60, 1), "fp64", False),  # 13, a few older values
    (lambda: D.config2(100, 25, 80, 1), "mixed", False),                      # 29, 33 thousand older values
    (lambda: D.config2(40, 10, 48, 3), "fp64", False),
])
def test_rule(make, precision, stream):
    rp, ci, v, _ = plans._system(make)
    kw = dict(plans.NAT, precision=precision)
    assert gpu.sweep_plan(rp, ci, None, **kw)["kind"] == 1
    assert (gpu.stream_plan(rp, ci, None, **kw) is not None) == stream
