"""The wavefront pass is credited with no byte that it does not move: the
algorithmic bytes stay at or below the DRAM traffic that a capture measured (2 %
for what a pass finds in L2 from the one before: 126 MB of 233 MB in FP32)."""
import pytest

from cgli_fu_flow_b200 import roofline
from cgli_fu_flow_b200.channel import Channel


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pass_bytes_are_moved(precision):
    r = roofline.sweep_roofline(Channel(160, 128, 128), 0.2, precision)
    assert r["algorithmic_bytes_per_launch"] <= 1.02 * r["traffic"]
    w = roofline.sweep_roofline(Channel(160, 128, 128, wavy=True), 0.2, precision)
    assert w["traffic"] is None
    assert w["algorithmic_bytes_per_launch"] > r["algorithmic_bytes_per_launch"]
