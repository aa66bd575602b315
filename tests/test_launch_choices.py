"""Which kernels a handle launches, by the rules on its systems' sizes, on the stand-in runtime."""
import pytest

from standin_runtime import run

PCLOSE = """
from helpers import config0_params, config1_params
from nuvort_b200.api import Handle
caps, tree = %r, %r
with Handle([config0_params()] * len(caps) + [config1_params("Tree")] * len(tree), caps + tree) as h:
    launched()
    h.stage("pclose")
    names = launched()
print([k for k in ("pclose_warps", "pclose_cells") if any(k in n for n in names)])
"""


@pytest.mark.parametrize("caps,tree,kernel", [
    ([600], [], "warps"), ([6144], [], "warps"), ([6145], [], "cells"),
    ([2200] * 8, [], "warps"), ([4200] * 8, [], "cells"),  # 3.9e7 and 1.4e8 pairs of slots
    ([800] * 64, [], "warps"), ([4200] * 512, [], "cells"),
    ([600], [100000], "warps"), ([600], [1000000], "cells"),  # a warp for every slot of the handle
])
def test_closest_points_of_systems_without_a_tree(tmp_path, caps, tree, kernel):
    assert f"['pclose_{kernel}']" in run(tmp_path, PCLOSE % (caps, tree))


def test_traffic_of_the_present_walk():
    # the walk by groups writes one sum a target, not 27: under 0.5 KB of DRAM a target, both ways
    import bench
    for workload, targets in (("tangle32k", 32768), ("tangle1m", 1048576), ("ensemble512", 2670000)):
        t = bench.present_traffic("k_tree_walk_mixed", workload)
        assert t["bytes_per_launch"] < 512 * targets and t["source"].endswith("k_tree_walk_mixed_groups.md")
    assert bench.present_traffic("k_tree_walk_fp64", "tangle32k") == bench.profile_traffic("k_tree_walk_fp64", "tangle32k")


MIXED = """
from helpers import config0_params
from nuvort_b200.api import Handle
caps = %r
with Handle([config0_params(precision="mixed")] * len(caps), caps) as h:
    launched()
    h.calc_velocity()
    names = launched()
print([w for w in (1, 8) if any("k_direct_mixedILi%%dE" %% w in n for n in names)])
"""


@pytest.mark.parametrize("caps,warps", [
    ([1000], [8]), ([88] * 2000, [1]), ([1000] * 4, [1]), ([1001] * 4, [8]), ([200] * 4, [8]),
    ([96] * 36, [8]), ([96] * 37, [1]),  # 2,916 and 2,997 items of 32 slots in 27 images, 20 an SM: 2,960
    ([88] * 2000 + [5000], [1, 8]),
])
def test_warps_of_the_mixed_direct_sum(tmp_path, caps, warps):
    assert str(warps) in run(tmp_path, MIXED % (caps,))
