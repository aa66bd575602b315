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
