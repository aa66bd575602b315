"""The closest-point search of ensembles without a tree, on either side of the lines between the
search by a warp per target and the cell list: the pairs of slots of all such systems together,
and the slots of the handle, tree systems' among them.  Equal to the oracle's either way."""
import numpy as np
import pytest

from helpers import config0_params, config1_params, tangle
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sys,cap", [(6, 3162), (6, 3163), (40, 1224), (40, 1225)])
def test_either_side_of_the_pairs(n_sys, cap):
    from nuvort_b200.api import Handle
    p = config0_params()
    states = [tangle(200 + s % 3, 0.002, n_points=500) for s in range(n_sys)]
    want = []
    for st in states[:3]:
        o = Oracle(p, st, t=0.0, itime=1)
        o.stage("pclose")
        want.append(o.download())
    with Handle([p] * n_sys, [cap] * n_sys, states=states) as h:
        for s in range(n_sys):
            h.set_clock(s, 0.0, 1)
        h.stage("pclose")
        for s in range(n_sys):
            a = h.download(s)
            assert np.array_equal(a.closest, want[s % 3].closest)
            assert np.array_equal(a.closestd, want[s % 3].closestd)


@pytest.mark.parametrize("tree_cap", [130000, 131000])
def test_either_side_of_the_handles_slots(tree_cap):
    from nuvort_b200.api import Handle
    p, q = config0_params(), config1_params("Tree")
    small, large = tangle(200, 0.002, n_points=500), tangle(201, 0.001, n_points=900)
    o = Oracle(p, small, t=0.0, itime=1)
    o.stage("pclose")
    with Handle([q, p], [tree_cap, 560], states=[large, small]) as h:
        h.set_clock(1, 0.0, 1)
        h.stage("construct_tree")
        h.stage("pclose")
        a, b = h.download(1), o.download()
        assert np.array_equal(a.closest, b.closest) and np.array_equal(a.closestd, b.closestd)

