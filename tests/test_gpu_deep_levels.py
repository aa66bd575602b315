"""The octree's levels below cells of about an eighth of delta, in states whose points lie far closer
than their delta: a line drawn at a finer delta than the run's, and clusters of a few, some
hundred and more than 2,048 points (a lane, a warp, a block and its warps for a cluster's
subtree), alone and together, in one system and in several.  Every node equal to the oracle's."""
import numpy as np
import pytest

from helpers import config1_params, tangle
from nuvort_b200.rings import single_ring
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _clusters(sizes, radius, seed):
    """A tangle of 0.001 spacing whose last points stand in clusters around points of it."""
    rng = np.random.default_rng(seed)
    st = tangle(seed, 0.001, n_points=2 * sum(sizes) + 900)
    at = st.pcount
    for k, m in enumerate(sizes):
        st.x[at - m:at] = st.x[17 * k] + rng.uniform(-radius, radius, (m, 3))
        at -= m
    return st


def _compare(params, states, extra=0):
    from nuvort_b200.api import Handle
    with Handle(params, [s.pcount + extra for s in states], states=states) as h:
        h.stage("ghostp")
        h.stage("construct_tree")
        for i, (p, st) in enumerate(zip(params, states)):
            o = Oracle(p, st)
            o.stage("ghostp")
            o.stage("construct_tree")
            a, b = h.tree_dump(i), o.tree_dump()
            assert len(a) == len(b)
            for f in ("pos", "width", "cent", "circ", "pcount", "depth", "leaf", "first_next"):
                assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("n,delta", [(3000, 0.02), (3000, 0.2), (20000, 0.05)])
def test_points_closer_than_delta(n, delta):
    _compare([config1_params("Tree", delta=delta, overide_timestep_check=True)], [tangle(5, 0.001, n_points=n)])


@pytest.mark.parametrize("n", [700, 40000])
def test_one_ring_of_points_far_closer_than_delta(n):
    # cells of an eighth of delta hold some hundred points each
    _compare([config1_params("Tree")], [single_ring(0.03 if n > 1000 else 0.003, n)], extra=3000)


@pytest.mark.parametrize("radius", [1e-6, 1e-8])
@pytest.mark.parametrize("sizes", [(2,) * 40, (16, 17, 3), (400, 2048), (2049,), (5000, 2100, 30, 2)])
def test_clusters(sizes, radius):
    _compare([config1_params("Tree")], [_clusters(sizes, radius, 7)], extra=9000)


def test_several_systems():
    p, q = config1_params("Tree"), config1_params("Tree", delta=0.03, overide_timestep_check=True)
    states = [_clusters((2100, 50), 1e-7, 8), tangle(9, 0.001, n_points=1500), _clusters((9, 40, 300), 1e-5, 10)]
    _compare([p, q, p], states, extra=4000)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [40, 1500, 4200])
def test_out_of_nodes_below_is_an_error(n, precision):
    # pairs 1e-11 apart: below the grid's levels they need more nodes than the slots allow
    from nuvort_b200.api import Handle, NuvortError
    p = config1_params("Tree", precision=precision)
    good = tangle(21, 0.001, n_points=3 * n + 200)
    bad = good.copy()
    m = bad.pcount // 2
    bad.x[m:2 * m] = bad.x[:m] + 1e-11
    with Handle(p, [good.pcount], states=[good]) as h:
        want = h.calc_velocity()
        for _ in range(3):
            h.upload(0, bad)
            with pytest.raises(NuvortError, match="octree node buffer exhausted"):
                h.calc_velocity()
        h.upload(0, good)
        assert np.array_equal(h.calc_velocity(), want)
