"""The plain path's segment terms take their square roots and quotients from shared seeds
(nuvort_b200/csrc/fp64.cuh), each rounded as the IEEE operation rounds it: on straight lines
along z, whose local term is exactly zero (x'' is zero, so log() does not enter), the velocities
equal the oracle's bit for bit."""
import numpy as np
import pytest

from helpers import config0_params
from nuvort_b200.abi import State
from oracle import Oracle

pytestmark = pytest.mark.gpu

L = 3.0 / 32.0


def _lines(n, seed):
    """n slots: periodic straight lines along z through random (x, y), the points of a line
    2^-6 .. 2^-10 apart (powers of two, so that x'' is zero without a rounding), the slots
    that no line fills left empty."""
    rng = np.random.Generator(np.random.PCG64(seed))
    x = np.zeros((n, 3))
    nxt, prv = np.zeros(n, np.int32), np.zeros(n, np.int32)
    base = int(rng.integers(0, 2))
    while n - base >= 6:
        m = int(rng.choice([v for v in (6, 12, 24, 48, 96) if v <= n - base]))
        k = np.arange(m)
        x[base:base + m, :2] = rng.uniform(-0.5, 0.5, 2) * L
        x[base:base + m, 2] = -L / 2 + (k + 0.5) * (L / m)
        nxt[base:base + m] = base + 1 + (k + 1) % m
        prv[base:base + m] = base + 1 + (k - 1) % m
        base += m
    z3 = lambda: np.zeros((n, 3))
    return State(x=x, infront=nxt, behind=prv, u=z3(), u1=z3(), u2=z3(), ghosti=z3(), ghostb=z3(),
                 closest=np.zeros(n, np.int32), closestd=np.zeros(n))


def _params(scale=1.0):
    return config0_params(box_size=L * scale, delta=0.02 * max(scale, 1.0))


# one tile and less, tile edges (128 or 256 segments), several tiles with a remainder
@pytest.mark.parametrize("n", [7, 127, 128, 129, 257, 650])
@pytest.mark.parametrize("split", [1, 2, 4, 8, 64])
def test_direct_sum_bit_identical_to_the_reference_order(n, split):
    from nuvort_b200.api import Handle
    st = _lines(n, n)
    p = _params()
    uo = Oracle(p, st).calc_velocity()
    with Handle(p, [n + 3], states=[st]) as h:
        h.set_direct_split(split)
        assert np.array_equal(h.calc_velocity(), uo)


@pytest.mark.parametrize("scale", [2.0**-232, 2.0**-66, 2.0**199])
def test_terms_outside_the_shared_seeds_range(scale):
    # box and positions scaled until 4ac - b^2 leaves the range the seeds serve (its fourth
    # power of the scale): such terms take the IEEE operations, with the same bits
    from nuvort_b200.api import Handle
    st = _lines(90, 5)
    st.x *= scale
    p = _params(scale)
    uo = Oracle(p, st).calc_velocity()
    for split in (2, 8, 64):
        with Handle(p, [96], states=[st]) as h:
            h.set_direct_split(split)
            assert np.array_equal(h.calc_velocity(), uo, equal_nan=True)


# one leaf level and less, several levels, rings across the box; the tree's own accepted nodes,
# single points among them, with the opening test by squares and by quotients (theta > 2/sqrt(3))
@pytest.mark.parametrize("n", [7, 129, 650])
@pytest.mark.parametrize("theta", [0.4, 0.9, 1.3])
@pytest.mark.parametrize("corr", [True, False])
def test_tree_walk_bit_identical_to_the_reference_order(n, theta, corr):
    from nuvort_b200.api import Handle
    st = _lines(n, n)
    p = config0_params(box_size=L, delta=0.02, velocity="Tree", tree_theta=theta, tree_extra_correction=corr)
    o = Oracle(p, st)
    uo = o.calc_velocity()
    with Handle(p, [n + 3], states=[st]) as h:
        for parts in (1, 2):
            h.set_walk_parts(parts)
            assert np.array_equal(h.calc_velocity(), uo)
            c = h.counters()
            assert (c.tree_eval, c.tree_tests) == (o.counters().tree_eval, o.counters().tree_tests)
