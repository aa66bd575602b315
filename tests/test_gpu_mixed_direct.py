"""The mixed direct sum at the edges of its tiles (pairs of segments, 32 segments a warp, 256 a
tile, a ring of four buffers), of its blocks of 32 targets, and of neighbouring systems' records
(odd capacities): within the mixed path's 1e-6 of the plain path, which the tests of the plain
path hold to the oracle."""
import numpy as np
import pytest

from helpers import config0_params, rms_rel, tangle

pytestmark = pytest.mark.gpu

TOL = 1e-6  # the mixed path's stated bound (relative RMS)


def _both(states, caps):
    from nuvort_b200.api import Handle
    out = []
    for precision in ("fp64", "mixed"):
        with Handle([config0_params(precision=precision)] * len(states), caps, states=states) as h:
            out.append([h.calc_velocity(s) for s in range(len(states))])
    return out


@pytest.mark.parametrize("n", [64, 65, 255, 256, 257, 1023, 1025, 1281])
def test_sizes(n):
    st = tangle(n, 0.002, n_points=n)
    (plain,), (mixed,) = _both([st], [n])
    assert rms_rel(mixed, plain) <= TOL


def test_systems_of_odd_capacities_side_by_side():
    # a pair's second half past an odd capacity lies in the next system's first record
    states = [tangle(s, 0.002, n_points=n) for s, n in enumerate((65, 101, 99, 130))]
    plain, mixed = _both(states, [65, 103, 99, 131])
    for u, v in zip(mixed, plain):
        assert rms_rel(u, v) <= TOL


def test_empty_slots_contribute_nothing():
    st = tangle(3, 0.002, n_rings=6)
    ends = [k for k in range(1, st.pcount + 1) if st.infront[k - 1] < k]  # last slot of each ring
    a, b = ends[1], ends[2]
    for f in (st.infront, st.behind, st.x):
        f[a:b] = 0
    (plain,), (mixed,) = _both([st], [st.pcount + 5])
    assert np.all(mixed[a:b] == 0)
    assert rms_rel(mixed, plain) <= TOL
