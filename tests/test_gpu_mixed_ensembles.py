"""The mixed direct sum of ensembles of small systems, by a warp per 32 targets and image: sizes around
its sub-sums of 32 segments and its tiles of 64, empty systems' slots, odd capacities, systems of
either kind in one handle; within the mixed path's 1e-6 of the plain path, system by system."""
import numpy as np
import pytest

from helpers import config0_params, rms_rel, small_rings, tangle

pytestmark = pytest.mark.gpu

TOL = 1e-6  # the mixed path's stated bound (relative RMS)


def _both(states, caps):
    from nuvort_b200.api import Handle
    out = []
    for precision in ("fp64", "mixed"):
        with Handle([config0_params(precision=precision)] * len(states), caps, states=states) as h:
            out.append([h.calc_velocity(s) for s in range(len(states))])
    return out


@pytest.mark.parametrize("extra", [0, 1, 40])
@pytest.mark.parametrize("sizes", [(6,), (31, 32, 33), (63, 64, 65), (127, 128, 129, 192), (30, 700, 5, 257)])
def test_sizes(sizes, extra):
    states = [small_rings(100 + i, 1, sizes[i % len(sizes)], 0.01) for i in range(150)]
    plain, mixed = _both(states, [s.pcount + extra for s in states])
    for u, v in zip(mixed, plain):
        assert rms_rel(u, v) <= TOL


def test_small_and_large_systems_in_one_handle():
    states = [small_rings(i, 3, 20, 0.006) for i in range(80)] + [tangle(1, 0.002, n_points=1500)]
    states[40].infront[20:40] = states[40].behind[20:40] = 0
    plain, mixed = _both(states, [s.pcount + 2 * (i % 3) for i, s in enumerate(states)])
    for u, v in zip(mixed, plain):
        assert rms_rel(u, v) <= TOL
    assert not mixed[40][20:40].any()


def test_whole_steps_have_the_plain_path_s_events():
    from nuvort_b200.api import Handle
    states = [tangle(i, 0.002, n_points=120) for i in range(60)]
    events = []
    for precision in ("fp64", "mixed"):
        with Handle([config0_params(precision=precision)] * 60, [400] * 60, states=states) as h:
            h.step(12)
            events.append([h.events(s) for s in range(60)])
    assert events[0] == events[1] and any(events[0])
