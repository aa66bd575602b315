"""The mixed tree walk's work lists: groups of 32 targets shared by 1, 2, 4 or 8 warps, small and
ragged systems, systems side by side, rings across the periodic faces (a target's own segments
then lie a box length away), a second opening criterion (theta above 2/sqrt(3)) and guards that
send every term to FP64.  Accepted nodes and opening tests are the plain walk's, number for
number; velocities within the mixed path's 1e-6 of the plain path's."""
import numpy as np
import pytest

from helpers import config0_params, rms_rel, tangle

pytestmark = pytest.mark.gpu

TOL = 1e-6  # the mixed path's stated bound (relative RMS)


def _run(states, caps, parts=0, guards=None, **kw):
    from nuvort_b200.api import Handle
    p = config0_params(velocity="Tree", dt=1e-6, **kw)
    with Handle([p] * len(states), caps, states=states) as h:
        h.set_walk_parts(parts)
        if guards:
            h.set_fp32_guards(*guards)
        out = []
        for s in range(len(states)):
            u = h.calc_velocity(s)
            c = h.counters(s)
            out.append((u, c.tree_eval, c.tree_tests))
    return out


def _compare(plain, mixed, tol=TOL):
    for (u, e, t), (v, f, r) in zip(plain, mixed):
        assert (f, r) == (e, t)
        assert rms_rel(v, u) <= tol


@pytest.mark.parametrize("parts", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [64, 65, 97, 1500])
def test_sizes(n, parts):
    st = tangle(3, 0.002, n_points=n)
    kw = dict(tree_theta=0.4)
    _compare(_run([st], [n + 7], **kw), _run([st], [n + 7], parts, precision="mixed", **kw))


@pytest.mark.parametrize("theta", [0.05, 0.8, 1.3])
def test_opening_angles(theta):
    st = tangle(8, 0.002, n_points=700)
    kw = dict(tree_theta=theta)
    _compare(_run([st], [900], **kw), _run([st], [900], precision="mixed", **kw))


def test_systems_side_by_side():
    states = [tangle(s, 0.002, n_points=n) for s, n in enumerate((130, 64, 999))]
    caps = [131, 200, 1003]
    kw = dict(tree_theta=0.4)
    _compare(_run(states, caps, **kw), _run(states, caps, precision="mixed", **kw))


def test_every_term_in_fp64():
    # the angle guard at 2 sends every term to the FP64 queue; each agrees with the plain path's
    # to a few roundings, far below the mixed tolerance
    st = tangle(5, 0.002, n_points=400)
    kw = dict(tree_theta=0.4)
    plain = _run([st], [450], **kw)
    for parts in (1, 8):
        _compare(plain, _run([st], [450], parts, guards=(2.0, 1e-3, 1e-2), precision="mixed", **kw), tol=1e-9)
