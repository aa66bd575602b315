"""The mixed direct sum where its records end and where its guards act: an odd number of segments,
whose last pair has an empty second half at the origin, with targets near the origin."""
import numpy as np
import pytest

from helpers import config0_params, rms_rel, tangle
from nuvort_b200.abi import NV_PREC_FP64, NV_PREC_MIXED, State
from nuvort_b200.rings import single_ring

pytestmark = pytest.mark.gpu

TOL = 1e-6  # the mixed path's stated bound (relative RMS)


def _velocities(params, states, caps, guards=None):
    from nuvort_b200.api import Handle
    out = []
    for precision in ("fp64", "mixed"):
        ps = []
        for p in params:
            q = type(p).from_buffer_copy(p)
            q.precision = NV_PREC_MIXED if precision == "mixed" else NV_PREC_FP64
            ps.append(q)
        with Handle(ps, caps, states=states) as h:
            if guards and precision == "mixed":
                h.set_fp32_guards(*guards)
            out.append([h.calc_velocity(s) for s in range(len(states))])
    return out


@pytest.mark.parametrize("n", [33, 63, 65, 255, 257, 1281])
@pytest.mark.parametrize("spare", [0, 1])
def test_full_odd_system_around_the_origin(n, spare):
    # the last pair's second half is an empty record at the origin, inside every target's near
    # radius (delta 0.002, ring of radius 0.0015): it is no segment, whatever lies behind the
    # FP64 records -- here, with a second system, the second one's
    near, far = single_ring(0.0015, n), tangle(n, 0.002, n_points=301)
    p = config0_params()
    for states in ([near], [far, near], [near, far]):
        plain, mixed = _velocities([p] * len(states), states, [s.pcount + spare for s in states])
        for u, v in zip(mixed, plain):
            assert np.isfinite(u).all()
            assert rms_rel(u, v) <= TOL


def _needle(m, step, eps, axis):
    """A closed line that runs m steps along an axis and back, 2 eps apart at most."""
    k = np.arange(2 * m)
    along = np.where(k <= m, k, 2 * m - k) * step - 0.5 * m * step
    aside = eps * np.sin(np.pi * k / m)
    e = np.linalg.qr(np.array([axis, [0.3, 1.0, 0.2], [0.1, -0.4, 1.0]]).T)[0]
    z = lambda: np.zeros((2 * m, 3))
    x = np.ascontiguousarray(along[:, None] * e[:, 0] + aside[:, None] * e[:, 1])
    return State(x=x, infront=((k + 1) % (2 * m) + 1).astype(np.int32), behind=((k - 1) % (2 * m) + 1).astype(np.int32),
                 u=z(), u1=z(), u2=z(), ghosti=z(), ghostb=z(), closest=np.zeros(2 * m, np.int32),
                 closestd=np.zeros(2 * m))


@pytest.mark.parametrize("m", [60, 61])
@pytest.mark.parametrize("axis", [[0.3, 0.5, 0.8], [0.9, -0.2, 0.4]])
def test_line_guard_of_distant_segments(m, axis):
    # Every segment beyond the near radius lies within the line guard's angle of every target
    # (|r x d| < sqrt(1e-3) |r||d|), so every term is evaluated in FP64.  Point by point, away from
    # the ends, where the two sides meet: the plain path's own rounding of these terms is 2.2e-12
    # against long double; the far terms in FP32 would be off by 1.4e-10 to 1.3e-9.
    st = _needle(m, 7.5e-4, 2e-5, axis)
    p = config0_params(delta=0.001, boundary_x="open", boundary_y="open", boundary_z="open")
    (plain,), (mixed,) = _velocities([p], [st], [2 * m + 7])
    k = np.arange(2 * m)
    inner = np.abs(np.where(k <= m, k, 2 * m - k) - m / 2) < m / 3
    assert np.max(np.linalg.norm(mixed - plain, axis=1)[inner]) < 1e-11


@pytest.mark.parametrize("n", [65, 700])
@pytest.mark.parametrize("guards", [(0.1, 1.0, 1e-2), (2.0, 1e-3, 1e-2), (0.1, 1e-3, 1.0)])
def test_guards_widened_to_every_term(n, guards):
    # the line guard at 1 or the angle guard at 2 sends (nearly) every term to FP64, the end
    # guard at 1 those with |e| < |r|, about half; the others stay within the mixed path's bound
    st = tangle(n, 0.002, n_points=n)
    (plain,), (mixed,) = _velocities([config0_params()], [st], [n + 2], guards=guards)
    assert rms_rel(mixed, plain) <= (TOL if guards[2] == 1.0 else 1e-9)
