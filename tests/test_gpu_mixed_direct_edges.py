"""The mixed direct sum where its records end and where its guards act: an odd number of segments,
whose last pair has an empty second half at the origin, with targets near the origin."""
import numpy as np
import pytest

from helpers import config0_params, rms_rel, tangle
from nuvort_b200.abi import NV_PREC_FP64, NV_PREC_MIXED
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
