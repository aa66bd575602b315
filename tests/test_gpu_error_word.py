"""A system whose state is an error beside others that are not: blocks of one launch set the error
word while others of the launch start.  The call raises that error, every time, and the handle
then takes good states and gives what a new handle gives."""
import numpy as np
import pytest

from helpers import config0_params, config1_params, tangle

pytestmark = pytest.mark.gpu

REPEATS = 6  # the blocks meet the error word at other places each time


@pytest.mark.parametrize("precision,parts", [("fp64", 1), ("fp64", 2), ("mixed", 1), ("mixed", 2), ("mixed", 4),
                                             ("mixed", 8)])
def test_singular_pair_in_one_system(precision, parts):
    # two points 2e-17 apart on either side of a root cell's middle: 26,000 targets in 13 systems,
    # several times what is resident at once
    from nuvort_b200.api import Handle, NuvortError
    p = config1_params("Tree", precision=precision)
    good = [tangle(80 + i, 0.001, n_points=2000) for i in range(13)]
    bad = good[5].copy()
    far = int(np.argmax(np.linalg.norm(bad.x - bad.x[0], axis=1)))
    bad.x[far] = bad.x[0]
    bad.x[0, 0], bad.x[far, 0] = 1e-17, -1e-17
    caps = [st.pcount + 40 for st in good]
    with Handle([p] * len(good), caps, states=good) as h:
        h.set_walk_parts(parts)
        want = [h.calc_velocity(s) for s in range(len(good))]
        for _ in range(REPEATS):
            h.upload(5, bad)
            with pytest.raises(NuvortError, match="singularity"):
                h.calc_velocity(0)
            h.upload(5, good[5])
            for s in (0, 5, 12):
                assert np.array_equal(h.calc_velocity(s), want[s])


@pytest.mark.parametrize("what", ["capacity", "empty"])
def test_walled_system_that_cannot_insert(what):
    # 40 walled systems, each with hundreds of insertions; one has no room for its own, or no line
    from nuvort_b200.api import Handle, NuvortError
    from nuvort_b200.rings import half_loop
    p = config0_params(dt=2e-7, delta=0.0003, boundary_x="solid", boundary_y="periodic", boundary_z="periodic")
    good = [half_loop(250 + 3 * i, 0.0005) for i in range(40)]
    good[7] = half_loop(200, 0.0003)  # inserts nothing
    caps = [1200] * 40
    caps[7] = 300
    bad = half_loop(271, 0.0005)
    if what == "empty":
        bad.infront[:] = bad.behind[:] = bad.pinnedi[:] = bad.pinnedb[:] = 0
    with Handle([p] * 40, caps, states=good) as h:
        h.step(2)
        want = [h.download(s) for s in range(40)]
        for _ in range(REPEATS):
            for s in range(40):
                h.upload(s, bad if s == 7 else good[s])
                h.set_clock(s, 0.0, 0)
            with pytest.raises(NuvortError, match="capacity" if what == "capacity" else "length is 0"):
                h.step(2)
        for s in range(40):
            h.upload(s, good[s])
            h.set_clock(s, 0.0, 0)
        h.step(2)
        for s in range(40):
            a = h.download(s)
            assert np.array_equal(a.x, want[s].x) and np.array_equal(a.infront, want[s].infront)
