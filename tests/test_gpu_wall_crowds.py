"""The wall sweeps where events crowd (thread 0 goes on alone) and where they do not, in one sweep: lines
between walls with stretches of rough and smooth points, a part of the slots empty; loops of few
points, which are cleared, and of many next to lines that end in a wall.  Events, links, pinned
records and the margins of every test equal to the oracle's."""
import numpy as np
import pytest

from helpers import config0_params, small_rings
from nuvort_b200.rings import half_loop, lattice
from oracle import Oracle

pytestmark = pytest.mark.gpu

Z = dict(boundary_x="periodic", boundary_y="periodic", boundary_z="solid", overide_timestep_check=True)


def _rough(st, delta, seed):
    rng = np.random.default_rng(seed)
    rough = np.repeat(rng.choice([0.0, 0.05, 0.5], st.pcount // 40 + 1), 40)[:st.pcount]
    free = (st.pinnedi == 0) & (st.pinnedb == 0)
    st.x[free, 2] += (rough * delta * rng.standard_normal(st.pcount))[free]
    st.x[free, :2] += (0.3 * rough * delta)[free, None] * rng.standard_normal((int(free.sum()), 2))
    return st


@pytest.mark.parametrize("stage", ["pinsert", "premove", "precon", "wall_recon"])
@pytest.mark.parametrize("factor", [0.7, 0.9, 1.4, 1.9])
@pytest.mark.parametrize("lines", [2, 3])
def test_crowded_and_quiet_stretches(lines, factor, stage):
    from nuvort_b200.api import Handle
    delta = 0.0012
    st = _rough(lattice(lines, delta), delta, 3 * lines)
    p = config0_params(delta=delta * factor, **Z)
    o = Oracle(p, st, t=0.0, itime=1)
    o.set_event_margins(True)
    with Handle(p, [3 * st.pcount], states=[st]) as h:
        h.set_event_margins(True)
        h.set_clock(0, 0.0, 1)
        for s in ("ghostp", "pclose", stage, "ghostp", stage):  # twice: the second meets empty slots
            h.stage(s)
            o.stage(s)
        assert h.events() == o.events()
        a, b = h.download(), o.download()
        for f in ("x", "infront", "behind", "pinnedi", "pinnedb", "wpinned"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f
        assert h.event_margins() == o.event_margins()


@pytest.mark.parametrize("points", [3, 4, 5, 9])
def test_loops_of_few_points_between_walls(points):
    from nuvort_b200.api import Handle
    st = small_rings(1, 40, points, 0.0004, spread=0.03)
    for n, name in ((1, "pinnedi"), (1, "pinnedb"), (3, "wpinned")):
        setattr(st, name, np.zeros((st.pcount, 3) if n == 3 else st.pcount, np.int32))
    p = config0_params(delta=0.001, **Z)
    o = Oracle(p, st, t=0.0, itime=1)
    with Handle(p, [st.pcount + 64], states=[st]) as h:
        h.set_clock(0, 0.0, 1)
        for s in ("ghostp", "pclose", "precon", "premove"):
            h.stage(s)
            o.stage(s)
        assert len(o.events()) > 20
        assert h.events() == o.events()
        assert np.array_equal(h.download().infront, o.download().infront)
        assert h.counters().loop_kills == o.counters().loop_kills


def test_out_of_slots_in_a_crowd():
    from nuvort_b200.api import Handle, NuvortError
    st = half_loop(270, 0.0005)
    p = config0_params(delta=0.0003, boundary_x="solid", boundary_y="periodic", boundary_z="periodic",
                       overide_timestep_check=True)
    with Handle(p, [300], states=[st]) as h:
        h.set_clock(0, 0.0, 1)
        with pytest.raises(NuvortError, match="capacity"):
            h.stage("pinsert")
