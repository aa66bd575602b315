"""pinsert where many new points insert again: live and free slots in turn, so that the sweep reaches
most new points, and segments of many delta, so that the points inserted there insert in turn.
While the iteration's set of such positions is not yet right, several chains of insertions run
through the same slots (1,497 visits of 499 slots for 500 segments of 9 delta).  Events, links
and positions equal to the oracle's, with as many slots as the insertions need and with more, one
system and several side by side, whose sets lie next to one another."""
import numpy as np
import pytest

from helpers import config0_params
from nuvort_b200.abi import State
from nuvort_b200.rings import single_ring
from oracle import Oracle
from test_gpu_topology import _assert_same

pytestmark = pytest.mark.gpu


def _alternate(live, times):
    """A ring of `live` points in every other slot, and the delta its segments are `times` of."""
    r = single_ring(0.03, live)
    n = 2 * live
    f = lambda: np.zeros((n, 3))
    i = lambda: np.zeros(n, np.int32)
    st = State(x=f(), infront=i(), behind=i(), u=f(), u1=f(), u2=f(), ghosti=f(), ghostb=f(), closest=i(),
               closestd=np.zeros(n))
    st.x[::2] = r.x
    st.u[::2] = np.random.default_rng(live).standard_normal((live, 3))
    st.infront[::2], st.behind[::2] = 2 * r.infront - 1, 2 * r.behind - 1
    st.ghosti[::2], st.ghostb[::2] = r.x[r.infront - 1], r.x[r.behind - 1]
    return st, float(np.linalg.norm(r.x[0] - r.x[1])) / times


@pytest.mark.parametrize("iters", [1, 6, 40])
@pytest.mark.parametrize("room", [0, 1500])
@pytest.mark.parametrize("live,times", [((500,), 9), ((500,), 33), ((500, 97, 301), 33), ((16, 500, 31), 9)])
def test_new_points_that_insert_again(live, times, room, iters):
    from nuvort_b200.api import Handle
    states, params, want = [], [], []
    for m in live:
        st, delta = _alternate(m, times)
        p = config0_params(delta=delta, overide_timestep_check=True)
        o = Oracle(p, st, t=0.0, itime=1)
        o.stage("pinsert")
        assert len(o.events()) > 1.5 * m
        states.append(st)
        params.append(p)
        want.append(o)
    caps = [o.counters().pcount + room for o in want]
    with Handle(params, caps, states=states) as h:
        h.set_insert_iterations(iters)
        for s in range(len(live)):
            h.set_clock(s, 0.0, 1)
        h.stage("pinsert")
        serial = 0
        for s, o in enumerate(want):
            a, b = h.download(s), o.download()
            assert h.events(s) == o.events()
            _assert_same(a, b)
            assert h.counters(s).pcount == o.counters().pcount
            serial += h.diagnostics(s)[2]
        if iters == 40 and room:  # the iteration comes to rest
            assert serial == 0


def test_more_of_them_than_a_few_thousand():
    # 12,000 segments of 5 delta: some 10,000 new points insert again, found by the iteration as well
    from nuvort_b200.api import Handle
    st, delta = _alternate(12000, 5)
    p = config0_params(delta=delta, overide_timestep_check=True)
    o = Oracle(p, st, t=0.0, itime=1)
    o.stage("pinsert")
    for extra in (0, 250000):  # rounds by a block, rounds over the whole GPU
        with Handle(p, [o.counters().pcount + 12000 + extra], states=[st]) as h:
            h.set_insert_iterations(40)
            h.set_clock(0, 0.0, 1)
            h.stage("pinsert")
            assert h.events() == o.events()
            _assert_same(h.download(), o.download())
            diag = h.diagnostics(0)
            assert diag[2] == 0 and diag[5] > 8000
