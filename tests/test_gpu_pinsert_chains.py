"""pinsert where the outcome of one slot's test depends on its predecessor's, that one's on its own,
and so on along thousands of slots: rings of equal segments, every one of which passes delta with
its ghosts of the step's start and not with those of its neighbour's insertion, or the reverse.
Equal to the oracle's sweep, with the slots along the ring in order, against it and shuffled; and
such chains do not make the stage long."""
import time

import numpy as np
import pytest

from helpers import config0_params
from nuvort_b200.rings import single_ring
from oracle import Oracle
from test_gpu_topology import _assert_same
from test_gpu_topology_passes import _shuffled

pytestmark = pytest.mark.gpu


def _ring(n, which, seed=0):
    """(state, params): `which` slots are undecided, stale test passing where +1, fresh where -1."""
    st = single_ring(0.03, n)
    rng = np.random.default_rng(seed)
    gap = float(np.linalg.norm(st.x[0] - st.x[1]))
    sign = {"stale": np.ones(n), "fresh": -np.ones(n), "both": rng.choice([-1.0, 1.0], n),
            "some": rng.choice([-1.0, 0.0, 1.0], n, p=[0.45, 0.1, 0.45])}[which]
    d = st.x[st.infront - 1] - st.x
    if which == "fresh":  # the segment itself exceeds delta, its ghost does not
        delta = gap * (1 - 1e-5)
        scale = 1 - 1e-4 * np.ones(n)
    else:
        delta = gap * (1 + 1e-5)
        scale = 1 + 1e-4 * (sign > 0)
    st.ghosti = st.x + d * scale[:, None]
    st.ghostb = st.x[st.behind - 1].copy()
    if which in ("both", "some"):  # some segments longer than delta, with ghosts that are not
        long = np.nonzero(sign < 0)[0]
        st.x[long] -= d[long] * 3e-5
        st.ghosti[long] = st.x[long] + (st.x[st.infront[long] - 1] - st.x[long]) * (1 - 1e-4)
    return st, config0_params(delta=delta, dt=1e-9, overide_timestep_check=True)


@pytest.mark.parametrize("order", ["along", "against", "shuffled"])
@pytest.mark.parametrize("which", ["stale", "fresh", "both", "some"])
@pytest.mark.parametrize("n", [33, 1023, 4097])
def test_chains_of_undecided_slots(n, which, order):
    from nuvort_b200.api import Handle
    st, p = _ring(n, which, n)
    if order == "against":
        st.infront, st.behind, st.ghosti, st.ghostb = (st.infront[::-1].copy(), st.behind[::-1].copy(),
                                                       st.ghosti[::-1].copy(), st.ghostb[::-1].copy())
        st.x = st.x[::-1].copy()
        st.infront, st.behind = (n + 1 - st.infront).astype(np.int32), (n + 1 - st.behind).astype(np.int32)
    elif order == "shuffled":
        st = _shuffled(st, n)
    o = Oracle(p, st, t=0.0, itime=1)
    o.stage("pinsert")
    with Handle([p, p], [2 * n + 40] * 2, states=[st, st]) as h:
        for _ in range(2):  # a second pass over the same slots
            for s in (0, 1):
                h.upload(s, st)
                h.set_clock(s, 0.0, 1)
            h.stage("pinsert")
        for s in (0, 1):
            assert h.events(s)[-len(o.events()):] == o.events()
            _assert_same(h.download(s), o.download())


def test_long_chains_are_short_work():
    # 131,072 slots, each depending on the one before: 296 ms when every slot walked to the chain's start
    from nuvort_b200.api import Handle
    st, p = _ring(131072, "stale")
    with Handle(p, [210000], states=[st]) as h:
        best = 1e9
        for _ in range(4):
            h.upload(0, st)
            h.counters()
            t = time.perf_counter()
            h.stage("pinsert")
            best = min(best, time.perf_counter() - t)
        assert h.counters().pcount == 131072 + 65536
    assert best < 0.08
