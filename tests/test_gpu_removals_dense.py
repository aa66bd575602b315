"""Removals by the rounds that apply events alone in their neighbourhood together and by those that
take them one after the other, in one sweep: lines along which stretches lose many points and
others few, so that the sweep goes from one kind of round to the other and back.  Equal to the
oracle's, event for event; and a line that loses most of its points is not long work."""
import time

import numpy as np
import pytest

from helpers import config0_params, tangle
from nuvort_b200.abi import event_digest
from nuvort_b200.rings import single_ring
from test_gpu_topology import _assert_same, _moved_state, _run_stage
from test_gpu_topology_passes import _shuffled

pytestmark = pytest.mark.gpu


def _stretches(n, rng, jitter):
    """A ring whose points are jittered along it by stretches of some thousand slots."""
    st = single_ring(0.03, n)
    gap = float(np.linalg.norm(st.x[0] - st.x[1]))
    where = np.repeat(rng.choice(jitter, n // 1500 + 1), 1500)[:n]
    d = st.x[st.infront - 1] - st.x
    st.x += d * (where * rng.standard_normal(n))[:, None]
    return st, gap


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("scale", [1.0, 1.6, 1.9])
@pytest.mark.parametrize("margins", [False, True])
def test_dense_and_sparse_stretches(scale, shuffle, margins):
    from nuvort_b200.api import Handle
    from oracle import Oracle
    st, gap = _stretches(12000, np.random.default_rng(int(scale * 10)), (0.02, 0.15, 0.4, 1.0))
    if shuffle:
        st = _shuffled(st, 5)
    p = config0_params(delta=gap * scale / 0.99, overide_timestep_check=True)
    o = Oracle(p, st, t=0.0, itime=1)
    o.set_event_margins(margins)
    o.stage("premove")
    with Handle(p, [st.pcount + 8], states=[st]) as h:
        h.set_event_margins(margins)
        h.set_clock(0, 0.0, 1)
        h.stage("premove")
        assert len(o.events()) > 1000
        assert h.events() == o.events()
        _assert_same(h.download(), o.download())
        assert h.counters().event_hash == event_digest(o.events())
        if margins:
            assert 0.0 <= h.event_margins()["remove"] <= o.event_margins()["remove"]


@pytest.mark.parametrize("share", [0.1, 0.2, 0.5, 0.95])
def test_crowded_lines(share):
    st = _moved_state(config0_params(), tangle(33, 0.002, n_rings=60))
    st.x[:st.pcount] += np.random.default_rng(1).normal(0.0, 4e-4, (st.pcount, 3))
    ahead = st.infront[st.infront - 1] - 1
    two = np.linalg.norm(st.x - st.x[ahead], axis=1)
    p = config0_params(delta=float(np.quantile(two, share)) / 0.99, overide_timestep_check=True)
    a, b, ea, eb, ca, cb = _run_stage(p, st, ["premove"])
    assert ea == eb
    _assert_same(a, b)
    assert (ca.remove_count, ca.loop_kills, ca.event_hash) == (cb.remove_count, cb.loop_kills, event_digest(eb))


def test_a_line_that_loses_most_of_its_points():
    # in slot order: no event is alone.  32,768 points, 95 % pass: 38 ms, 17 times as long as where 5 %
    # pass and most events are alone (68 ms, 31 times, when every round looked for such events with
    # the neighbourhoods in its map)
    from nuvort_b200.api import Handle
    st = tangle(3, 0.001, n_points=32768)
    st.x = st.x + np.random.default_rng(1).normal(0.0, 1.5e-4, st.x.shape)
    ahead = st.infront[st.infront - 1] - 1
    two = np.linalg.norm(st.x - st.x[ahead], axis=1)
    took = []
    for share in (0.05, 0.95):
        p = config0_params(delta=float(np.quantile(two, share)) / 0.99, overide_timestep_check=True)
        with Handle(p, [st.pcount + 8], states=[st]) as h:
            best = 1e9
            for _ in range(4):
                h.upload(0, st)
                h.set_clock(0, 0.0, 1)
                h.counters()
                t = time.perf_counter()
                h.stage("premove")
                best = min(best, time.perf_counter() - t)
            took.append(best)
            removed = h.counters().remove_count
    assert removed > 12000
    assert took[1] < 24 * took[0]
