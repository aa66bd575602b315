"""Edges of the topology stages' kernels and of the tree build: the ordered one-pass lists (blocks
of 1,024 slots, warps of 128) at slot counts around whole blocks, the wall sweeps' chunks of 256
slots, pinsert's rounds over the whole GPU (handles above 262,144 slots) and by a block per
system, with too few rounds allowed, the removal and reconnection sweeps with events few and far
between, in clusters and everywhere, the closest-point search by a warp per target and by the
cell list on either side of the line between them, the octrees of systems of unlike sizes and the
levels of the octree that one block splits, and the rows of a velocity call.  Everything equal to the oracle's, event for event."""
import numpy as np
import pytest

from helpers import config0_params, config1_params, tangle
from nuvort_b200.abi import event_digest
from nuvort_b200.rings import half_loop
from oracle import Oracle
from test_gpu_topology import _assert_same, _moved_state, _ring_slots, _run_stage

pytestmark = pytest.mark.gpu


def _holed(st, rings):
    for r in rings:
        idx = np.asarray(r) - 1
        for name in ("x", "u", "u1", "u2", "ghosti", "ghostb", "infront", "behind"):
            getattr(st, name)[idx] = 0
    return st


@pytest.mark.parametrize("slots", [1021, 1022, 1023, 1024, 1151, 2046, 2048])
def test_lists_around_whole_blocks(slots):
    # the handle's slots are the capacity and a dummy; live points up to the last slot but 40
    from nuvort_b200.api import Handle
    st = tangle(slots, 0.002, n_points=slots - 60)
    p = config0_params()
    o = Oracle(p, st)
    o.step(12)
    with Handle(p, [slots], states=[st]) as h:
        h.step(12)
        assert h.events() == o.events()
        a, b = h.download(), o.download()
        assert np.array_equal(a.infront, b.infront) and np.array_equal(a.closest, b.closest)


@pytest.mark.parametrize("iters", [1, 2, 6])
@pytest.mark.parametrize("extra", [16384, 270000])
def test_pinsert_rounds(iters, extra):
    st = tangle(31, 0.002, n_rings=12)
    mv = _moved_state(config0_params(), _holed(st, _ring_slots(st)[2::3]))
    p_ins = config0_params(delta=0.0009, overide_timestep_check=True)
    diag = []
    a, b, ea, eb, ca, cb = _run_stage(p_ins, mv, ["pinsert"], cap_extra=extra, insert_iterations=iters, diag=diag)
    assert ea == eb and len(eb) > 200
    _assert_same(a, b)
    assert ca.insert_count == cb.insert_count and ca.pcount == cb.pcount
    if iters != 2:  # one round: new points insert again, so the serial sweep takes over
        assert diag[2] == (1 if iters == 1 else 0)


@pytest.mark.parametrize("cap", [6144, 6145])
def test_closest_points_either_side_of_the_line(cap):
    from nuvort_b200.api import Handle
    st = tangle(9, 0.002, n_points=1301)
    st.x[700] = st.x[17]  # two points in one place: ties, lowest slot first
    o = Oracle(config0_params(), st, t=0.0, itime=1)
    o.stage("pclose")
    b = o.download()
    for method in (0, 1):
        with Handle(config0_params(), [cap], states=[st]) as h:
            h.set_pclose_method(method)
            h.set_clock(0, 0.0, 1)
            h.stage("pclose")
            a = h.download()
        assert np.array_equal(a.closest, b.closest) and np.array_equal(a.closestd, b.closestd)


@pytest.mark.parametrize("n", [255, 256, 257, 300])
@pytest.mark.parametrize("delta", [0.0003, 0.0008])
def test_wall_sweeps_around_whole_chunks(n, delta):
    # segments of 0.75 * 0.0005: at delta 0.0003 every one inserts, at 0.0008 points are removed
    from nuvort_b200.api import Handle
    st = half_loop(n, 0.0005)
    p = config0_params(dt=2e-7, delta=delta, boundary_x="solid", boundary_y="periodic", boundary_z="periodic")
    o = Oracle(p, st)
    o.step(4)
    with Handle(p, [1200], states=[st]) as h:
        h.step(4)
        assert len(o.events()) > 50
        assert h.events() == o.events()
        a, b = h.download(), o.download()
        for f in ("infront", "behind", "pinnedi", "pinnedb", "wpinned"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f
        assert np.max(np.abs(a.x - b.x)) < 1e-12


@pytest.mark.parametrize("pairs", [0, 3, 60])
@pytest.mark.parametrize("sizes", [(1021,), (700, 1, 1300, 90), (2046, 1025)])
def test_octrees_and_their_deep_levels(sizes, pairs):
    # pairs of points 1e-10 apart: some 25 levels below the cells of a segment's width
    from nuvort_b200.api import Handle
    p = config1_params("Tree")
    states = []
    for i, n in enumerate(sizes):
        st = tangle(20 + i, 0.001, n_points=max(n - 40, 20))
        m = min(pairs, st.pcount // 3)
        st.x[st.pcount - m:st.pcount] = st.x[:m] + 1e-10
        states.append(st)
    with Handle([p] * len(sizes), [max(n, s.pcount) for n, s in zip(sizes, states)], states=states) as h:
        h.stage("ghostp")
        h.stage("construct_tree")
        for i, st in enumerate(states):
            o = Oracle(p, st)
            o.stage("ghostp")
            o.stage("construct_tree")
            a, b = h.tree_dump(i), o.tree_dump()
            assert len(a) == len(b)
            for f in ("pos", "width", "cent", "circ", "pcount", "depth", "leaf", "first_next"):
                assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_octree_out_of_nodes_is_an_error(precision):
    # 320 pairs 1e-10 apart need some 7,000 nodes below the segments' cells; 981 slots have 4,000
    from nuvort_b200.api import Handle, NuvortError
    p = config1_params("Tree", precision=precision)
    st = tangle(21, 0.001, n_points=940)
    good = st.copy()
    st.x[-320:] = st.x[:320] + 1e-10
    with Handle(p, [980], states=[st]) as h:
        with pytest.raises(NuvortError, match="octree node buffer exhausted"):
            h.calc_velocity()
        h.upload(0, good)
        u = h.calc_velocity()
    with Handle(p, [980], states=[good]) as h:
        assert np.array_equal(u, h.calc_velocity())


def _shuffled(st, seed):
    """The same lines with their points in random slots."""
    to = np.random.default_rng(seed).permutation(st.pcount)
    out = st.copy()
    for name in ("x", "u", "u1", "u2", "ghosti", "ghostb"):
        getattr(out, name)[to] = getattr(st, name)
    for name in ("infront", "behind"):
        link = getattr(st, name)
        getattr(out, name)[to] = np.where(link > 0, to[link - 1] + 1, 0)
    return out


def _crowded(seed, shuffle, n_rings, jitter):
    st = _moved_state(config0_params(), tangle(seed, 0.002, n_rings=n_rings))
    st.x[:st.pcount] += np.random.default_rng(seed).normal(0.0, jitter, (st.pcount, 3))
    return _shuffled(st, seed) if shuffle else st


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("share", [0.003, 0.05, 0.3, 0.8])
def test_removals_apart_and_in_clusters(share, shuffle):
    st = _crowded(31, shuffle, 40, 4e-4)
    live = st.infront[:st.pcount] > 0
    ahead = st.infront[np.maximum(st.infront[:st.pcount], 1) - 1] - 1
    gap = np.linalg.norm(st.x[:st.pcount] - st.x[ahead], axis=1)[live]
    p = config0_params(delta=float(np.quantile(gap, share)) / 0.99, overide_timestep_check=True)
    a, b, ea, eb, ca, cb = _run_stage(p, st, ["premove"])
    assert len(eb) > 5
    assert ea == eb
    _assert_same(a, b)
    assert (ca.remove_count, ca.loop_kills, ca.event_hash) == (cb.remove_count, cb.loop_kills, event_digest(eb))


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("n_rings,delta", [(12, 0.002), (60, 0.002), (60, 0.006), (150, 0.01)])
def test_reconnections_apart_and_in_clusters(n_rings, delta, shuffle):
    st = _crowded(32, shuffle, n_rings, 2e-4)
    p = config0_params(delta=delta, overide_timestep_check=True)
    a, b, ea, eb, ca, cb = _run_stage(p, st, ["pclose", "precon", "premove"])
    assert len(eb) > 0
    assert ea == eb
    _assert_same(a, b)
    assert (ca.recon_count, ca.loop_kills, ca.event_hash) == (cb.recon_count, cb.loop_kills, event_digest(eb))


@pytest.mark.parametrize("velocity,precision", [("BS", "fp64"), ("Tree", "fp64"), ("Tree", "mixed")])
@pytest.mark.parametrize("extra", [0, 1, 300])
def test_velocity_rows(velocity, precision, extra):
    # as many rows as points, those of empty slots zero, the others the handle's u
    from nuvort_b200.api import Handle
    p = config1_params(velocity, precision=precision)
    states = [tangle(60 + i, 0.001, n_points=n) for i, n in enumerate((700, 255, 1024))]
    _holed(states[1], _ring_slots(states[1])[:1])
    with Handle([p] * 3, [s.pcount + extra for s in states], states=states) as h:
        for i, st in enumerate(states):
            u = h.calc_velocity(i)
            live = st.infront[:st.pcount] > 0
            assert u.shape == (st.pcount, 3) and u.flags.c_contiguous and u.flags.owndata
            assert np.array_equal(u[live], h.download(i).u[:st.pcount][live])
            assert not u[~live].any() and u[live].any(axis=1).all()
