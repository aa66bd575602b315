"""The work that users of this framework have it do, as timed cases.

Two kinds of call make up a vortex-filament run, and both go through the public API
(nuvort_b200.api.Handle, BatchBuffers):

* ``step``: a host program hands over a filament state (packed page-locked arrays, one copy
  per array), has it advanced by some whole time steps (ghosts, tree build, velocity, AB3,
  insertion, closest points, reconnection, removal, wrap), and takes the state back: the loop
  of a drop-in run, of a parameter sweep, and of a run that writes a snapshot every few steps.
* ``velocity``: the velocity of every point of a state that is on the device, read back: the
  call behind spectra, velocity statistics and comparisons of the two precisions.

The plain FP64 path returns its velocities in FP64.  The mixed path promises them to 1e-6
relative (FP32 far field), so a program that keeps them keeps them as float32; positions are
FP64 in both.

Sizes follow the repository's workloads: rings of 0.015 to 0.03 cm radius in a periodic cube
of 0.1 cm, delta = 0.002 cm for small tangles and ensembles, 0.001 cm for tens of thousands
of points, 0.0005 cm for hundreds of thousands and more.  A step case's state is a seeded
ring tangle after a few plain FP64 steps: the first steps of random overlapping rings
reconnect far more than the steps of a run.
"""
import math

import numpy as np
import torch

from nuvort_b200 import api
from nuvort_b200.abi import State, make_params
from nuvort_b200.rings import lattice, random_rings

BOX = 0.1
COREA = 1.3e-8
KAPPA = 9.97e-4
FRICTION = (0.1, 0.01)


def listed():
    return [
        # the smallest runs: a handful of rings, direct sum, an output every 10 steps; the
        # drop-in's plain arithmetic and the mixed path
        _step("rings_steps_fp64", "BS", "fp64", 600, steps=10),
        _step("rings_steps_mixed", "BS", "mixed", 1501, steps=10),
        # one developed tangle, tree velocity, mutual friction with a normal flow
        _step("tangle32k_steps_fp64", "Tree", "fp64", 32768, steps=2),
        _step("tangle32k_steps_mixed", "Tree", "mixed", 32768, steps=4),
        # the largest single tangle
        _step("tangle1m_step_mixed", "Tree", "mixed", 1048576, steps=1),
        # a parameter sweep: many independent systems advanced by the same launches
        _step("ensemble_steps_mixed", "Tree", "mixed", 12000, steps=2, systems=48, nmin=500),
        # filaments between two solid walls: pinned ends, mirror sums, serial wall topology
        _step("walls_steps_fp64", "BS", "fp64", 1273, steps=4, lines=3),
        # velocity of every point by the direct sum (no tree error), both precisions
        _velocity("direct_velocity_fp64", "BS", "fp64", 12289),
        _velocity("direct_velocity_mixed", "BS", "mixed", 30011),
        # velocity of every point by the tree, both precisions
        _velocity("tree_velocity_fp64", "Tree", "fp64", 100003),
        _velocity("tree_velocity_mixed", "Tree", "mixed", 262144),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    precision = rng.choice(("fp64", "mixed"))
    kind = rng.choice(("rings", "tangle", "tangle", "ensemble", "direct", "tree"))
    if kind == "rings":
        c = _step("", "BS", precision, size(300, 4000), steps=rng.randint(1, 12))
    elif kind == "tangle":
        c = _step("", "Tree", precision, size(6000, 300000), steps=rng.randint(1, 4))
    elif kind == "ensemble":
        c = _step("", "Tree", "mixed", size(3000, 16000), steps=rng.randint(1, 3), systems=rng.randint(8, 64), nmin=500)
    elif kind == "direct":
        c = _velocity("", "BS", precision, size(1000, 12000 if precision == "fp64" else 32000))
    else:
        c = _velocity("", "Tree", precision, size(6000, 150000 if precision == "fp64" else 400000))
    del c["name"]
    return c


def _step(name, velocity, precision, n, steps, systems=1, nmin=0, lines=0):
    """n: points of the system; of an ensemble the most points of one, sizes log-uniform from
    nmin to n.  lines: line_count of a lattice between solid z walls (0: periodic box)."""
    return {"name": name, "kind": "step", "velocity": velocity, "precision": precision, "points": n, "steps": steps,
            "systems": systems, "nmin": nmin, "lines": lines}


def _velocity(name, velocity, precision, n):
    return {"name": name, "kind": "velocity", "velocity": velocity, "precision": precision, "points": n}


# ---- what a program has in hand --------------------------------------------------------------
def _scales(case):
    """(delta, dt, tree_theta) of a system of the case's size."""
    if case["points"] < 20000:
        return 0.002, 2e-5, 0.4
    if case["points"] < 200000:
        return 0.001, 5e-6, 0.4
    return 0.0005, 1e-6, 0.5


def _counts(case):
    """Points of each system: of an ensemble, spread over the range's logarithm."""
    m = case.get("systems", 1)
    if m == 1:
        return [case["points"]]
    lo, hi = math.log(case["nmin"]), math.log(case["points"])
    return [int(round(math.exp(lo + (hi - lo) * (k + 0.5) / m))) for k in range(m)]


def _flow(seed, s):
    """Uniform normal flow of system s (cm/s)."""
    rng = np.random.Generator(np.random.PCG64([seed, 2, s]))
    a = rng.standard_normal(3)
    return tuple(float(v) for v in a / np.linalg.norm(a) * rng.uniform(0.2, 1.0))


def _params(case, precision, seed, s):
    delta, dt, theta = _scales(case)
    kw = dict(dt=dt, delta=delta, box_size=BOX, corea=COREA, quant_circ=KAPPA, velocity=case["velocity"],
              tree_theta=theta if case["velocity"] == "Tree" else 0.0, precision=precision, alpha=FRICTION,
              normal_velocity="uniform", norm_vel_vec=_flow(seed, s))
    if case.get("lines"):
        kw["boundary_z"] = "solid"
    return make_params(**kw)


def _tangle(n, delta, seed, s=0):
    sub = int(np.random.Generator(np.random.PCG64([seed, 3, s])).integers(0, 2**31 - 1))
    return random_rings(sub, delta, (BOX, BOX, BOX), n_points=n)


def _walls(case, delta, seed):
    """A lattice of lines between the z walls, each bent by a few long waves."""
    st = lattice(case["lines"], delta, (BOX, BOX, BOX))
    rng = np.random.Generator(np.random.PCG64([seed, 4]))
    z = st.x[:, 2] / BOX + 0.5
    for k in (1, 2, 3):
        phase = rng.uniform(0, 2 * np.pi, 2)
        amp = rng.uniform(0.3, 1.0, 2) * 0.0015 / k
        for c in (0, 1):
            st.x[:, c] += amp[c] * np.sin(np.pi * k * z) * np.cos(phase[c] + 40.0 * st.x[:, 1 - c])
    return st


class _State:
    """A case's handle and host arrays, given back when the program drops them."""

    def __init__(self, case):
        self.case, self.h, self.buffers, self.start, self.out = case, None, [], None, None

    def __del__(self):
        for b in self.buffers:
            b.close()
        if self.h is not None:
            self.h.close()


def prepare(case, seed):
    s = _State(dict(case))
    delta = _scales(case)[0]
    counts = _counts(case)
    if case["kind"] == "velocity":
        st = _tangle(case["points"], delta, seed)
        s.h = api.Handle(_params(case, case["precision"], seed, 0), [st.pcount + 256], states=[st])
        return s
    if case["lines"]:
        s.start = _walls(case, delta, seed)
        s.h = api.Handle(_params(case, "fp64", seed, 0), [2 * s.start.pcount], states=[s.start])
        s.out = State.empty(s.h.capacity[0])
        return s
    states = [_tangle(n, delta, seed, k) for k, n in enumerate(counts)]
    caps = [int(1.6 * st.pcount) + 256 for st in states]
    with api.Handle([_params(case, "fp64", seed, k) for k in range(len(states))], caps, states=states) as h:
        h.step(3)
        states = h.download_many()
    s.h = api.Handle([_params(case, case["precision"], seed, k) for k in range(len(states))], caps)
    s.h.upload_many(states)
    start = api.BatchBuffers(s.h)
    start.download()
    s.buffers = [start, api.BatchBuffers(s.h, fields=("x", "u", "infront", "behind"))]
    if case["precision"] == "mixed":
        s.out = np.zeros(s.buffers[1].arrays["u"].shape, np.float32)
    return s


# ---- one pass --------------------------------------------------------------------------------
def run(s):
    case = s.case
    mixed = case["precision"] == "mixed"
    if case["kind"] == "velocity":
        return {"u": s.h.calc_velocity().astype(np.float32 if mixed else np.float64, copy=False)}
    if case["lines"]:
        s.h.upload(0, s.start)
        s.h.step(case["steps"])
        fields = ("x", "u", "infront", "behind", "pinnedi", "pinnedb")
        s.h.download(0, out=s.out, fields=fields)
        return {f: getattr(s.out, f) for f in fields}
    start, out = s.buffers
    start.upload()
    s.h.step(case["steps"])
    out.download()
    a = dict(out.arrays)  # rows of all systems, packed; the arrays have room for more
    if mixed:
        n = out.rec.pcount
        s.out[:n] = a["u"][:n]
        a["u"] = s.out
    a["points"] = np.array(out.pcounts())
    return a


# ---- what a pass cannot do without -------------------------------------------------------------
PAIR_FLOPS, TEST_FLOPS = 43, 12  # per segment term, per opening test (adds, multiplies, 2 sqrt, 3 div)


def _interactions(case, n):
    """(segment terms, opening tests) of one velocity pass over n points with 27 images."""
    if case["velocity"] == "BS":
        images = 27 if not case.get("lines") else 9 + 2
        return images * n * n, 0
    theta = _scales(case)[2]
    # accepted nodes per target of ring tangles: a fit of the counts at 8K to 1M points
    per = 85.0 * (0.5 / theta) ** 1.67 * math.log2(n)
    return per * n, 1.19 * per * n


def work(case):
    if case["kind"] == "velocity":
        n = case["points"]
        t, o = _interactions(case, n)
        return {"bytes": n * (24 + 8 + 24), "flops": t * PAIR_FLOPS + o * TEST_FLOPS}
    counts = _counts(case)
    flops = bytes_ = 0.0
    for n in counts:
        t, o = _interactions(case, n)
        flops += case["steps"] * (t * PAIR_FLOPS + o * TEST_FLOPS)
        # state in and out; per step the streaming stages (AB3, ghosts, local term + friction)
        bytes_ += n * (104 + 56 + case["steps"] * (168 + 128 + 96))
    return {"bytes": bytes_, "flops": flops}


# ---- the same velocities in plain 64-bit torch -------------------------------------------------
def exact(case, seed):
    """Velocities from the definition: local term, sum over segments (or accepted tree nodes)
    of the 27 images, mutual friction.  A whole step ends in serial topology events: None."""
    if case["kind"] != "velocity":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    delta, _, theta = _scales(case)
    st = _tangle(case["points"], delta, seed)
    x = torch.tensor(st.x, device=dev)
    nxt = torch.tensor(st.infront.astype(np.int64) - 1, device=dev)
    prv = torch.tensor(st.behind.astype(np.int64) - 1, device=dev)
    gi, gb = _unwrap(x, x[nxt]), _unwrap(x, x[prv])
    u, tangent = _local(x, gi, gb)
    if case["velocity"] == "BS":
        u = u + _direct(x, gi - x, prv)
    else:
        u = u + _tree(x, gi - x, prv, theta)
    vn = torch.tensor(_flow(seed, 0), device=dev, dtype=torch.float64)
    c1 = torch.linalg.cross(tangent, vn - u)
    u = u + FRICTION[0] * c1 - FRICTION[1] * torch.linalg.cross(tangent, c1)
    return {"u": u.cpu().numpy()}


def _unwrap(x, g):
    d = x - g
    return g + BOX * ((d > BOX / 2).double() - (d < -BOX / 2).double())


def _local(x, gi, gb):
    li, lb = (gi - x).norm(dim=1, keepdim=True), (gb - x).norm(dim=1, keepdim=True)
    d1 = (lb * gi + (li - lb) * x - li * gb) / (2 * li * lb)
    d2 = 2 * (gi / (li * (li + lb)) - x / (li * lb) + gb / (lb * (li + lb)))
    beta = KAPPA / (4 * math.pi) * torch.log(1.1 / COREA * torch.sqrt(li * lb))
    return beta * torch.linalg.cross(d1, d2), d1


def _images():
    r = (-1, 0, 1)
    return [(i, j, k) for i in r for j in r for k in r]


def _terms(r, d):
    """One segment each: r from the target to its start, d along it.  The form that cancels
    nothing; the reference drops the terms with 4ac - b^2 at or below rounding."""
    e = r + d
    nr, ne = r.norm(dim=-1), e.norm(dim=-1)
    cr = torch.linalg.cross(r, d)
    re = (r * e).sum(-1)
    cr2 = (cr * cr).sum(-1)
    pp = nr * ne
    den = torch.where(re < 0, cr2 / (pp - re), pp + re)
    f = KAPPA / (4 * math.pi) * (1 / nr + 1 / ne) / den
    return cr * f[..., None], cr2


def _direct(x, d, prv):
    n = x.shape[0]
    u = torch.zeros_like(x)
    own = torch.arange(n, device=x.device)
    rows = max(1, int(3e7) // n)
    for im in _images():
        shifted = x + torch.tensor(im, device=x.device, dtype=torch.float64) * BOX
        for a in range(0, n, rows):
            b = min(n, a + rows)
            t, cr2 = _terms(shifted[None] - x[a:b, None], d[None].expand(b - a, n, 3))
            skip = cr2 == 0
            k = own[a:b]
            skip[k - a, prv[a:b]] = True
            if im == (0, 0, 0):
                skip[k - a, k] = True
            u[a:b] += torch.where(skip[..., None], 0.0, t).sum(1)
    return u


def _octree(x, d):
    """Cells with their points' mean position and summed segment vectors, level by level; a
    list of (centre, vector, count, width, first child, children, member) per level."""
    n, dev = x.shape[0], x.device
    node = torch.zeros(n, dtype=torch.long, device=dev)   # each point's cell on this level
    who = torch.arange(n, device=dev)
    corner = torch.full((1, 3), -BOX / 2, dtype=torch.float64, device=dev)
    width, levels = BOX, []
    while who.numel():
        m = corner.shape[0]
        p = x[who]
        cnt = torch.bincount(node, minlength=m)
        cen = torch.zeros(m, 3, dtype=torch.float64, device=dev).index_add_(0, node, p) / cnt[:, None]
        vec = torch.zeros(m, 3, dtype=torch.float64, device=dev).index_add_(0, node, d[who])
        member = torch.zeros(m, dtype=torch.long, device=dev).scatter_(0, node, who)
        half = width / 2.0
        keep = cnt[node] > 1
        up = p[keep] >= corner[node[keep]] + half
        key = node[keep] * 8 + 4 * up[:, 1] + 2 * up[:, 2] + 1 * up[:, 0]
        child, inverse = torch.unique(key, return_inverse=True)
        kids = torch.bincount(child // 8, minlength=m)
        first = torch.cumsum(kids, 0) - kids
        levels.append((cen, vec, cnt, width, first, kids, member))
        o = child % 8
        step = torch.stack([o & 1, (o >> 2) & 1, (o >> 1) & 1], 1).double() * half
        corner = corner[child // 8] + step
        who, node, width = who[keep], inverse, half
    return levels


def _tree(x, d, prv, theta):
    levels = _octree(x, d)
    n, dev = x.shape[0], x.device
    u = torch.zeros_like(x)
    for im in _images():
        shift = torch.tensor(im, device=dev, dtype=torch.float64) * BOX
        for a in range(0, n, 32768):
            who = torch.arange(a, min(n, a + 32768), device=dev)
            cell = torch.zeros_like(who)
            for k, (cen, vec, cnt, width, first, kids, member) in enumerate(levels):
                r = cen[cell] + shift - x[who]
                dist = r.norm(dim=1)
                mid = cen[cell] - _middle(levels, k, cell)
                gap = dist - mid.norm(dim=1)
                angle = width / torch.where(gap > 0, gap, dist)
                leaf = cnt[cell] == 1
                take = leaf | (angle < theta)
                if k > 0:
                    j = member[cell]
                    ok = take
                    if im == (0, 0, 0):
                        ok = ok & ~(leaf & ((j == who) | (j == prv[who])))
                    t, cr2 = _terms(r[ok], vec[cell[ok]])
                    u.index_add_(0, who[ok], torch.where((4 * cr2 < 2.220446049250313e-16)[:, None], 0.0, t))
                who, cell = who[~take], cell[~take]
                reps = kids[cell]
                start = torch.repeat_interleave(torch.cumsum(reps, 0) - reps, reps)
                nxt = torch.repeat_interleave(first[cell], reps)
                cell = nxt + torch.arange(nxt.shape[0], device=dev) - start
                who = torch.repeat_interleave(who, reps)
                if not who.numel():
                    break
    return u


def _middle(levels, k, cell):
    """The middle of the cells (from any of their points: cells tile the box)."""
    cen, width = levels[k][0], levels[k][3]
    return (torch.floor((cen[cell] + BOX / 2) / width) + 0.5) * width - BOX / 2
