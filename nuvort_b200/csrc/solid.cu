// solid.cu -- the topology stages of systems with solid walls, as exact ordered sweeps.
//
// Points pinned to a wall (pinnedi: the segment in front ends in the wall, infront is the
// point itself; pinnedb: the same behind) change every topology stage of the reference:
// pinsert and premove skip them and clean up pairs of wall points (src/line.f90:36,109-127),
// loop_killer stops at them (src/reconnection.f90:164), and wall_recon (:66-150) cuts a
// filament that reaches a wall into two pinned ends.  Solid-wall runs are small (the
// reference's lattice example has a few thousand points), so here each of those stages is
// one block per solid-wall system (ordered_sweep below), an acting slot's statements by one
// thread in the reference's order on the live device state; the parallel stages of topo.cu
// skip these systems.  Events go to the same log and digest as the parallel stages'.
#include "handle.cuh"

namespace {

struct SolidState {
  double *X, *U, *U1, *U2, *GI, *GB, *CD;
  int *nxt, *prv, *cl, *pin;
  long long T;
  DevEvent *ev;
  int *ev_count;
  int ev_cap;
};

__device__ bool solid_system(const SysConst &sc) { return sc.solid[0] || sc.solid[1] || sc.solid[2]; }

// clear_particle (general.f90:10-20): u_mf, u_sup, curv and stretch are kept, as there.
__device__ void clear_slot(const SolidState &S, int g) {
  for (int c = 0; c < 3; ++c) {
    S.X[c * S.T + g] = 0; S.U[c * S.T + g] = 0; S.U1[c * S.T + g] = 0; S.U2[c * S.T + g] = 0;
    S.GI[c * S.T + g] = 0; S.GB[c * S.T + g] = 0;
  }
  S.nxt[g] = 0; S.prv[g] = 0; S.cl[g] = 0; S.CD[g] = 0; S.pin[g] = 0;
}

// get_ghost_p (boundary.f90:26-84) of slot g on the current state
__device__ void refresh(const SysConst &sc, const SolidState &S, int g) {
  double x[3], xi[3], xb[3], gi[3], gb[3];
  load3(S.X, S.T, g, x);
  load3(S.X, S.T, S.nxt[g], xi);
  load3(S.X, S.T, S.prv[g], xb);
  ghosts_of(sc, S.pin[g], x, xi, xb, gi, gb);
  store3(S.GI, S.T, g, gi);
  store3(S.GB, S.T, g, gb);
}

// One logged event; j is a count for loop kills, wall cuts and wall-pair clean-ups.
__device__ void log_event(const SolidState &S, SysDyn &d, int s, int base, int kind, int i, int j) {
  const bool count = kind == NV_EV_LOOPKILL || kind == NV_EV_WALL || kind == NV_EV_CLEAR;
  const int seq = d.event_seq++;
  d.ev_hash += event_digest(seq, d.itime, kind, i - base, count ? j : j - base);
  const int a = atomicAdd(S.ev_count, 1);
  if (a < S.ev_cap) S.ev[a] = DevEvent{s, seq, d.itime, kind, i, j};
}

// loop_killer (reconnection.f90:155-182): a loop that meets a pinned point is left alone.  Only
// fewer than four points matter, so the count stops after three hops.
__device__ void loop_killer(const SolidState &S, SysDyn &d, int s, int base, int particle) {
  const int pc = d.pcount;
  int counter = 1, next = particle;
  for (int it = 1; it <= min(pc, 3); ++it) {
    if (pin_i(S.pin[next]) || pin_b(S.pin[next])) return;
    next = S.nxt[next];
    if (next == particle) break;
    counter = counter + 1;
  }
  if (counter < 4) {
    log_event(S, d, s, base, NV_EV_LOOPKILL, particle, counter);
    d.loop_kills += 1;
    d.nlive -= counter;
    next = particle;
    for (int it = 1; it <= pc; ++it) {
      const int store_next = S.nxt[next];
      clear_slot(S, next);
      next = store_next;
      if (next == particle) break;
    }
  }
}

// The reference's sweep over slots 1..n in ascending order, by a block: the threads take test(g)
// of kSweep consecutive slots on the current state -- whether slot g does more than be looked at
// -- and thread 0 runs act(g), the reference's statements, for the first slot whose test passes;
// the slots after it are tested again on the state it left.  passed(g, i) is called for every
// slot that only is looked at, i its place in the chunk, and after(k) once its first k slots have
// been.  So events happen one by one and in
// order, and everything between them costs a chunk of tests instead of a chain of loads per
// slot: 1,273 points, in us a step, premove 590 -> 8, pinsert 500 -> 17, wall_recon 370 -> 7,
// precon 296 -> 5 (before: one thread per system).  Where events crowd, the chunks and barriers
// would cost more than they save: after two events within kNear slots thread 0 goes on alone, by
// serial(g), the reference's statements whatever slot g does, until kNear slots pass without an
// event; it says whether g had one (24,297 points that all insert: 84 ms; 121 with a chunk for
// every event, 78 by one thread).  Not for the cuts, of which the time goes into the events.
constexpr int kSweep = 256, kCrowd = 3;

// Whether an earlier launch failed.  One thread reads the error word for the block: other
// systems' blocks of this launch may set it meanwhile (pinsert's), and a block whose threads
// disagreed would part at the sweep's barriers.
__device__ bool failed_before(const unsigned *err) {
  __shared__ unsigned s_err;
  if (threadIdx.x == 0) s_err = *err;
  __syncthreads();
  return s_err != 0;
}

template <int kNear, class Test, class Passed, class After, class Act, class Serial>
__device__ void ordered_sweep(int base, int n, Test test, Passed passed, After after, Act act, Serial serial) {
  __shared__ int s_first, s_next, s_last;
  const int tid = threadIdx.x;
  int last = -kNear;  // the last event's slot
  for (int i0 = 1; i0 <= n;) {
    const int i = i0 + tid;
    if (tid == 0) s_first = INT_MAX;
    __syncthreads();
    if (i <= n && test(base + i)) atomicMin(&s_first, i);
    __syncthreads();
    const int first = s_first;
    if (i <= n && i < first) passed(base + i, tid);
    __syncthreads();
    after(min(first, min(n + 1, i0 + kSweep)) - i0);
    if (first == INT_MAX) {
      i0 += kSweep;
    } else if (kNear == 0 || first - last > kNear) {
      act(base + first);  // every thread: thread 0 applies, the others may help
      last = first;
      i0 = first + 1;
    } else {
      if (tid == 0) {
        int k = first, l = first;
        for (; k <= n && k - l <= kNear; ++k)
          if (serial(base + k)) l = k;
        s_next = k;
        s_last = l;
      }
      __syncthreads();
      last = s_last;
      i0 = s_next;
    }
    __syncthreads();
  }
}

// The first slot in from..n (system-local) with an empty infront link, n + 1 if none; by the block.
__device__ int first_free(const SolidState &S, int base, int from, int n) {
  __shared__ int s_free;
  for (; from <= n; from += kSweep) {
    if (threadIdx.x == 0) s_free = INT_MAX;
    __syncthreads();
    const int i = from + threadIdx.x;
    if (i <= n && S.nxt[base + i] == 0) atomicMin(&s_free, i);
    __syncthreads();
    const int f = s_free;
    __syncthreads();
    if (f != INT_MAX) return f;
  }
  return n + 1;
}

// pinsert (line.f90:18-96) for one system.
__global__ void __launch_bounds__(kSweep) k_solid_pinsert(const SysConst *__restrict__ scs, SysDyn *dyn, int nsys,
                                                          SolidState S, unsigned *err) {
  __shared__ double s_len[kSweep];
  const int s = blockIdx.x, tid = threadIdx.x;
  if (s >= nsys || !solid_system(scs[s]) || failed_before(err)) return;
  const SysConst &sc = scs[s];
  SysDyn &d = dyn[s];
  const int base = sc.base;
  const long long T = S.T;
  const int old_pcount = d.pcount;
  bool live = false;
  for (int i = 1 + tid; i <= old_pcount; i += kSweep) live |= S.nxt[base + i] > 0;
  if (__syncthreads_or(live) == 0) {
    if (tid == 0) atomicOr(err, DERR_EMPTY);
    return;
  }
  if (tid == 0) d.old_pcount = old_pcount;
  double total_length = 0.0;  // thread 0: in slot order, as the reference adds
  __shared__ int s_free_at;   // no slot below it is empty, nor empties during the sweep
  __shared__ bool s_full;
  if (tid == 0) {
    s_free_at = 1;
    s_full = false;
  }
  __syncthreads();
  auto length = [&](int g) {
    double x[3], gi[3];
    load3(S.X, T, g, x);
    load3(S.GI, T, g, gi);
    return dist_gen(x, gi);
  };
  auto tested = [&](int g) { return S.nxt[g] != 0 && !pin_i(S.pin[g]); };
  // The insertion at slot g, its length measured: into slot s_free_at (by thread 0).  False: out of slots.
  auto insert = [&](int g, double disti, int pc) {
    if (s_free_at > pc && pc + 1 > sc.cap) {
      s_full = true;
      atomicOr(err, DERR_CAPACITY);
      return false;
    }
    double x[3], gi[3], gb[3];
    load3(S.X, T, g, x);
    load3(S.GI, T, g, gi);
    load3(S.GB, T, g, gb);
    const int pn = base + s_free_at;
    if (s_free_at > pc) {
      d.pcount = pc + 1;
      clear_slot(S, pn);
    }
    // the new point (line.f90:62-84)
    double xn[3];
    new_point(x, gi, gb, disti, xn);
    const int nx = S.nxt[g];
    for (int c = 0; c < 3; ++c) {
      S.X[c * T + pn] = xn[c];
      S.U[c * T + pn] = e_mul(0.5, e_add(S.U[c * T + g], S.U[c * T + nx]));
      S.U1[c * T + pn] = 0.0;
      S.U2[c * T + pn] = 0.0;
    }
    S.pin[pn] = 0;  // the pinned conditions zeroed (line.f90:82-84)
    S.prv[pn] = g;
    S.nxt[pn] = nx;
    refresh(sc, S, pn);
    S.prv[nx] = pn;
    refresh(sc, S, nx);
    S.nxt[g] = pn;
    refresh(sc, S, g);
    log_event(S, d, s, base, NV_EV_INSERT, g, pn);
    d.insert_count += 1;
    d.nlive += 1;
    return true;
  };
  auto measure = [&](int g) {  // by thread 0, in slot order
    const double disti = length(g);
    total_length = e_add(total_length, disti);
    margin_note(d, 0, disti, sc.delta);
    return disti;
  };
  ordered_sweep<kCrowd>(
      base, old_pcount, [&](int g) { return !s_full && tested(g) && length(g) > sc.delta; },
      [&](int g, int k) {
        const bool t = tested(g);
        s_len[k] = t ? length(g) : 0.0;
        if (t) margin_note(d, 0, s_len[k], sc.delta);
      },
      [&](int n) {  // in order (0 for the slots that are not tested)
        if (tid == 0)
          for (int k = 0; k < n; ++k) total_length = e_add(total_length, s_len[k]);
      },
      [&](int g) {
        // the first empty slot (minloc(f(:)%infront)), else the array grows by one
        const int pc = *(volatile int *)&d.pcount;
        const int f = first_free(S, base, s_free_at, pc);
        if (tid != 0) return;
        s_free_at = f;
        insert(g, measure(g), pc);
      },
      [&](int g) {
        if (s_full || !tested(g)) return false;
        const double disti = measure(g);
        if (!(disti > sc.delta)) return false;
        const int pc = d.pcount;
        int f = s_free_at;
        while (f <= pc && S.nxt[base + f] != 0) ++f;
        s_free_at = f;
        return insert(g, disti, pc);
      });
  const bool full = s_full;
  if (full) return;
  int empty = 0;
  const int pc = *(volatile int *)&d.pcount;
  for (int i0 = 1; i0 <= pc; i0 += kSweep)
    empty += __syncthreads_count(i0 + tid <= pc && S.nxt[base + i0 + tid] == 0);
  if (tid == 0) {
    d.total_length = total_length;
    d.avg_sep = total_length / (double)(old_pcount - empty);
  }
}

// Two wall points next to each other, i pinned behind and its point in front pinned in
// front, are cleared together (line.f90:125-127, reconnection.f90:71-75).
__device__ bool clear_wall_pair(const SolidState &S, SysDyn &d, int s, int base, int g) {
  if (!pin_b(S.pin[g])) return false;
  const int nx = S.nxt[g];
  if (!pin_i(S.pin[nx])) return false;
  const int n = nx == g ? 1 : 2;
  log_event(S, d, s, base, NV_EV_CLEAR, g, n);
  clear_slot(S, nx);
  clear_slot(S, g);
  d.nlive -= n;
  return true;
}

// precon (reconnection.f90:11-61) for one system; pinned points never reach it as i or j
// (pclose gives them closestd = 100 and skips them as candidates).
__global__ void __launch_bounds__(kSweep) k_solid_precon(const SysConst *__restrict__ scs, SysDyn *dyn, int nsys,
                                                         SolidState S, const unsigned *err) {
  const int s = blockIdx.x;
  if (s >= nsys || !solid_system(scs[s]) || failed_before(err)) return;
  const SysConst &sc = scs[s];
  SysDyn &d = dyn[s];
  if ((d.itime % sc.recon_shots) != 0) return;
  const int base = sc.base;
  const long long T = S.T;
  // The reference's statements for slot g (by thread 0); whether its closest point was near enough.
  auto slot = [&](int g) {
    if (S.nxt[g] == 0) return false;
    const int pari = S.nxt[g], parb = S.prv[g];
    const double cd = S.CD[g];
    if (cd > NV_EPS) margin_note(d, 2, cd, sc.delta / 2.);
    if (!((cd < sc.delta / 2.) && (cd > NV_EPS))) return false;
    const int j = S.cl[g];
    if (j == pari || j == parb || j == 0) return true;
    if (S.nxt[j] == 0) return true;
    const int parjb = S.prv[j];
    double t1[3], t2[3], x[3], gi_[3], gb_[3];
    for (int q = 0; q < 2; ++q) {  // norm_tanf (general.f90:106-117)
      double *t = q ? t2 : t1;
      const int p = q ? j : g;
      load3(S.X, T, p, x);
      load3(S.GI, T, p, gi_);
      load3(S.GB, T, p, gb_);
      deriv1(x, gi_, gb_, t);
      const double len = e_sqrt(e_add(e_add(e_sq(t[0]), e_sq(t[1])), e_sq(t[2])));
      for (int c = 0; c < 3; ++c) t[c] = e_div(t[c], len);
    }
    const double dot_val = dot3(t1, t2);
    margin_note(d, 3, dot_val, 0.9);
    if (dot_val > 0.9) return true;
    double xi[3], gii[3], gbi[3], xj[3], gij[3], gbj[3], xpi[3], xpj[3];
    load3(S.X, T, g, xi);
    load3(S.GI, T, g, gii);
    load3(S.GB, T, g, gbi);
    load3(S.X, T, j, xj);
    load3(S.GI, T, j, gij);
    load3(S.GB, T, j, gbj);
    load3(S.X, T, pari, xpi);
    load3(S.X, T, parjb, xpj);
    const double l_before =
        e_add(e_add(e_add(dist_gen(xi, gii), dist_gen(xi, gbi)), dist_gen(xj, gij)), dist_gen(xj, gbj));
    const double l_after =
        e_add(e_add(e_add(dist_gen(xi, gbi), dist_gen(xi, xj)), dist_gen(xj, gij)), dist_gen(xpi, xpj));
    if (!(l_after <= l_before)) return true;
    d.recon_count += 1;
    log_event(S, d, s, base, NV_EV_RECON, g, j);
    S.nxt[parjb] = pari;
    S.prv[pari] = parjb;
    S.nxt[g] = j;
    S.prv[j] = g;
    loop_killer(S, d, s, base, pari);
    loop_killer(S, d, s, base, g);
    return true;
  };
  ordered_sweep<0>(
      base, d.pcount,
      [&](int g) {
        const double cd = S.CD[g];
        return S.nxt[g] != 0 && cd < sc.delta / 2. && cd > NV_EPS;
      },
      [&](int g, int) {
        if (S.nxt[g] != 0 && S.CD[g] > NV_EPS) margin_note(d, 2, S.CD[g], sc.delta / 2.);
      },
      [](int) {},
      [&](int g) {
        if (threadIdx.x == 0) slot(g);
      },
      slot);
}

// wall_recon (reconnection.f90:66-150) for one system: a point within delta/2 of a solid
// wall is removed and the filament cut there, its neighbours pinned to that wall.
__global__ void __launch_bounds__(kSweep) k_solid_wall_recon(const SysConst *__restrict__ scs, SysDyn *dyn, int nsys,
                                                             SolidState S, const unsigned *err) {
  const int s = blockIdx.x;
  if (s >= nsys || !solid_system(scs[s]) || failed_before(err)) return;
  const SysConst &sc = scs[s];
  SysDyn &d = dyn[s];
  if ((d.itime % sc.recon_shots) != 0) return;
  const int base = sc.base;
  const long long T = S.T;
  // The reference's statements for slot g (by thread 0); whether they did anything.
  auto slot = [&](int g) {
    if (S.nxt[g] == 0) return false;
    // a cleared pair: the reference goes on to test the cleared i at x = 0, inside every
    // wall while delta < box, so nothing more happens to it
    if (clear_wall_pair(S, d, s, base, g)) return true;
    if (pin_i(S.pin[g]) || pin_b(S.pin[g])) return false;
    bool cut = false;
    for (int a = 0; a < 3; ++a) {  // x, y, z walls in turn, each on the state the last left
      if (!sc.solid[a]) continue;
      const double xa = S.X[a * T + g];
      const double lim = e_mul(0.5, e_sub(sc.box[a], sc.delta));
      int side = 0;
      if (xa > lim) side = 1;
      else if (xa < -lim) side = -1;
      if (side == 0) continue;
      cut = true;
      const int pari = S.nxt[g], parb = S.prv[g];
      int w[3] = {0, 0, 0};
      w[a] = side;
      S.pin[pari] = pin_encode(pin_i(S.pin[pari]), 1, w);
      S.prv[pari] = pari;
      S.pin[parb] = pin_encode(1, pin_b(S.pin[parb]), w);
      S.nxt[parb] = parb;
      clear_slot(S, g);
      int cleared = 1;
      if (pin_i(S.pin[pari]) && pin_b(S.pin[pari])) {
        clear_slot(S, pari);
        ++cleared;
      }
      if (pin_i(S.pin[parb]) && pin_b(S.pin[parb])) {
        clear_slot(S, parb);
        ++cleared;
      }
      log_event(S, d, s, base, NV_EV_WALL, g, cleared);
      d.wall_recon_count += 1;
      d.nlive -= cleared;
    }
    return cut;
  };
  ordered_sweep<0>(
      base, d.pcount,
      [&](int g) {
        if (S.nxt[g] == 0) return false;
        const int pin = S.pin[g];
        if (pin_b(pin) && pin_i(S.pin[S.nxt[g]])) return true;  // a pair to clear
        if (pin_i(pin) || pin_b(pin)) return false;
        for (int a = 0; a < 3; ++a)
          if (sc.solid[a] && fabs(S.X[a * T + g]) > e_mul(0.5, e_sub(sc.box[a], sc.delta))) return true;
        return false;
      },
      [](int, int) {}, [](int) {},
      [&](int g) {
        if (threadIdx.x == 0) slot(g);
      },
      slot);
}

// premove (line.f90:103-129) for one system.
__global__ void __launch_bounds__(kSweep) k_solid_premove(const SysConst *__restrict__ scs, SysDyn *dyn, int nsys,
                                                          SolidState S, const unsigned *err) {
  const int s = blockIdx.x;
  if (s >= nsys || !solid_system(scs[s]) || failed_before(err)) return;
  const SysConst &sc = scs[s];
  SysDyn &d = dyn[s];
  if ((d.itime % sc.recon_shots) != 0) return;
  const int base = sc.base;
  const long long T = S.T;
  const double thr = e_mul(.99, sc.delta);
  auto looked_at = [&](int g) { return S.nxt[g] != 0 && !pin_i(S.pin[g]) && !pin_i(S.pin[S.nxt[g]]); };
  auto distance = [&](int g) {
    double x[3], y[3];
    load3(S.X, T, g, x);
    load3(S.X, T, S.nxt[S.nxt[g]], y);
    return dist_gen(x, y);
  };
  // The reference's statements for slot g (by thread 0); whether its test passed.
  auto slot = [&](int g) {
    if (S.nxt[g] == 0) return false;
    if (pin_i(S.pin[g])) return false;
    const int infront = S.nxt[g];
    if (pin_i(S.pin[infront])) return false;
    const int tinfront = S.nxt[infront];
    double xi[3], xt[3];
    load3(S.X, T, g, xi);
    load3(S.X, T, tinfront, xt);
    const double dii = dist_gen(xi, xt);
    margin_note(d, 1, dii, thr);
    if (dii < thr) {
      S.prv[tinfront] = g;
      S.nxt[g] = tinfront;
      clear_slot(S, infront);
      log_event(S, d, s, base, NV_EV_REMOVE, g, infront);
      d.nlive -= 1;
      loop_killer(S, d, s, base, g);
      d.remove_count += 1;
    }
    clear_wall_pair(S, d, s, base, g);
    return dii < thr;
  };
  ordered_sweep<kCrowd>(
      base, d.pcount, [&](int g) { return looked_at(g) && distance(g) < thr; },
      [&](int g, int) {
        if (looked_at(g)) margin_note(d, 1, distance(g), thr);
      },
      [](int) {},
      [&](int g) {
        if (threadIdx.x == 0) slot(g);
      },
      slot);
}

}  // namespace

static SolidState solid_state(nv_handle *h) {
  return SolidState{h->x,   h->u,   h->u1,      h->u2,  h->gi,        h->gb,           h->closestd,
                    h->nxt, h->prv, h->closest, h->pin, h->T,         h->d_events,     h->d_event_count,
                    h->event_cap};
}

void launch_solid_pinsert(nv_handle *h) {
  if (!h->any_solid) return;
  k_solid_pinsert<<<h->nsys, kSweep, 0, h->stream>>>(h->d_sc, h->d_dyn, h->nsys, solid_state(h), h->d_err);
}
void launch_solid_precon(nv_handle *h) {
  if (!h->any_solid) return;
  k_solid_precon<<<h->nsys, kSweep, 0, h->stream>>>(h->d_sc, h->d_dyn, h->nsys, solid_state(h), h->d_err);
}
void launch_wall_recon(nv_handle *h) {
  if (!h->any_solid) return;
  ++h->links_epoch;
  k_solid_wall_recon<<<h->nsys, kSweep, 0, h->stream>>>(h->d_sc, h->d_dyn, h->nsys, solid_state(h), h->d_err);
}
void launch_solid_premove(nv_handle *h) {
  if (!h->any_solid) return;
  k_solid_premove<<<h->nsys, kSweep, 0, h->stream>>>(h->d_sc, h->d_dyn, h->nsys, solid_state(h), h->d_err);
}
