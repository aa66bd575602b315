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

// loop_killer (reconnection.f90:155-182): a loop that meets a pinned point is left alone.
__device__ void loop_killer(const SolidState &S, SysDyn &d, int s, int base, int particle) {
  const int pc = d.pcount;
  int counter = 1, next = particle;
  for (int it = 1; it <= pc; ++it) {
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
// precon 296 -> 5 (before: one thread per system).
constexpr int kSweep = 256;

// Whether an earlier launch failed.  One thread reads the error word for the block: other
// systems' blocks of this launch may set it meanwhile (pinsert's), and a block whose threads
// disagreed would part at the sweep's barriers.
__device__ bool failed_before(const unsigned *err) {
  __shared__ unsigned s_err;
  if (threadIdx.x == 0) s_err = *err;
  __syncthreads();
  return s_err != 0;
}

template <class Test, class Passed, class After, class Act>
__device__ void ordered_sweep(int base, int n, Test test, Passed passed, After after, Act act) {
  __shared__ int s_first;
  const int tid = threadIdx.x;
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
    } else {
      act(base + first);  // every thread: thread 0 applies, the others may help
      i0 = first + 1;
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
  int free_at = 1;            // no slot below the first empty one empties during the sweep
  bool full = false;
  auto length = [&](int g) {
    double x[3], gi[3];
    load3(S.X, T, g, x);
    load3(S.GI, T, g, gi);
    return dist_gen(x, gi);
  };
  auto tested = [&](int g) { return S.nxt[g] != 0 && !pin_i(S.pin[g]); };
  ordered_sweep(
      base, old_pcount, [&](int g) { return !full && tested(g) && length(g) > sc.delta; },
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
        free_at = first_free(S, base, free_at, pc);
        if (free_at > pc && pc + 1 > sc.cap) {
          full = true;
          if (tid == 0) atomicOr(err, DERR_CAPACITY);
          return;
        }
        if (tid != 0) return;
        double x[3], gi[3], gb[3];
        load3(S.X, T, g, x);
        load3(S.GI, T, g, gi);
        load3(S.GB, T, g, gb);
        const double disti = dist_gen(x, gi);
        total_length = e_add(total_length, disti);
        margin_note(d, 0, disti, sc.delta);
        const int pn = base + free_at;
        if (free_at > pc) {
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
      });
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
  ordered_sweep(
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
        if (threadIdx.x != 0) return;
        if (S.nxt[g] == 0) return;
        const int pari = S.nxt[g], parb = S.prv[g];
        const double cd = S.CD[g];
        if (cd > NV_EPS) margin_note(d, 2, cd, sc.delta / 2.);
        if (!((cd < sc.delta / 2.) && (cd > NV_EPS))) return;
        const int j = S.cl[g];
        if (j == pari || j == parb || j == 0) return;
        if (S.nxt[j] == 0) return;
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
        if (dot_val > 0.9) return;
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
        if (!(l_after <= l_before)) return;
        d.recon_count += 1;
        log_event(S, d, s, base, NV_EV_RECON, g, j);
        S.nxt[parjb] = pari;
        S.prv[pari] = parjb;
        S.nxt[g] = j;
        S.prv[j] = g;
        loop_killer(S, d, s, base, pari);
        loop_killer(S, d, s, base, g);
      });
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
  ordered_sweep(
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
        if (threadIdx.x != 0) return;
        if (S.nxt[g] == 0) return;
        // a cleared pair: the reference goes on to test the cleared i at x = 0, inside every
        // wall while delta < box, so nothing more happens to it
        if (clear_wall_pair(S, d, s, base, g)) return;
        if (pin_i(S.pin[g]) || pin_b(S.pin[g])) return;
        for (int a = 0; a < 3; ++a) {  // x, y, z walls in turn, each on the state the last left
          if (!sc.solid[a]) continue;
          const double xa = S.X[a * T + g];
          const double lim = e_mul(0.5, e_sub(sc.box[a], sc.delta));
          int side = 0;
          if (xa > lim) side = 1;
          else if (xa < -lim) side = -1;
          if (side == 0) continue;
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
      });
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
  ordered_sweep(
      base, d.pcount, [&](int g) { return looked_at(g) && distance(g) < thr; },
      [&](int g, int) {
        if (looked_at(g)) margin_note(d, 1, distance(g), thr);
      },
      [](int) {},
      [&](int g) {
        if (threadIdx.x != 0) return;
        if (S.nxt[g] == 0) return;
        if (pin_i(S.pin[g])) return;
        const int infront = S.nxt[g];
        if (pin_i(S.pin[infront])) return;
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
      });
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
