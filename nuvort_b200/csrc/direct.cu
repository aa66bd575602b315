// direct.cu -- the direct Biot-Savart sum over all segments and their periodic images.
//
// Plain FP64 kernel (k_direct_fp64): one thread per target point, the segment records of
// the target's system streamed through shared memory in tiles by 1-D bulk copies
// (cp.async.bulk + mbarrier, double-buffered).  The summation order is the reference's:
//   u_bs = sum_j ascending (unshifted)                   timestep.f90:83-85
//   u_bs' = sum_images (in periodic_loop_array order) sum_j ascending   :88-92
// with every operation rounded once (the quotients as fp64.cuh says), so the result is
// bit-identical to the reference arithmetic except for the ulp-level difference of the device
// log() in the local term.  The image loop is outside the tile loop for that reason: each image
// re-streams the tiles (from L2; the kernel is FP64-pipe bound, not memory bound).
#include <vector>

#include "fp64.cuh"
#include "handle.cuh"
#include "tma.cuh"

namespace {

constexpr int kDirectTJ = 128;  // segments per staged tile (64 B each)

template <int TJ>
__global__ void __launch_bounds__(64) k_direct_fp64(
    const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn, const int2 *__restrict__ work,
    const double *__restrict__ X, const double *__restrict__ GI, const double *__restrict__ GB,
    const int *__restrict__ nxt, const int *__restrict__ prv, const double4 *__restrict__ seg,
    double *__restrict__ U, long long T, unsigned *err, const int *__restrict__ targets = nullptr, int ntargets = 0,
    double *__restrict__ Uout = nullptr) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double4 *tiles = reinterpret_cast<double4 *>(smem_raw);  // [2][2*TJ]
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ int s_abort;

  const int2 w = work[blockIdx.x];
  const SysConst &sc = scs[w.x];
  const int base = sc.base;
  const int pc = dyn[w.x].pcount;
  const int tid = threadIdx.x;
  int g;
  bool active;
  if (targets) {  // listed targets (k-th thread of block b takes targets[64 b + k])
    const int idx = w.y + tid;
    g = idx < ntargets ? targets[idx] : base;
    active = idx < ntargets && g > base && g - base <= pc && nxt[g] != 0;
  } else {
    if (w.y - base > pc) return;  // block-uniform: every target beyond pcount
    g = w.y + tid;
    active = (g - base <= pc) && (g - base <= sc.cap) && nxt[g] != 0;
  }

  // One thread reads the sticky error word so that the whole block agrees on it.
  if (tid == 0) {
    s_abort = (*err != 0);
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (s_abort) return;

  double xi[3] = {0, 0, 0};
  int pi = -1;
  if (active) {
    load3(X, T, g, xi);
    pi = prv[g];
  }
  const int nt = (pc + TJ - 1) / TJ;
  const int Q = (1 + sc.n_shift) * nt;
  const double qc = sc.quant_circ, two_pi = sc.two_pi;

  auto issue = [&](int q) {
    const int t = q % nt;
    const int n = min(TJ, pc - t * TJ);
    const int buf = q & 1;
    mbar_expect_tx(&bar[buf], (unsigned)(n * 64));
    bulk_g2s(tiles + buf * 2 * TJ, seg + 2 * (long long)(base + 1 + t * TJ), (unsigned)(n * 64), &bar[buf]);
  };
  int issued = 0;
  if (tid == 0) {
    if (Q > 0) issue(0);
    if (Q > 1) issue(1);
  }
  issued = Q < 2 ? Q : 2;

  double ub0[3] = {0, 0, 0}, ubs[3] = {0, 0, 0};
  int consumed = 0;
  for (int q = 0; q < Q; ++q) {
    const int buf = q & 1;
    const bool ok = mbar_wait(&bar[buf], (unsigned)((q >> 1) & 1));
    if (__syncthreads_or(!ok)) {
      if (tid == 0) atomicOr(err, DERR_TIMEOUT);
      break;
    }
    consumed = q + 1;
    const int m = q / nt, t = q % nt;
    const int n = min(TJ, pc - t * TJ);
    const int j0 = base + 1 + t * TJ;
    const double4 *tl = tiles + buf * 2 * TJ;
    if (active) {
      // the unshifted image as a shift of +0.0, which leaves the positions as they are; a
      // skipped term adds +0.0, which leaves a sum that starts at +0.0 as it is (so do empty
      // slots, whose records are zero, and the target's own segment, r = 0)
      const double s0 = m ? sc.shift[m - 1][0] : 0.0, s1 = m ? sc.shift[m - 1][1] : 0.0,
                   s2 = m ? sc.shift[m - 1][2] : 0.0;
      double ub[3] = {m ? ubs[0] : ub0[0], m ? ubs[1] : ub0[1], m ? ubs[2] : ub0[2]};
#pragma unroll 2
      for (int jj = 0; jj < n; ++jj) {
        const double4 A = tl[2 * jj], B = tl[2 * jj + 1];
        const int gj = j0 + jj;
        const double r[3] = {e_sub(e_add(A.x, s0), xi[0]), e_sub(e_add(A.y, s1), xi[1]), e_sub(e_add(A.z, s2), xi[2])};
        const double d[3] = {B.x, B.y, B.z};
        const double a = e_add(e_add(e_sq(r[0]), e_sq(r[1])), e_sq(r[2]));
        double tm[3];
        bs_term(gj != pi, r, d, a, B.w, qc, two_pi, tm);
        ub[0] = e_add(ub[0], tm[0]);
        ub[1] = e_add(ub[1], tm[1]);
        ub[2] = e_add(ub[2], tm[2]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) (m ? ubs[c] : ub0[c]) = ub[c];
    }
    __syncthreads();
    if (q + 2 < Q) {
      if (tid == 0) issue(q + 2);
      issued = q + 3;
    }
  }
  // A give-up leaves copies in flight: wait for them (bounded) before shared memory is
  // released.
  if (tid == 0)
    for (int q = consumed; q < issued; ++q) mbar_wait(&bar[q & 1], (unsigned)((q >> 1) & 1));
  if (!active) return;

  // solid walls: the mirror images, in mirror order, each over j ascending (timestep.f90:94-98)
  double um[3] = {0, 0, 0};
  if (sc.n_mirror) {
    const int pin_g = sc.pin[g];
    for (int m = 0; m < sc.n_mirror; ++m) {
      const bool own = mirror_skips_own(sc, pin_g, m);
      for (int j = base + 1; j <= base + pc; ++j) {
        double tm[3];
        mirror_term_sum(sc, m, X, GI, nxt, T, j, g, pi, pin_g, own, xi, tm);
        for (int c = 0; c < 3; ++c) um[c] = e_add(um[c], tm[c]);
      }
    }
  }

  double gi[3], gb[3], u[3], fdot[3];
  load3(GI, T, g, gi);
  load3(GB, T, g, gb);
  local_velocity(sc, xi, gi, gb, u, fdot);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], ub0[c]);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], ubs[c]);
  if (sc.n_mirror)
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], um[c]);
  mf_epilogue(sc, dyn[w.x], xi, fdot, u, targets ? -1 : g);
  if (targets) {
    const int idx = w.y + tid;
    for (int c = 0; c < 3; ++c) Uout[3 * (long long)idx + c] = u[c];
    return;
  }
  store3(U, T, g, u);
}

// The same sums with the work of a target spread over a block, one summing warp and eight
// computing warps to G targets.  The computing warps take the terms of a step -- TJ consecutive
// segments for each target, of the sequence unshifted image, shifted images, mirror images,
// each over j ascending -- into shared memory while the summing
// warp adds the previous step's, one lane per (target, component), in sequence order: the
// additions are the reference's, in the reference's order, only the terms are computed
// elsewhere.  Skipped terms are stored as +0.0: the accumulators start at +0.0 and a
// round-to-nearest sum is never -0.0 unless both operands are, so adding +0.0 leaves them bit
// for bit unchanged, exactly as skipping does.
//
// Bound: the FP64 pipe (84 FP64 instructions a term, see fp64.cuh) where the blocks fill the
// GPU: 12,289 points 31.4 ms (102 ms with the IEEE operations one by one, three computing warps
// and a barrier every 192 terms), 18.4 ms at the pipe's full rate.  With few targets the
// summing lanes' chain, one addition of 8 cycles per segment and image, which is why they only
// load (ahead of the chain) and add: 600 points 183 us, before 357 us.  A step is one tile of
// one image, so that the image and its shift are uniform; four terms a thread and step with
// G = 8 share the cost of the barrier and of the staging (two: 32.6 ms).  The lanes of a warp
// take G targets x 32/G segments, and a step's segment records are staged in shared memory a
// step ahead, each read from global memory once for the block's G targets.
constexpr int kSplitWarps = 8;
constexpr int kSplitComp = 32 * kSplitWarps;       // computing threads
constexpr int kSplitThreads = 32 + kSplitComp;
constexpr int kSegPad = 5;  // 16-byte units per staged record (4 used): no bank conflicts at any G

constexpr int split_per(int G) { return G == 8 ? 4 : G == 4 ? 2 : 1; }
constexpr size_t split_smem(int G) {  // the terms and segments of two steps
  const int terms = kSplitComp * split_per(G);
  return 2 * (3 * (terms + (G == 8 ? 8 : 4)) * sizeof(double) + terms / G * kSegPad * sizeof(double2));
}

// acc + p[0] + p[stride] + ... in order, n terms and +0.0s up to a multiple of 16: two sets of
// 8 in turn, one loading while the other is added, without a branch between (the last set
// loaded, from past the end but inside the block's shared memory, is not used).  9.2 cycles per addition alone on its SM; 12.4 as a plain
// loop unrolled by 8, whose loads wait for the chain; 13.5 with the last loads left out.
template <int kStride>
__device__ __forceinline__ double add_in_order(double acc, const double *p, int n) {
  constexpr int kU = 8;
  double a[kU], b[kU];
#pragma unroll
  for (int u = 0; u < kU; ++u) a[u] = p[u * kStride];
  for (int k = 0; k < n; k += 2 * kU) {
#pragma unroll
    for (int u = 0; u < kU; ++u) b[u] = p[(kU + u) * kStride];
#pragma unroll
    for (int u = 0; u < kU; ++u) acc = e_add(acc, a[u]);
    p += 2 * kU * kStride;
#pragma unroll
    for (int u = 0; u < kU; ++u) a[u] = p[u * kStride];
#pragma unroll
    for (int u = 0; u < kU; ++u) acc = e_add(acc, b[u]);
  }
  return acc;
}

template <int G>
__global__ void __launch_bounds__(kSplitThreads, G == 8 ? 2 : 3) k_direct_fp64_split(
    const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn, const int2 *__restrict__ work,
    const double *__restrict__ X, const double *__restrict__ GI, const double *__restrict__ GB,
    const int *__restrict__ nxt, const int *__restrict__ prv, const double4 *__restrict__ seg,
    double *__restrict__ U, long long T, const unsigned *err, const int *__restrict__ targets, int ntargets,
    double *__restrict__ Uout) {
  constexpr int kPer = split_per(G);               // terms per computing thread and step
  constexpr int kTerms = kSplitComp * kPer;        // terms per step
  constexpr int TJ = kTerms / G;                   // segments per step
  constexpr int kStep = kSplitComp / G;            // segments between a thread's terms
  constexpr int kLoads = 4 * TJ / kSplitComp;      // 16-byte loads per thread that stage a step
  static_assert(4 * TJ % kSplitComp == 0 && TJ % 16 == 0, "whole loads per thread, whole sets of additions");
  // component rows of a step's terms, [segment][target]; padded so that the summing lanes of
  // the components read different banks
  constexpr int LD = kTerms + (G == 8 ? 8 : 4);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto s_terms = reinterpret_cast<double(*)[3][LD]>(smem_raw);  // [2][3][LD]
  auto s_seg = reinterpret_cast<double2(*)[TJ * kSegPad]>(smem_raw + sizeof(double) * 2 * 3 * LD);  // [2]
  static_assert(split_smem(G) == sizeof(double) * 2 * 3 * LD + sizeof(double2) * 2 * TJ * kSegPad, "layout");
  __shared__ double s_x[G][3], s_shift[27][3];
  __shared__ double s_sum[G][3][3];
  __shared__ int s_g[G], s_p[G], s_act[G], s_pin[G];
  __shared__ int s_abort;

  const int2 w = work[blockIdx.x];
  const SysConst &sc = scs[w.x];
  const int base = sc.base;
  const int pc = dyn[w.x].pcount;
  const int tid = threadIdx.x;
  if (!targets && w.y - base > pc) return;  // block-uniform: every target beyond pcount
  if (tid == 0) s_abort = (*err != 0);
  for (int k = tid; k < 81; k += kSplitThreads) s_shift[k / 3][k % 3] = k < 3 ? 0.0 : sc.shift[k / 3 - 1][k % 3];
  if (tid < G) {
    int g;
    bool act;
    if (targets) {
      const int idx = w.y + tid;
      g = idx < ntargets ? targets[idx] : base;
      act = idx < ntargets && g > base && g - base <= pc && nxt[g] != 0;
    } else {
      g = w.y + tid;
      act = g - base <= pc && g - base <= sc.cap && nxt[g] != 0;
    }
    s_g[tid] = g;
    s_act[tid] = act;
    s_p[tid] = act ? prv[g] : -1;
    s_pin[tid] = act && sc.pin ? sc.pin[g] : 0;
    double xi[3] = {0, 0, 0};
    if (act) load3(X, T, g, xi);
    for (int c = 0; c < 3; ++c) s_x[tid][c] = xi[c];
  }
  __syncthreads();
  if (s_abort) return;

  const double qc = sc.quant_circ, two_pi = sc.two_pi;
  double acc0 = 0.0, accs = 0.0, accm = 0.0;  // summing lanes: unshifted, shifted, mirror sums
  const bool comp = tid >= 32;
  const int e0 = comp ? tid - 32 : 0;
  const int tq = e0 % G;  // computing threads: their target
  const bool act = s_act[tq];  // used by the mirror images; other inactive targets' sums go nowhere
  {  // the unshifted and the shifted images; a step is one tile of one image
    const double2 *rec = reinterpret_cast<const double2 *>(seg + 2 * (long long)(base + 1));
    const int nt = (pc + TJ - 1) / TJ, Q = (1 + sc.n_shift) * nt;
    const double x0 = s_x[tq][0], x1 = s_x[tq][1], x2 = s_x[tq][2];
    const int behind = s_p[tq] - base - 1;  // as a segment counted from 0
    int m = 0, t = 0;                       // image and tile of the step, of the summing warp's step
    int tl = 0;                             // tile staged next
    double2 ld[kLoads];
    auto fetch = [&]() {
#pragma unroll
      for (int k = 0; k < kLoads; ++k) {
        const int jl = tl * TJ + e0 / 4 + k * (kSplitComp / 4);
        ld[k] = jl < pc ? __ldg(rec + 4 * (long long)jl + (e0 & 3)) : make_double2(0., 0.);
      }
      if (++tl == nt) tl = 0;
    };
    auto stage = [&](int b) {
#pragma unroll
      for (int k = 0; k < kLoads; ++k) s_seg[b][(e0 / 4 + k * (kSplitComp / 4)) * kSegPad + (e0 & 3)] = ld[k];
    };
    if (comp) {
      fetch();
      stage(0);
    }
    __syncthreads();
    for (int q = 0; q <= Q; ++q) {
      const int b = q & 1;
      if (comp) {
        if (q < Q) {
          fetch();  // the next step's tile, stored once this step's terms are done
          const double sh0 = s_shift[m][0], sh1 = s_shift[m][1], sh2 = s_shift[m][2];
          // records past the end of the list and empty slots are zero, and the target's own
          // segment has r = 0: all have 4ac - b^2 = 0 and drop out like the reference's
#pragma unroll 2
          for (int r = 0; r < kPer; ++r) {
            const double2 *sp = &s_seg[b][(e0 / G + r * kStep) * kSegPad];
            const double2 A0 = sp[0], A1 = sp[1], B0 = sp[2], B1 = sp[3];
            const double rr[3] = {e_sub(e_add(A0.x, sh0), x0), e_sub(e_add(A0.y, sh1), x1), e_sub(e_add(A1.x, sh2), x2)};
            const double d[3] = {B0.x, B0.y, B1.x};
            const double a = e_add(e_add(e_sq(rr[0]), e_sq(rr[1])), e_sq(rr[2]));
            double tm[3];
            bs_term(t * TJ + e0 / G + r * kStep != behind, rr, d, a, B1.y, qc, two_pi, tm);
#pragma unroll
            for (int c = 0; c < 3; ++c) s_terms[b][c][e0 + r * kSplitComp] = tm[c];
          }
          stage(b ^ 1);
          if (++t == nt) {
            t = 0;
            ++m;
          }
        }
      } else if (q >= 1 && tid < 3 * G) {  // add the terms of step q-1, in slot order
        const double *row = &s_terms[b ^ 1][tid / G][tid % G];
        const int n = min(TJ, pc - t * TJ);
        if (m == 0) acc0 = add_in_order<G>(acc0, row, n);
        else accs = add_in_order<G>(accs, row, n);
        if (++t == nt) {
          t = 0;
          ++m;
        }
      }
      __syncthreads();
    }
  }
  if (sc.n_mirror) {  // solid walls: the mirror images, in mirror order
    const long long F = (long long)sc.n_mirror * pc;
    const int Q = (int)((F + TJ - 1) / TJ);
    for (int q = 0; q <= Q; ++q) {
      if (comp) {
        for (int r = 0; r < kPer; ++r) {
          const long long f = (long long)q * TJ + e0 / G + r * kStep;
          double tm[3] = {0.0, 0.0, 0.0};
          if (act && f < F) {
            const int mm = (int)(f / pc), jj = (int)(f - (long long)mm * pc);
            mirror_term_sum(sc, mm, X, GI, nxt, T, base + 1 + jj, s_g[tq], s_p[tq], s_pin[tq],
                            mirror_skips_own(sc, s_pin[tq], mm), s_x[tq], tm);
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) s_terms[q & 1][c][e0 + r * kSplitComp] = tm[c];
        }
      } else if (q >= 1 && tid < 3 * G) {
        const int n = (int)min((long long)TJ, F - (long long)(q - 1) * TJ);
        accm = add_in_order<G>(accm, &s_terms[(q - 1) & 1][tid / G][tid % G], n);
      }
      __syncthreads();
    }
  }
  if (tid < 3 * G) {
    s_sum[tid % G][tid / G][0] = acc0;
    s_sum[tid % G][tid / G][1] = accs;
    s_sum[tid % G][tid / G][2] = accm;
  }
  __syncthreads();
  if (tid >= G || !s_act[tid]) return;
  const int g = s_g[tid];
  double xi[3] = {s_x[tid][0], s_x[tid][1], s_x[tid][2]};
  double gi[3], gb[3], u[3], fdot[3];
  load3(GI, T, g, gi);
  load3(GB, T, g, gb);
  local_velocity(sc, xi, gi, gb, u, fdot);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], s_sum[tid][c][0]);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], s_sum[tid][c][1]);
  if (sc.n_mirror)
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], s_sum[tid][c][2]);
  mf_epilogue(sc, dyn[w.x], xi, fdot, u, targets ? -1 : g);
  if (targets) {
    const int idx = w.y + tid;
    for (int c = 0; c < 3; ++c) Uout[3 * (long long)idx + c] = u[c];
    return;
  }
  store3(U, T, g, u);
}

template <int G>
void launch_split(cudaStream_t st, const nv_handle *h, const int2 *work, int nwork, const int *targets, int ntargets,
                  double *Uout) {
  k_direct_fp64_split<G><<<nwork, kSplitThreads, split_smem(G), st>>>(h->d_sc, h->d_dyn, work, h->x, h->gi, h->gb, h->nxt, h->prv,
                                                   h->seg, h->u, h->T, h->d_err, targets, ntargets, Uout);
}

void launch_split_g(int G, cudaStream_t st, const nv_handle *h, const int2 *work, int nwork, const int *targets,
                    int ntargets, double *Uout) {
  switch (G) {
    case 1: launch_split<1>(st, h, work, nwork, targets, ntargets, Uout); break;
    case 2: launch_split<2>(st, h, work, nwork, targets, ntargets, Uout); break;
    case 4: launch_split<4>(st, h, work, nwork, targets, ntargets, Uout); break;
    default: launch_split<8>(st, h, work, nwork, targets, ntargets, Uout); break;
  }
}

template <int G>
cudaError_t allow_split() {
  return cudaFuncSetAttribute(k_direct_fp64_split<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)split_smem(G));
}

}  // namespace

cudaError_t direct_kernels_setup() {
  for (cudaError_t e : {allow_split<1>(), allow_split<2>(), allow_split<4>(), allow_split<8>()})
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

// Direct-sum targets per block in use for this many target slots (direct_split, set by
// nv_set_direct_split, overrides the choice): 8 per block of the split kernel, except
//   * 2 while the blocks of 2 (three to an SM) about fit the GPU at once, counting two thirds
//     of the slots as live: the summing chain sets the time then, and it is the shorter the
//     fewer terms an SM computes beside it (600 points: 181 us, 203 with 8; but 1000 points,
//     a second wave of blocks: 450 us, 322 with 8; 4 per block is nowhere ahead by 3 %).  Handles
//     allocated to their points lose by it from 889 to 1,332 slots, where the share of live
//     slots, known only at upload, would decide for 8 (714 us at 1000 points before either);
//   * one thread per target (64 to a block) from 80,000 slots on, four warps to each
//     scheduler, which need no exchange (50,000 points: 623 ms, 488 with 8; 80,000: 1.22 s,
//     1.23 s).
int direct_targets_per_block(const nv_handle *h, long long slots) {
  if (h->direct_split > 0) return h->direct_split;
  if (slots >= 80000) return 64;
  return slots <= 9LL * n_sms_host() ? 2 : 8;
}

void launch_direct(nv_handle *h) {
  if (h->n_work_direct == 0) return;
  if (h->direct_g < 64) {
    launch_split_g(h->direct_g, h->stream, h, h->d_work_split, h->n_work_split, nullptr, 0, nullptr);
    return;
  }
  const size_t smem = 2 * 2 * kDirectTJ * sizeof(double4);
  k_direct_fp64<kDirectTJ><<<h->n_work_direct, 64, smem, h->stream>>>(
      h->d_sc, h->d_dyn, h->d_work_direct, h->x, h->gi, h->gb, h->nxt, h->prv, h->seg, h->u, h->T, h->d_err);
}

// Direct sum on explicitly given buffers (used by the static-scratch entry point).
void launch_direct_raw(cudaStream_t st, const SysConst *sc, const SysDyn *dyn, const int2 *work, int nwork,
                       const double *x, const double *gi, const double *gb, const int *nxt, const int *prv,
                       const double4 *seg, double *u, long long T, unsigned *err) {
  if (nwork == 0) return;
  const size_t smem = 2 * 2 * kDirectTJ * sizeof(double4);
  k_direct_fp64<kDirectTJ><<<nwork, 64, smem, st>>>(sc, dyn, work, x, gi, gb, nxt, prv, seg, u, T, err);
}

// FP64 direct-sum velocity (the reference's BS scheme, whatever the system's own scheme) at
// listed target slots; u3 is a device buffer of 3*n doubles (point-major, listed order).
void launch_direct_targets(nv_handle *h, int sys, const int *d_targets, int n, double *d_u3) {
  if (n <= 0) return;
  const int G = direct_targets_per_block(h, n);
  std::vector<int2> w;
  for (int b = 0; b < (n + G - 1) / G; ++b) w.push_back(make_int2(sys, G * b));
  int2 *dw = nullptr;
  cudaMallocAsync((void **)&dw, w.size() * sizeof(int2), h->stream);
  cudaMemcpyAsync(dw, w.data(), w.size() * sizeof(int2), cudaMemcpyHostToDevice, h->stream);
  if (G < 64) {
    launch_split_g(G, h->stream, h, dw, (int)w.size(), d_targets, n, d_u3);
  } else {
    const size_t smem = 2 * 2 * kDirectTJ * sizeof(double4);
    k_direct_fp64<kDirectTJ><<<(int)w.size(), 64, smem, h->stream>>>(h->d_sc, h->d_dyn, dw, h->x, h->gi, h->gb,
                                                                     h->nxt, h->prv, h->seg, h->u, h->T, h->d_err,
                                                                     d_targets, n, d_u3);
  }
  cudaFreeAsync(dw, h->stream);
}
