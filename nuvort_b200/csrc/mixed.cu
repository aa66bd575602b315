// mixed.cu -- mixed-precision direct sum and the FP64 epilogue shared with the mixed tree walk.
//
// k_direct_mixed<W>: a block of W warps per 32 targets and periodic image, each warp (a lane per
// target) over its share of every tile of the target system's segments (W = 8; 1 for ensembles of
// small systems).  The tiles stream through shared memory by 1-D bulk copies (pairs of segments
// side by side, 96 bytes a pair: position hi, position lo, segment vector).  r = x_j - x_i is formed from the hi/lo split, so
// it is exact to ~1e-16 before rounding to FP32.  Every 32 terms are summed in FP32 and those
// sums are added with Kahan compensation; pairs closer than near_radius are evaluated in FP64
// with the reference expression from the FP64 segment records.  The warps' sums are added in
// FP64, in warp order; per-image partial sums go to a buffer; k_mixed_combine adds them per
// target in FP64, in image order, to the FP64 local term and mutual friction
// (timestep.f90:79-140).
#include "handle.cuh"
#include "mixed.cuh"
#include "tma.cuh"

namespace {

constexpr int kWarpPairs = 16;  // segment pairs (96 B each) of an FP32 sub-sum
// A block of W warps that share 32 targets (8, or 1 for many small systems): pairs per staged tile,
// tiles in flight
template <int W>
struct MixedShape {
  static constexpr int kPairs = W == 8 ? 128 : 32, kStages = W == 8 ? 4 : 3;
  static constexpr size_t kSmem = (size_t)kStages * kPairs * 96;
};

// One term in FP64 from the FP64 segment records, for near and ill-conditioned pairs: the
// reference's skip decision (4ac - b^2 == 0, timestep.f90:166,192) in its own arithmetic, the
// value from the cancellation-free form.
__device__ __noinline__ double3 direct_term64(const double4 *__restrict__ rec, double s0, double s1, double s2,
                                              double x0, double x1, double x2, double gq) {
  const double4 A = rec[0], B = rec[1];
  const double r[3] = {e_sub(e_add(A.x, s0), x0), e_sub(e_add(A.y, s1), x1), e_sub(e_add(A.z, s2), x2)};
  const double d[3] = {B.x, B.y, B.z};
  const double a = e_add(e_add(e_sq(r[0]), e_sq(r[1])), e_sq(r[2]));
  const double b = e_mul(2.0, dot3(r, d));
  if (e_sub(e_mul(e_mul(4.0, a), B.w), e_mul(b, b)) == 0.0) return make_double3(0., 0., 0.);
  double t[3];
  term64_stable(r, d, a, gq, t);
  return make_double3(t[0], t[1], t[2]);
}

// What the lanes of a warp hold of their targets.
struct MixedTarget : LaneTarget {
  double x[3], s[3];  // position, image shift
  int behind, own;    // segments (from 0) that are skipped
  int n;              // segments of the system: the last pair's second half may lie past them
  bool active;
};

// The halves of pair p that this lane's guards send to FP64, into n.
__device__ __forceinline__ void add_exact(const bool bad[2], const MixedTarget &t, int p,
                                          const double4 *__restrict__ seg64, double gq64, double n[3]) {
  if (!(t.active && (bad[0] || bad[1]))) return;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int j = 2 * p + h;
    if (!(h ? bad[1] : bad[0]) || j >= t.n || j == t.behind || j == t.own) continue;
    const double3 v = direct_term64(seg64 + 2 * (long long)j, t.s[0], t.s[1], t.s[2], t.x[0], t.x[1], t.x[2], gq64);
    n[0] += v.x;
    n[1] += v.y;
    n[2] += v.z;
  }
}

// A pair that some lane of the warp is not far from: every lane's own guards decide between
// FP32 and FP64 (into n).
__device__ __forceinline__ void pair_guarded(const PairVec &r, const PairSeg &d, const MixedTarget &t, int p,
                                             float near2, const Fp32Guards &gd, const double4 *__restrict__ seg64,
                                             double gq64, f32x2 u[3], double n[3]) {
  const PairGeo g = pair_geo(r, d);
  const f32x2 c = square2(d.dx, d.dy, d.dz), cr2 = square2(g.cx, g.cy, g.cz);
  float f[2];
  bool bad[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    auto of = [&](f32x2 v) { return h ? hi2(v) : lo2(v); };
    const float a = of(r.a), ee = of(g.ee), re = of(g.re), pp = of(g.pp), cc = of(c), k2 = of(cr2);
    const int j = 2 * p + h;
    bad[h] = j == t.behind || j == t.own || a < near2 || !(a > 0.f) || k2 < gd.line * cc * fminf(a, ee) ||
             ee < gd.end * fmaxf(a, cc) || pp + re < gd.angle * pp;
    // pp + r.e = |r x d|^2 / (pp - r.e) when r.e < 0: no cancellation either way
    const bool obtuse = re < 0.f;
    f[h] = bad[h] ? 0.f : of(g.num) * (obtuse ? pp - re : 1.f) * rcp_fast(obtuse ? k2 : pp + re);
  }
  const f32x2 ff = pack2(f[0], f[1]);
  u[0] = fma2(ff, g.cx, u[0]);
  u[1] = fma2(ff, g.cy, u[1]);
  u[2] = fma2(ff, g.cz, u[2]);
  add_exact(bad, t, p, seg64, gq64, n);
}

// floats as integers in the same order, and back
__device__ __forceinline__ int ordered(float x) {
  const int i = __float_as_int(x);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float float_of(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

// The pairs of a sub-sum (bit p: pair p) that need no guard for any of the warp's targets: all targets
// lie within a ball around the point that `c` holds as a target, of radius R, so |r| of each lies
// between |rc| - R and |rc| + R and |r x d| is at least |rc x d| - R |d|.  A pair is beyond every
// target's far bound where (|rc| - R)^2 exceeds it, and the line guard cannot act where |rc x d|
// exceeds |d| (R + sqrt(line) (|rc| + R)).  A lane takes one pair for all targets.
struct WarpBall {
  LaneTarget c;
  float radius, reach, slope;  // R, R (1 + sqrt(line)) and sqrt(line), widened for the FP32 rounding
};
__device__ __forceinline__ unsigned clean_mask(const ulonglong2 *pairs, int np, const WarpBall &ball) {
  const int lane = threadIdx.x & 31;
  static_assert(kWarpPairs <= 32, "a lane per pair");
  bool clean = false;
  if (lane < np) {
    const PairVec r = pair_vec(pairs + 6 * lane, ball.c);
    const PairSeg d = pair_seg(pairs + 6 * lane);
    const f32x2 kMinus = pack2(-1.f, -1.f), reach = pack2(ball.reach, ball.reach), slope = pack2(ball.slope, ball.slope),
                radius = pack2(-ball.radius, -ball.radius), shrink = pack2(0.99999f, 0.99999f);
    const f32x2 cx = fma2(r.ry, d.dz, mul2(r.rz, d.ndy)), cy = fma2(r.rz, d.dx, mul2(mul2(r.rx, kMinus), d.dz)),
                cz = fma2(r.rx, d.dy, mul2(r.ry, d.ndx));
    const f32x2 rl = pack2(sqrt_fast(lo2(r.a)), sqrt_fast(hi2(r.a)));
    const f32x2 over = fma2(slope, rl, reach), gap = fma2(shrink, rl, radius), gap2 = mul2(gap, gap);
    const f32x2 cr2 = square2(cx, cy, cz), lim = mul2(square2(d.dx, d.dy, d.dz), mul2(over, over));
    clean = lo2(gap) > 0.f && hi2(gap) > 0.f && lo2(gap2) > lo2(d.far) && hi2(gap2) > hi2(d.far) &&
            lo2(cr2) >= lo2(lim) && hi2(cr2) >= hi2(lim);
  }
  return __ballot_sync(0xffffffffu, clean);
}

// Bound: the FP32 pipe (about 35 lane operations a far term, the adds, multiplies and FMAs of
// two segments packed into one instruction) and the special-function unit.  Nearly all pairs of a
// tangle need no guard for any target of the warp; clean_mask finds them, once per sub-sum, and
// they are taken four at a time without a test or a vote.  Of the others, those that every
// target is far from take the line guard alone, target by target, the rest all guards.  The tiles
// pass through a ring of kStages buffers with an mbarrier for full and one for empty each, so
// that no warp waits for the block's others.
// 30,011 points: 36.6 ms; 1,501 points: 138 us (a lane per target and image with scalar
// arithmetic and all guards, 113 issue slots a term: 74.1 ms and 409 us; packed, but all guards
// and a barrier per tile: 55.4 ms and 236 us; a vote per pair on the far bound, the line guard's
// exact test on every far pair: 44.8 ms and 153 us, without that guard 38.8 ms and 136 us).
template <int W>
__global__ void __launch_bounds__(32 * W, 24 / W) k_direct_mixed(
    const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn, const int4 *__restrict__ work,
    const double *__restrict__ X, const int *__restrict__ nxt, const int *__restrict__ prv,
    const float *__restrict__ seg32, const double4 *__restrict__ seg64, double *__restrict__ partial, long long T,
    double near_factor, Fp32Guards gd, unsigned *err) {
  constexpr int kPairs = MixedShape<W>::kPairs, kStages = MixedShape<W>::kStages;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  ulonglong2 *tiles = reinterpret_cast<ulonglong2 *>(smem_raw);  // [kStages][6 * kPairs]
  __shared__ double s_red[3][W][32];
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages];
  __shared__ int s_abort;

  const int4 w = work[blockIdx.x];  // system, image, first slot
  const SysConst &sc = scs[w.x];
  const int base = sc.base, m = w.y;
  const int pc = dyn[w.x].pcount;
  if (w.z - base > pc) return;  // block-uniform
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int g = w.z + lane;
  MixedTarget t;
  t.active = (g - base <= pc) && (g - base <= sc.cap) && nxt[g] != 0;
  if (tid == 0) {
    s_abort = (*err != 0);
    for (int k = 0; k < kStages; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], W);
    }
    mbar_fence_init();
  }
  __syncthreads();
  if (s_abort) return;

  // target, moved by minus the image shift: r = (x_j + s) - x_i = x_j - (x_i - s); a lane
  // without one is far from everything.  The behind segment is skipped in every image, the
  // target's own in the central one (their pairs take the guarded path, which skips them).
  t.behind = t.own = -1;
  t.n = pc;
  for (int c = 0; c < 3; ++c) {
    t.s[c] = m > 0 ? sc.shift[m - 1][c] : 0.0;
    t.x[c] = -1e9;
  }
  if (t.active) {
    load3(X, T, g, t.x);
    t.behind = prv[g] - base - 1;
    if (m == 0) t.own = g - base - 1;
  }
  for (int c = 0; c < 3; ++c) {
    const double v = t.s[c] - t.x[c];
    const float h = (float)v, l = (float)(v - (double)h);
    t.h[c] = pack2(h, h);
    t.l[c] = pack2(l, l);
  }
  const int behind_p = t.behind >= 0 ? t.behind >> 1 : -1;
  const bool any = __any_sync(0xffffffffu, t.active);
  WarpBall ball;
  {
    const float sin_line = sqrtf(gd.line);
    float half2 = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {  // the ball around the box of the targets, by FP32 positions
      const float x = (float)t.x[c];
      const float lo = float_of(__reduce_min_sync(0xffffffffu, t.active ? ordered(x) : INT_MAX)),
                  hi = float_of(__reduce_max_sync(0xffffffffu, t.active ? ordered(x) : INT_MIN));
      const float mid = any ? 0.5f * lo + 0.5f * hi : 0.f;
      const double v = t.s[c] - (double)mid;
      const float h = (float)v, l = (float)(v - (double)h);
      const float half = any ? fmaxf(hi - mid, mid - lo) + 1e-6f * fmaxf(fabsf(lo), fabsf(hi)) : 0.f;
      ball.c.h[c] = pack2(h, h);
      ball.c.l[c] = pack2(l, l);
      half2 = fmaf(half, half, half2);
    }
    ball.slope = sin_line * 1.00001f + 1e-6f;
    ball.radius = sqrtf(half2) * 1.00001f;
    ball.reach = ball.radius * (1.f + ball.slope);
  }
  const double gq64 = sc.quant_circ / (4.0 * NV_PI);
  const double nr = near_factor * sc.delta;
  const float near2 = (float)(nr * nr);
  const double4 *rec64 = seg64 + 2 * (long long)(base + 1);

  const int np = (pc + 1) / 2;  // pairs of the system (an odd last one is half empty)
  const int nt = (np + kPairs - 1) / kPairs;
  const float *src = seg32 + seg32_at(base, 1);
  auto issue = [&](int k) {
    const unsigned bytes = (unsigned)min(kPairs, np - k * kPairs) * 96u;
    mbar_expect_tx(&full[k % kStages], bytes);
    bulk_g2s(tiles + (k % kStages) * 6 * kPairs, src + 24ll * k * kPairs, bytes, &full[k % kStages]);
  };
  int issued = 0;
  if (tid == 0)
    for (; issued < nt && issued < kStages - 1; ++issued) issue(issued);
  float hs[3] = {0, 0, 0}, hc[3] = {0, 0, 0};  // Kahan sums
  double n[3] = {0, 0, 0};                     // FP64 terms
  for (int k = 0; k < nt; ++k) {
    bool ok = true;
    if (tid == 0 && issued < nt) {  // the next tile, once every warp has left its buffer
      if (issued >= kStages) ok = mbar_wait(&empty[issued % kStages], (unsigned)((issued / kStages - 1) & 1));
      if (ok) issue(issued++);
    }
    ok = ok && mbar_wait(&full[k % kStages], (unsigned)((k / kStages) & 1));
    if (!__all_sync(0xffffffffu, ok)) {  // gave up: the other warps give up at their own waits
      if (lane == 0) atomicOr(err, DERR_TIMEOUT);
      break;
    }
    const ulonglong2 *tile = tiles + (k % kStages) * 6 * kPairs;
    const int in_tile = min(kPairs, np - k * kPairs);
    for (int p0 = wid * kWarpPairs; p0 < in_tile; p0 += W * kWarpPairs) {
      const int p1 = min(in_tile, p0 + kWarpPairs);
      const int bp = behind_p - k * kPairs;
      // (a pair that holds some target's behind segment is never clean)
      unsigned clean = clean_mask(tile + 6 * p0, p1 - p0, ball) &
                       ~__reduce_or_sync(0xffffffffu, bp >= p0 && bp < p1 ? 1u << (bp - p0) : 0u);
      f32x2 u[3] = {pack2(0.f, 0.f), pack2(0.f, 0.f), pack2(0.f, 0.f)};
      auto fast = [&](int p) {
        const ulonglong2 *q = tile + 6 * p;
        const PairVec r = pair_vec(q, t);
        const PairGeo g2 = pair_geo(r, pair_seg(q));
        const f32x2 sum = add2(g2.pp, g2.re);
        const f32x2 f = mul2(g2.num, pack2(rcp_fast(lo2(sum)), rcp_fast(hi2(sum))));
        u[0] = fma2(f, g2.cx, u[0]);
        u[1] = fma2(f, g2.cy, u[1]);
        u[2] = fma2(f, g2.cz, u[2]);
      };
#pragma unroll 1
      for (int p = p0; p < p1; ++p) {
        if ((clean & 15u) == 15u) {  // (no bits past p1)
          fast(p);
          fast(p + 1);
          fast(p + 2);
          fast(p + 3);
          clean >>= 4;
          p += 3;
          continue;
        }
        const bool plain = clean & 1u;
        clean >>= 1;
        if (plain) {
          fast(p);
          continue;
        }
        const ulonglong2 *q = tile + 6 * p;
        const PairVec r = pair_vec(q, t);
        const PairSeg d = pair_seg(q);
        if (__all_sync(0xffffffffu, lo2(r.a) > lo2(d.far) && hi2(r.a) > hi2(d.far) && p != bp)) {
          // the line guard alone, target by target
          const PairGeo g2 = pair_geo(r, d);
          const f32x2 sum = add2(g2.pp, g2.re), c = square2(d.dx, d.dy, d.dz), cr2 = square2(g2.cx, g2.cy, g2.cz);
          const bool bad[2] = {lo2(cr2) < gd.line * lo2(c) * fminf(lo2(r.a), lo2(g2.ee)),
                               hi2(cr2) < gd.line * hi2(c) * fminf(hi2(r.a), hi2(g2.ee))};
          const f32x2 f = mul2(g2.num, pack2(bad[0] ? 0.f : rcp_fast(lo2(sum)), bad[1] ? 0.f : rcp_fast(hi2(sum))));
          u[0] = fma2(f, g2.cx, u[0]);
          u[1] = fma2(f, g2.cy, u[1]);
          u[2] = fma2(f, g2.cz, u[2]);
          add_exact(bad, t, k * kPairs + p, rec64, gq64, n);
        } else {
          pair_guarded(r, d, t, k * kPairs + p, near2, gd, rec64, gq64, u, n);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) kahan_add(hs[c], hc[c], lo2(u[c]) + hi2(u[c]));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[k % kStages]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) s_red[c][wid][lane] = gq64 * ((double)hs[c] - (double)hc[c]) + n[c];
  __syncthreads();
  // A give-up leaves copies in flight: wait for them (bounded) before shared memory is released.
  if (tid == 0)
    for (int k = max(0, issued - kStages); k < issued; ++k) mbar_wait(&full[k % kStages], (unsigned)((k / kStages) & 1));
  if (!t.active) return;
  for (int c = wid; c < 3; c += W) {
    double v = 0.;
#pragma unroll
    for (int k = 0; k < W; ++k) v += s_red[c][k][lane];
    partial[((long long)m * 3 + c) * T + g] = v;
  }
}

// Per target: u = local + partial[image 0] + sum_{images 1..n} partial[image], then MF and
// the imposed flow, all in FP64 (timestep.f90:79-92,123-140).
__global__ void k_mixed_combine(const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn,
                                const int2 *__restrict__ work, const double *__restrict__ X,
                                const double *__restrict__ GI, const double *__restrict__ GB,
                                const int *__restrict__ nxt, const double *__restrict__ partial,
                                double *__restrict__ U, long long T, bool per_image, const int *__restrict__ iperm,
                                const unsigned *err) {
  if (*err) return;
  const int2 w = work[blockIdx.x];
  const SysConst &sc = scs[w.x];
  const int g = w.y + threadIdx.x;
  const int k = g - sc.base;
  if (k > dyn[w.x].pcount || k > sc.cap || nxt[g] == 0) return;
  if (iperm && (sc.walk_lo > 1 || sc.walk_hi <= sc.cap)) {  // a walk range: its targets only
    const int q = iperm[g] - sc.base;
    if (q < sc.walk_lo || q >= sc.walk_hi) return;
  }
  double xi[3], gi[3], gb[3], u[3], fdot[3];
  load3(X, T, g, xi);
  load3(GI, T, g, gi);
  load3(GB, T, g, gb);
  local_velocity(sc, xi, gi, gb, u, fdot);
  double b0[3], bs[3] = {0, 0, 0};
  for (int c = 0; c < 3; ++c) b0[c] = partial[(long long)c * T + g];
  if (per_image)  // the direct sum's images; the tree walk's one sum holds them all
    for (int m = 1; m <= sc.n_shift; ++m)
      for (int c = 0; c < 3; ++c) bs[c] += partial[((long long)m * 3 + c) * T + g];
  for (int c = 0; c < 3; ++c) u[c] = e_add(e_add(u[c], b0[c]), bs[c]);
  mf_epilogue(sc, dyn[w.x], xi, fdot, u, g);
  store3(U, T, g, u);
}

}  // namespace

cudaError_t mixed_kernels_setup() {
  return cudaFuncSetAttribute(k_direct_mixed<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)MixedShape<8>::kSmem);
}

void launch_direct_mixed(nv_handle *h) {
  auto launch = [&](auto kernel, int w, size_t smem, const int4 *work, int n) {
    if (n > 0)
      kernel<<<n, 32 * w, smem, h->stream>>>(h->d_sc, h->d_dyn, work, h->x, h->nxt, h->prv, h->seg32, h->seg, h->partial,
                                             h->T, h->near_factor, h->guards, h->d_err);
  };
  launch(k_direct_mixed<8>, 8, MixedShape<8>::kSmem, h->d_work_img, h->n_work_img);
  launch(k_direct_mixed<1>, 1, MixedShape<1>::kSmem, h->d_work_img1, h->n_work_img1);
}

void launch_mixed_combine(nv_handle *h, int which) {
  const int2 *wl = which == 1 ? h->d_work_direct : h->d_work_tree;
  const int n = which == 1 ? h->n_work_direct : h->n_work_tree;
  if (n == 0) return;
  k_mixed_combine<<<n, h->direct_tb, 0, h->stream>>>(h->d_sc, h->d_dyn, wl, h->x, h->gi, h->gb, h->nxt, h->partial,
                                                     h->u, h->T, which == 1, which == 2 ? tree_iperm(h) : nullptr,
                                                     h->d_err);
}
