// tree.cu -- Barnes-Hut octree on the device: build, velocity walk, closest-point walk.
//
// Build (construct_tree/build_tree/new_tree, src/tree.f90:38-157), top-down, one level per
// pass, all systems of the handle at once:
//   * Node k's members are kept as a contiguous list of slots in ascending slot order.
//     Splitting a node is a stable 8-way partition of that list by octant, so every child's
//     list is again in ascending slot order -- the order in which the reference sums a
//     node's centre and circulation (tree.f90:124-143), reproduced exactly.
//   * The octant of a point is decided by the reference's own membership test against the
//     child's corner, computed with the same FP64 additions (child corner = parent corner
//     (+ width/2)); a point that fails its child's upper bound (rounding can make a child's
//     far face differ by an ulp from the parent's) belongs to no child, as in the reference.
//   * Octant digit = 4*[y upper] + 2*[z upper] + [x upper]: the child order fbl, fbr, ftl,
//     ftr, bbl, bbr, btl, btr of tree.f90:71-93.  Only non-empty children are stored;
//     siblings are contiguous, so a preorder walk follows first_child / skip links.
//   * The root holds every slot (pcount includes empty slots, tree.f90:48), its centre is
//     the mean over live slots and its circulation is zero (tree.f90:50-54).
// Walks: one thread per target point, stackless preorder over first_child/skip, with the
// reference's opening test and arithmetic (tree_walk tree.f90:250-316, closest_tree
// :206-244) in the same order, so the accumulated velocity is the reference's bit for bit.
#include <cmath>

#include <cub/cub.cuh>

#include "fp64.cuh"
#include "handle.cuh"
#include "lists.cuh"
#include "mixed.cuh"

constexpr int kMaxLevels = NV_TREE_MAX_DEPTH;
constexpr int kEnd = -1;
constexpr int kBigNode = 2048;  // nodes with more members are split by a whole block
constexpr int kBlockSumNode = 8192;  // nodes with more members are summed by a whole block
constexpr int kCtrBig = kMaxLevels + 6;  // ctr[kCtrBig]: entries of the block-summed node list
constexpr int kCtrBigSnap = kMaxLevels + 7;  // entries listed when the early block sums start
constexpr int kSnapLevel = 1;  // the early block sums: the big nodes of depth 1, listed by the root's split
// ctr[kCtrSplit + b]: entries of the level lists of nodes to split, by level % 3 = b:
// [+0..+2] nodes above kBigNode members (split by a block), [+3..+5] the others with >= 2
constexpr int kCtrSplit = kMaxLevels + 8;
constexpr int kCtrFail = kMaxLevels + 14;  // lowest level at which a split ran out of room, or INT_MAX
constexpr int kCtrSize = kMaxLevels + 16;
constexpr int kDeferCap = 1 << 20;  // targets with a deferred root test listed per velocity pass

struct TreeBuffers {
  int max_nodes = 0;
  long long max_members = 0;
  double4 *nA = nullptr;  // cent.xyz, width
  double4 *nB = nullptr;  // circ.xyz, geo_dist
  double4 *nP = nullptr;  // corner posx,posy,posz
  int4 *nI = nullptr;     // pcount, first_child, skip, first_next
  int2 *nR = nullptr;     // member range start, member count
  int *nDepth = nullptr;
  int *nLeaf = nullptr;
  int *nKids = nullptr;   // number of children (contiguous from first_child)
  int *members = nullptr;
  // roots: a parallel estimate of the centre with a bound on its distance to the exact
  // (sequential) one, so the walks need not wait for the exact sum; (target, image) pairs
  // whose root test the bound cannot settle are listed and redone once the exact sum is in
  // the roots' split by an ordered pass over the slots (k_root_lists)
  unsigned char *rdig = nullptr;  // per slot: its octant, 8 for none
  int *rrank = nullptr;           // per slot: its rank among its octant's slots
  int *root_rank = nullptr;       // per system and list: the rank at its first slot
  int *root_mb = nullptr;         // per system and octant: member entry of rank 0
  int *root_ok = nullptr;         // per system: the children were made
  unsigned long long *pass_state = nullptr;
  unsigned *pass_ctl = nullptr;
  double4 *root_apx = nullptr;  // per system: centre estimate, bound
  double *root_part = nullptr;  // per system and part: partial sums of x, y, z, |x|, |y|, |z|
  int root_parts = 1;
  int *defer = nullptr;         // slots of the deferred targets
  int *defer_n = nullptr;
  int *bigl = nullptr;    // non-root nodes with more than kBlockSumNode members
  int max_big = 0;
  int *split_blk[3] = {nullptr, nullptr, nullptr};  // nodes of a level split by a block, by level % 3
  int *split_wrp[3] = {nullptr, nullptr, nullptr};  // nodes of a level split by a warp
  int max_blk = 0, max_wrp = 0;
  int grid_levels = kMaxLevels;  // levels below this one are split by the whole GPU
  int *ctr = nullptr;     // [0] n_nodes [1] n_members [2 + L] first node of level L
  // walk order: each system's slots sorted along a Hilbert curve (live slots first)
  unsigned long long *okey[2] = {nullptr, nullptr};
  int *oval[2] = {nullptr, nullptr};
  int *perm = nullptr;  // = oval[1]: position base+q of system s -> slot
  int *iperm = nullptr; // slot -> its position in the walk order (inverse of perm)
  void *sort_tmp = nullptr;
  size_t sort_bytes = 0;
  int key_bits = 0;
  bool built = false;
  MixedNodes mx;
  unsigned prep_epoch = ~0u;  // the handle's links epoch when the mixed records took prv
};

namespace {

constexpr int TB = 256;

// Sort keys of the walk order: (system, class, place of the position on a Hilbert curve through a
// 1024^3 grid of the box); class 0 is the dummy slot, 1 live slots, 2 the rest.  The order only
// decides which lanes walk together; every target's accepted nodes are independent of it.
// Neighbours on the Hilbert curve stay closer together than on the Morton curve (no jumps):
// the mixed walk of 100,000 points visits 5 % fewer nodes and tests 23 % fewer target by target
// (1.54 -> 1.41 ms), the plain walk of 32,768 points takes 2.49 instead of 3.13 ms.
__device__ __forceinline__ unsigned spread3(unsigned v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}
// Grid coordinates (10 bits) to the transposed Hilbert index (J. Skilling, AIP Conf. Proc. 707,
// 381, 2004): interleaving the three words' bits, q[0] first, gives the place on the curve.
__device__ __forceinline__ void hilbert3(unsigned q[3]) {
#pragma unroll
  for (unsigned b = 512; b > 1; b >>= 1) {
    const unsigned low = b - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const unsigned t = (q[0] ^ q[i]) & low;
      if (q[i] & b) {
        q[0] ^= low;
      } else {
        q[0] ^= t;
        q[i] ^= t;
      }
    }
  }
  q[1] ^= q[0];
  q[2] ^= q[1];
  unsigned t = 0;
#pragma unroll
  for (unsigned b = 512; b > 1; b >>= 1)
    if (q[2] & b) t ^= b - 1;
#pragma unroll
  for (int i = 0; i < 3; ++i) q[i] ^= t;
}
__global__ void k_order_keys(const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn,
                             const int *__restrict__ sys_of, const double *__restrict__ X,
                             const int *__restrict__ nxt, unsigned long long *key, int *val, long long T) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= T) return;
  const int s = sys_of[g];
  const SysConst &sc = scs[s];
  const int k = (int)(g - sc.base);
  unsigned long long inner;
  if (k == 0) {
    inner = 0;
  } else if (k <= dyn[s].pcount && nxt[g] != 0) {
    unsigned q[3];
    for (int c = 0; c < 3; ++c) {
      const double f = (X[c * T + g] / sc.bsize + 0.5) * 1024.0;
      q[c] = f <= 0. ? 0u : f >= 1023. ? 1023u : (unsigned)f;
    }
    hilbert3(q);
    inner = (1ull << 32) | (spread3(q[2]) | (spread3(q[1]) << 1) | (spread3(q[0]) << 2));
  } else {
    inner = (2ull << 32) | (unsigned)k;
  }
  key[g] = ((unsigned long long)s << 34) | inner;
  val[g] = (int)g;
}

__global__ void k_inv_perm(const int *__restrict__ perm, int *__restrict__ iperm, long long T) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < T) iperm[perm[i]] = (int)i;
}

__global__ void k_iota(int *v, long long n) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n) v[g] = (int)g;
}

// Octant of x in node (corner P, half-width h), or 8 when x lies in no child.
__device__ __forceinline__ int octant(const double x[3], const double4 P, double h) {
  const double p[3] = {P.x, P.y, P.z};
  int up[3];
  bool in = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double mid = e_add(p[c], h);  // child corner posx+(width/2)      tree.f90:74
    if (x[c] >= mid) {
      up[c] = 1;
      in = in && (x[c] < e_add(mid, h));  // x < posx+width of the upper child
    } else {
      up[c] = 0;
      in = in && (x[c] >= p[c]);  // lower child: posx <= x < posx+width (= mid)
    }
  }
  return in ? (4 * up[1] + 2 * up[2] + up[0]) : 8;
}

__device__ __forceinline__ void load_x(const double *__restrict__ X, long long T, int g, double x[3]) {
  x[0] = __ldg(X + g);
  x[1] = __ldg(X + T + g);
  x[2] = __ldg(X + 2 * T + g);
}

// Whether a split at a level above this one ran out of room (the same answer to every thread of
// this level's kernel, which may itself lower the level noted).
__device__ __forceinline__ bool failed_above(const TreeBuffers &tb, int level) {
  return *(const volatile int *)&tb.ctr[kCtrFail] < level;
}

// What a node's split reserves: child ids, member slots, entries of the next level's block
// and warp split lists (kList), entries of the block-summed node list.
struct SplitNeeds {
  int nchild, kept, nblk, nwrp, nbig;
};
template <bool kList = true>
__device__ SplitNeeds split_needs(const int cnt[8]) {
  SplitNeeds n{0, 0, 0, 0, 0};
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    n.nchild += cnt[d] != 0;
    n.kept += cnt[d];
    if (kList && cnt[d] >= 2) {
      if (cnt[d] > kBigNode) ++n.nblk;
      else ++n.nwrp;
    }
    if (cnt[d] > kBlockSumNode) ++n.nbig;
  }
  return n;
}

// The children of node p at reserved offsets (id0, mb0, qb, qw, qg); false when they do not
// fit the buffers (error set).  The counters have then moved past entries never written, which
// the levels below, the sums and the walks must not read: they return (failed_above).  (Marking
// the entries unused here instead cost the levels' kernel 36 of 157 us at 32,768 points.)
template <bool kList = true>
__device__ bool write_children(TreeBuffers &tb, int p, const int cnt[8], const SplitNeeds &n, int id0, int mb0,
                               int qb, int qw, int qg, unsigned *err) {
  if (id0 + n.nchild > tb.max_nodes || (long long)mb0 + n.kept > tb.max_members || qb + n.nblk > tb.max_blk ||
      qw + n.nwrp > tb.max_wrp || qg + n.nbig > tb.max_big) {
    atomicOr(err, DERR_TREE_NODES);
    atomicMin(&tb.ctr[kCtrFail], tb.nDepth[p]);
    return false;
  }
  const int4 Ip = tb.nI[p];
  const int depth = tb.nDepth[p] + 1;
  const int lb = depth % 3;
  const double4 P = tb.nP[p];
  const double h = tb.nA[p].w / 2.0;
  int off = 0, k = 0, kb = 0, kw = 0, kg = 0;
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    if (!cnt[d]) continue;
    const int id = id0 + k;
    const bool last = (k == n.nchild - 1);
    const double cx = (d & 1) ? e_add(P.x, h) : P.x;
    const double cz = (d & 2) ? e_add(P.z, h) : P.z;
    const double cy = (d & 4) ? e_add(P.y, h) : P.y;
    tb.nP[id] = make_double4(cx, cy, cz, 0);
    tb.nA[id] = make_double4(0, 0, 0, h);
    tb.nI[id] = make_int4(cnt[d], kEnd, last ? Ip.z : id + 1, 0);
    tb.nR[id] = make_int2(mb0 + off, cnt[d]);
    tb.nDepth[id] = depth;
    tb.nKids[id] = 0;
    if (kList && cnt[d] >= 2) {  // the child's level list of nodes still to split
      if (cnt[d] > kBigNode) tb.split_blk[lb][qb + kb++] = id;
      else tb.split_wrp[lb][qw + kw++] = id;
    }
    if (cnt[d] > kBlockSumNode) tb.bigl[qg + kg++] = id;
    off += cnt[d];
    ++k;
  }
  tb.nI[p].y = id0;
  tb.nKids[p] = n.nchild;
  return true;
}

// Create the non-empty children of node p (counts cnt[0..7]); returns first child id via
// *id0 and member base via *mb0 (or -1 on overflow).  Called by one thread.
template <bool kList = true>
__device__ void make_children(TreeBuffers &tb, int p, const int cnt[8], int *id0_out, int *mb0_out, unsigned *err) {
  *id0_out = *mb0_out = -1;
  const SplitNeeds nd = split_needs<kList>(cnt);
  if (nd.nchild == 0) return;
  // one reservation per counter for the whole node, the atomics issued together
  const int lb = (tb.nDepth[p] + 1) % 3;
  const int id0 = atomicAdd(&tb.ctr[0], nd.nchild);
  const int mb0 = atomicAdd(&tb.ctr[1], nd.kept);
  const int qb = nd.nblk ? atomicAdd(&tb.ctr[kCtrSplit + lb], nd.nblk) : 0;
  const int qw = nd.nwrp ? atomicAdd(&tb.ctr[kCtrSplit + 3 + lb], nd.nwrp) : 0;
  const int qg = nd.nbig ? atomicAdd(&tb.ctr[kCtrBig], nd.nbig) : 0;
  if (!write_children<kList>(tb, p, cnt, nd, id0, mb0, qb, qw, qg, err)) return;
  *id0_out = id0;
  *mb0_out = mb0;
}

// The roots' member lists (the live slots, in slot order) and their split (build_tree at the root,
// tree.f90:66-94), every system at once, by one ordered pass over the slots: list 0 holds the
// live slots, list 1 + d those in octant d of their root's cell.  A slot keeps its octant and
// its rank in that list; the ranks at the systems' first slots (and past the last) tell each
// root's counts.
constexpr unsigned kPassFirst = 1u << 31;  // the slot is a system's first (its dummy)
__global__ void __launch_bounds__(kPassThreads) k_root_lists(const SysConst *__restrict__ scs,
                                                            const SysDyn *__restrict__ dyn,
                                                            const int *__restrict__ sys_of,
                                                            const double *__restrict__ X, const int *__restrict__ nxt,
                                                            TreeBuffers tb, int nsys, long long T, unsigned *err) {
  ordered_pass<9>(
      PassBuffers{tb.pass_state, tb.pass_ctl}, T, err,
      [&](long long gl) -> unsigned {
        if (gl == 0) {
          for (int b = 0; b < 6; ++b) tb.ctr[kCtrSplit + b] = 0;
          tb.ctr[0] = nsys;
          tb.ctr[2] = 0;
          tb.ctr[3] = nsys;
          tb.ctr[kCtrBig] = 0;
          tb.ctr[kCtrFail] = INT_MAX;
        }
        if (gl >= T) return kPassFirst;
        const int g = (int)gl, s = sys_of[g];
        const SysConst &sc = scs[s];
        const int k = g - sc.base;
        int d = 8;
        unsigned f = k == 0 ? kPassFirst : 0u;
        if ((sc.use_tree || sc.sched_tree) && k >= 1 && k <= dyn[s].pcount && nxt[g] != 0) {
          f |= 1u;
          // a point pinned in front (its segment goes into the wall) counts in the root's centre
          // but belongs to no child (new_tree, tree.f90:128)
          if (dyn[s].pcount >= 2 && !(sc.pin && pin_i(sc.pin[g]))) {
            double x[3];
            load_x(X, T, g, x);
            const double h = -sc.bsize / 2.0;
            d = octant(x, make_double4(h, h, h, 0), sc.bsize / 2.0);
            if (d < 8) f |= 2u << d;
          }
        }
        tb.rdig[g] = (unsigned char)d;
        return f;
      },
      [&](long long gl, int k, int p, unsigned word) {
        if (word & kPassFirst) tb.root_rank[9 * (gl < T ? sys_of[gl] : nsys) + k] = p;
        if (k == 0) {
          if (word & 1u) tb.members[p] = (int)gl;
          if (gl == T) tb.ctr[1] = p;
        } else if ((word >> k) & 1u) {
          tb.rrank[gl] = p;
        }
      });
}

// Root of every system (construct_tree, tree.f90:38-59) and its children.
__global__ void k_roots(const SysConst *__restrict__ scs, SysDyn *dyn, int nsys, const int *__restrict__ nxt,
                        TreeBuffers tb, unsigned *err) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const SysConst &sc = scs[s];
  const bool lost = *err & DERR_TIMEOUT;  // the pass before gave up: its ranks say nothing
  const int pc = (sc.use_tree || sc.sched_tree) && !lost ? dyn[s].pcount : 0;
  const double h = -sc.bsize / 2.0;
  const int *r0 = tb.root_rank + 9 * s, *r1 = r0 + 9;  // this system's first slot, the next one's
  tb.nP[s] = make_double4(h, h, h, 0);
  tb.nA[s] = make_double4(0, 0, 0, sc.bsize);
  tb.nB[s] = make_double4(0, 0, 0, 0);
  tb.nI[s] = make_int4(pc, kEnd, kEnd, pc >= 1 ? nxt[sc.base + 1] : 0);
  tb.nR[s] = lost ? make_int2(0, 0) : make_int2(r0[0], r1[0] - r0[0]);
  tb.nDepth[s] = 0;
  tb.nKids[s] = 0;
  tb.nLeaf[s] = pc == 1 ? sc.base + 1 : 0;
  dyn[s].tree_eval = 0;
  dyn[s].tree_tests = 0;
  dyn[s].diag[8] = dyn[s].diag[9] = dyn[s].diag[10] = 0;
  int cnt[8], id0 = -1, mb0 = -1;
  for (int d = 0; d < 8; ++d) cnt[d] = r1[1 + d] - r0[1 + d];
  if (pc >= 2) make_children(tb, s, cnt, &id0, &mb0, err);
  tb.root_ok[s] = mb0 >= 0;
  int off = mb0;
  for (int d = 0; d < 8; ++d) {  // the slot of rank r in octant d is member entry root_mb + r
    tb.root_mb[8 * s + d] = off - r0[1 + d];
    off += cnt[d];
  }
}

// The children's member lists; also notes the block-summed nodes listed so far (depth 1).
__global__ void k_root_scatter(const int *__restrict__ sys_of, TreeBuffers tb, int nsys, const unsigned *err) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p == 0) tb.ctr[kCtrBigSnap] = min(tb.ctr[kCtrBig], tb.max_big);
  if (*err & DERR_TIMEOUT || p >= tb.root_rank[9 * nsys]) return;  // (the live slots of all systems)
  const int g = tb.members[p], d = tb.rdig[g], s = sys_of[g];
  if (d < 8 && tb.root_ok[s]) tb.members[tb.root_mb[8 * s + d] + tb.rrank[g]] = g;
}

// Split node p (at most kBigNode members) with one warp: count the members per octant, make
// the children, then write each member to its child's list in member order (stable).  Each
// lane takes kUnroll members per pass (k0 + 32 u + lane), their loads in flight together.
constexpr int kUnroll = 4;
constexpr int kSplitThreads = 512;

// Octants (8: outside every child, or past `end`) and slots of members k0 + 32 u + lane of
// the list mem[0 .. end).
__device__ __forceinline__ void octants_of(const double *__restrict__ X, long long T, const int *mem, int k0, int end,
                                           int lane, const double4 &P, double h, int d[kUnroll], int slot[kUnroll]) {
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int k = k0 + 32 * u + lane;
    slot[u] = k < end ? mem[k] : -1;
  }
  double x[kUnroll][3];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u)
    if (slot[u] >= 0) load_x(X, T, slot[u], x[u]);
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) d[u] = slot[u] >= 0 ? octant(x[u], P, h) : 8;
}

// Members k0 .. of a pass ranked in member order: the stable position of each in its child's
// list (base_off + run + the lanes before it with the same octant), -1 for none.
__device__ __forceinline__ void rank_and_write(TreeBuffers &tb, int mb0, const int base_off[8], int run[8],
                                               const int d[kUnroll], const int slot[kUnroll], int lane) {
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    int mypos = -1;
#pragma unroll
    for (int dd = 0; dd < 8; ++dd) {
      const unsigned b = __ballot_sync(0xffffffffu, d[u] == dd);
      if (d[u] == dd) mypos = mb0 + base_off[dd] + run[dd] + __popc(b & lt);
      run[dd] += __popc(b);
    }
    if (mypos >= 0) tb.members[mypos] = slot[u];
  }
}

// Node p's member count per octant (the warp's lanes over its member list).
__device__ void warp_count(const double *__restrict__ X, long long T, const TreeBuffers &tb, int p, int lane,
                           int cnt[8]) {
  const int2 R = tb.nR[p];
  const double4 P = tb.nP[p];
  const double h = tb.nA[p].w / 2.0;
  for (int k0 = 0; k0 < R.y; k0 += 32 * kUnroll) {
    int d[kUnroll], slot[kUnroll];
    octants_of(X, T, tb.members + R.x, k0, R.y, lane, P, h, d, slot);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
#pragma unroll
      for (int dd = 0; dd < 8; ++dd) cnt[dd] += __popc(__ballot_sync(0xffffffffu, d[u] == dd));
  }
}

// Node p's members into its children's lists (stable: slot order kept), from member slot mb0.
__device__ void warp_scatter(const double *__restrict__ X, long long T, TreeBuffers &tb, int p, int lane,
                             const int cnt[8], int mb0) {
  const int2 R = tb.nR[p];
  const double4 P = tb.nP[p];
  const double h = tb.nA[p].w / 2.0;
  int base_off[8], run[8];
  {
    int off = 0;
#pragma unroll
    for (int dd = 0; dd < 8; ++dd) {
      base_off[dd] = off;
      off += cnt[dd];
      run[dd] = 0;
    }
  }
  for (int k0 = 0; k0 < R.y; k0 += 32 * kUnroll) {
    int d[kUnroll], slot[kUnroll];
    octants_of(X, T, tb.members + R.x, k0, R.y, lane, P, h, d, slot);
    rank_and_write(tb, mb0, base_off, run, d, slot, lane);
  }
}

// The counters a split reserves from, for children at list level lb.
__device__ __forceinline__ int *split_ctr(TreeBuffers &tb, int c, int lb) {
  return c == 0 ? &tb.ctr[0]
       : c == 1 ? &tb.ctr[1]
       : c == 2 ? &tb.ctr[kCtrSplit + lb]
       : c == 3 ? &tb.ctr[kCtrSplit + 3 + lb]
                : &tb.ctr[kCtrBig];
}

// Node p split by the whole warp: count, lane 0 reserves and writes the children, scatter.
template <bool kList = true>
__device__ void warp_split_one(const double *__restrict__ X, long long T, TreeBuffers &tb, int p, int lane, int lb,
                               unsigned *err) {
  int cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  warp_count(X, T, tb, p, lane, cnt);
  const SplitNeeds nd = split_needs<kList>(cnt);
  int mb0 = -1;
  if (lane == 0 && nd.nchild > 0) {
    const int v[5] = {nd.nchild, nd.kept, nd.nblk, nd.nwrp, nd.nbig};
    int base[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) base[c] = v[c] ? atomicAdd(split_ctr(tb, c, lb), v[c]) : 0;
    if (write_children<kList>(tb, p, cnt, nd, base[0], base[1], base[2], base[3], base[4], err)) mb0 = base[1];
  }
  mb0 = __shfl_sync(0xffffffffu, mb0, 0);
  if (mb0 >= 0) warp_scatter(X, T, tb, p, lane, cnt, mb0);
}

// Nodes with at most kLaneNode members, when a level lists many (the deep levels), are split
// by one lane each: the lane counts its node's members per octant (digits kept, 4 bits a
// member), the warp makes one reservation per counter for its lanes' nodes, and each lane
// writes its children and scatters its members in member order.
constexpr int kLaneNode = 16;

template <bool kList = true>
__device__ void lane_split(const double *__restrict__ X, long long T, TreeBuffers &tb, int p, int2 R, int lane,
                           int lb, unsigned *err) {
  const bool mine = p >= 0;
  int cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  unsigned long long digs = 0;
  if (mine) {
    const double4 P = tb.nP[p];
    const double h = tb.nA[p].w / 2.0;
    unsigned long long cp = 0;  // eight counts of 5 bits
    for (int k = 0; k < R.y; ++k) {
      double x[3];
      load_x(X, T, tb.members[R.x + k], x);
      const int d = octant(x, P, h);
      digs |= (unsigned long long)d << (4 * k);
      if (d < 8) cp += 1ull << (5 * d);
    }
#pragma unroll
    for (int dd = 0; dd < 8; ++dd) cnt[dd] = (int)((cp >> (5 * dd)) & 31u);
  }
  const SplitNeeds nd = mine ? split_needs<kList>(cnt) : SplitNeeds{0, 0, 0, 0, 0};
  const int v[5] = {nd.nchild, nd.kept, nd.nblk, nd.nwrp, nd.nbig};
  int off[5], base[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) {  // exclusive prefix over the lanes, the total in lane 31
    int x = v[c];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    off[c] = x - v[c];
    base[c] = 0;
    if (lane == 31 && x) base[c] = atomicAdd(split_ctr(tb, c, lb), x);
    base[c] = __shfl_sync(0xffffffffu, base[c], 31);
  }
  if (!mine || nd.nchild == 0) return;
  const int mb0 = base[1] + off[1];
  if (!write_children<kList>(tb, p, cnt, nd, base[0] + off[0], mb0, base[2] + off[2], base[3] + off[3], base[4] + off[4],
                      err))
    return;
  unsigned long long op = 0, run = 0;  // children's list offsets and fill, 5 bits each
  int o = 0;
#pragma unroll
  for (int dd = 0; dd < 8; ++dd) {
    op |= (unsigned long long)o << (5 * dd);
    o += cnt[dd];
  }
  for (int k = 0; k < R.y; ++k) {
    const int d = (int)((digs >> (4 * k)) & 15u);
    if (d < 8) {
      const int at = (int)(((op >> (5 * d)) & 31u) + ((run >> (5 * d)) & 31u));
      run += 1ull << (5 * d);
      tb.members[mb0 + at] = tb.members[R.x + k];
    }
  }
}

// Split node p (more than kBigNode members) with a whole block: each warp takes a contiguous
// slice of the member list and the slices' counts are prefix-summed, so the partition stays
// stable.
template <bool kList = true>
__device__ void split_node_block(const double *__restrict__ X, long long T, TreeBuffers &tb, int p,
                                 unsigned *err) {
  __shared__ int wcnt[32][8];
  __shared__ int s_id0, s_mb0, s_cnt[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int2 R = tb.nR[p];
  const double4 P = tb.nP[p];
  const double h = tb.nA[p].w / 2.0;
  const int per = (R.y + nw - 1) / nw;
  const int s0 = w * per, s1 = min(R.y, s0 + per);
  int cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k0 = s0; k0 < s1; k0 += 32 * kUnroll) {
    int d[kUnroll], slot[kUnroll];
    octants_of(X, T, tb.members + R.x, k0, s1, lane, P, h, d, slot);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
#pragma unroll
      for (int dd = 0; dd < 8; ++dd) cnt[dd] += __popc(__ballot_sync(0xffffffffu, d[u] == dd));
  }
  if (lane == 0)
#pragma unroll
    for (int dd = 0; dd < 8; ++dd) wcnt[w][dd] = cnt[dd];
  __syncthreads();
  if (threadIdx.x < 8) {
    int tot = 0;
    for (int ww = 0; ww < nw; ++ww) {
      const int c = wcnt[ww][threadIdx.x];
      wcnt[ww][threadIdx.x] = tot;  // exclusive prefix over warps
      tot += c;
    }
    s_cnt[threadIdx.x] = tot;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int c[8];
    for (int dd = 0; dd < 8; ++dd) c[dd] = s_cnt[dd];
    int id0, mb0;
    make_children<kList>(tb, p, c, &id0, &mb0, err);
    s_id0 = id0;
    s_mb0 = mb0;
  }
  __syncthreads();
  const int mb0 = s_mb0;
  if (s_id0 >= 0) {
    int base_off[8], run[8];
    int off = 0;
#pragma unroll
    for (int dd = 0; dd < 8; ++dd) {
      base_off[dd] = off + wcnt[w][dd];
      off += s_cnt[dd];
      run[dd] = 0;
    }
    for (int k0 = s0; k0 < s1; k0 += 32 * kUnroll) {
      int d[kUnroll], slot[kUnroll];
      octants_of(X, T, tb.members + R.x, k0, s1, lane, P, h, d, slot);
      rank_and_write(tb, mb0, base_off, run, d, slot, lane);
    }
  }
}

// One level of the build: the listed big nodes by blocks, then the other listed nodes by
// warps.  One block of kSplitThreads per SM, with registers for the loads of several
// members (or nodes) per lane in flight at once.  The children's lists (level + 1) fill as nodes
// split; the list of level + 2 is idle during this level (read at level - 1, filled at
// level + 1) and is emptied here.
__global__ void __launch_bounds__(kSplitThreads, 1) k_split_level(const double *__restrict__ X, long long T, TreeBuffers tb,
                                                      int level, unsigned *err) {
  if (failed_above(tb, level)) return;
  const int block = blockIdx.x, blocks = gridDim.x;
  const int b = level % 3, b2 = (level + 2) % 3;
  if (block == 0 && threadIdx.x == 0) {
    tb.ctr[kCtrSplit + b2] = 0;
    tb.ctr[kCtrSplit + 3 + b2] = 0;
  }
  const int nbl = min(tb.ctr[kCtrSplit + b], tb.max_blk);
  for (int bq = block; bq < nbl; bq += blocks) {
    const int p = tb.split_blk[b][bq];
    if (tb.nDepth[p] >= kMaxLevels) {
      if (threadIdx.x == 0) atomicOr(err, DERR_TREE_DEPTH);
      continue;
    }
    split_node_block(X, T, tb, p, err);
    __syncthreads();
  }
  // The other listed nodes by warps.  Where they outnumber the warps twice over (the small,
  // numerous nodes of the deep levels) a warp takes an equal share of them, up to 32: each
  // lane splits its own when it has at most kLaneNode members, and the warp the larger ones
  // one at a time; elsewhere a warp splits one node at a time.
  const int lane = threadIdx.x & 31;
  const int warp = (block * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (blocks * blockDim.x) >> 5;
  const int nwl = min(tb.ctr[kCtrSplit + 3 + b], tb.max_wrp);
  const int lb = (level + 1) % 3;  // the children's level lists
  if (nwl >= 2 * nwarps) {
    const int per = min(32, (nwl + nwarps - 1) / nwarps);  // nodes per warp: every warp busy
    for (int wq0 = warp * per; wq0 < nwl; wq0 += nwarps * per) {
      int p = lane < per && wq0 + lane < nwl ? tb.split_wrp[b][wq0 + lane] : -1;
      if (p >= 0 && tb.nDepth[p] >= kMaxLevels) {
        atomicOr(err, DERR_TREE_DEPTH);
        p = -1;
      }
      const int2 R = p >= 0 ? tb.nR[p] : make_int2(0, 0);
      const bool small = p >= 0 && R.y <= kLaneNode;
      lane_split(X, T, tb, small ? p : -1, R, lane, lb, err);
      for (unsigned big = __ballot_sync(0xffffffffu, p >= 0 && !small); big; big &= big - 1) {
        const int pp = __shfl_sync(0xffffffffu, p, __ffs(big) - 1);
        warp_split_one(X, T, tb, pp, lane, lb, err);
      }
    }
  } else {
    for (int wq = warp; wq < nwl; wq += nwarps) {
      const int p = tb.split_wrp[b][wq];
      if (tb.nDepth[p] >= kMaxLevels) {
        if (lane == 0) atomicOr(err, DERR_TREE_DEPTH);
        continue;
      }
      warp_split_one(X, T, tb, p, lane, lb, err);
    }
  }
}

// Below cells a fraction of a segment wide only pairs of points from different filaments are left
// together, as a rule: a few nodes a level.  There the nodes listed at `level` are shared out over
// the blocks, and a block splits its share with all that lies below, level after level by lists in
// shared memory: nothing is waited for outside the block, and a state whose points lie closer
// than its delta, with as many nodes here as on the levels before, still has the whole GPU.
constexpr int kRestMembers = 8192;  // of the nodes that a block takes at once
struct RestShared {
  int list[2][kRestMembers / 2];  // nodes of this level and of the next (two members at least each)
  int n, warp_sum[kSplitThreads / 32], big[7 * kMaxLevels + 8], n_big;
};

// The subtrees of the n nodes in S.list[0] (kRestMembers members together at most, kBigNode each), by the
// block: a lane per node up to kLaneNode members, a warp above that.
__device__ void split_below(const double *__restrict__ X, long long T, TreeBuffers &tb, int n, RestShared &S,
                            unsigned *err) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int cur = 0; n > 0; cur ^= 1) {
    if (threadIdx.x == 0) S.n = 0;
    __syncthreads();
    const int per = min(32, (n + nwarps - 1) / nwarps);
    for (int q0 = wid * per; q0 < n; q0 += nwarps * per) {
      int p = lane < per && q0 + lane < n ? S.list[cur][q0 + lane] : -1;
      if (p >= 0 && tb.nDepth[p] >= kMaxLevels) {
        atomicOr(err, DERR_TREE_DEPTH);
        p = -1;
      }
      const int2 R = p >= 0 ? tb.nR[p] : make_int2(0, 0);
      lane_split<false>(X, T, tb, R.y <= kLaneNode ? p : -1, R, lane, 0, err);
      for (unsigned large = __ballot_sync(0xffffffffu, R.y > kLaneNode); large; large &= large - 1)
        warp_split_one<false>(X, T, tb, __shfl_sync(0xffffffffu, p, __ffs(large) - 1), lane, 0, err);
      __syncwarp();
      if (p >= 0) {
        const int kids = tb.nKids[p], id = tb.nI[p].y;
        for (int c = 0; c < kids; ++c)
          if (tb.nR[id + c].y >= 2) S.list[cur ^ 1][atomicAdd(&S.n, 1)] = id + c;
      }
    }
    __syncthreads();
    n = S.n;
    __syncthreads();
  }
}

// Up to blockDim.x nodes behind the n in S.list[0], as many as keep their members below kRestMembers
// (the first in any case, when the list is empty); returns how many, and adds to n and members.
__device__ int take_nodes(const TreeBuffers &tb, const int *nodes, int count, int &n, int &members, RestShared &S) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int p = tid < count ? nodes[tid] : -1, m = p >= 0 ? tb.nR[p].y : 0;
  int incl = m;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) S.warp_sum[wid] = incl;
  __syncthreads();
  for (int w = 0; w < wid; ++w) incl += S.warp_sum[w];
  const bool fits = p >= 0 && members + incl <= kRestMembers;
  if (fits) S.list[0][n + tid] = p;
  const int took = __syncthreads_count(fits);
  if (tid == took - 1) S.n = incl;
  __syncthreads();
  n += took;
  if (took) members += S.n;
  __syncthreads();
  return took;
}

// The subtree of node p (more than kBigNode members) by the block: its own splits one after the other,
// and below the other children.
__device__ void split_below_big(const double *__restrict__ X, long long T, TreeBuffers &tb, int p, RestShared &S,
                                unsigned *err) {
  __syncthreads();  // (every thread has left the last node's loop)
  if (threadIdx.x == 0) {
    S.big[0] = p;
    S.n_big = 1;
  }
  __syncthreads();
  while (S.n_big > 0) {
    p = S.big[S.n_big - 1];
    __syncthreads();
    if (threadIdx.x == 0) --S.n_big;
    int kids = 0, id = 0;
    if (tb.nDepth[p] >= kMaxLevels) {
      if (threadIdx.x == 0) atomicOr(err, DERR_TREE_DEPTH);
    } else {
      split_node_block<false>(X, T, tb, p, err);
      __syncthreads();
      kids = tb.nKids[p];
      id = tb.nI[p].y;
    }
    for (int c0 = 0; c0 < kids; c0 += kRestMembers / kBigNode) {
      if (threadIdx.x == 0) {
        S.n = 0;
        for (int c = c0; c < min(kids, c0 + kRestMembers / kBigNode); ++c) {
          const int m = tb.nR[id + c].y;
          if (m > kBigNode) S.big[S.n_big++] = id + c;
          else if (m >= 2) S.list[0][S.n++] = id + c;
        }
      }
      __syncthreads();
      const int n = S.n;
      __syncthreads();
      split_below(X, T, tb, n, S, err);
    }
    __syncthreads();
  }
}

// The nodes listed at `level` with all below them: 32,768 points 2.8 us, 1,048,576 points 22 us (by one
// block, level after level, 1.5 and 36 us; but with 1,048,576 points at a delta of 40 segments the
// tree stage took 15.2 ms so, 5.6 now and with a launch for every level; one ring of 300,000
// points, a segment's width 1,600 times theirs: 1.35 ms, 1.52 with a launch for every level, 2.10
// with each subtree by the warp that takes its root).
__global__ void __launch_bounds__(kSplitThreads, 1) k_split_rest(const double *__restrict__ X, long long T, TreeBuffers tb,
                                                     int level, unsigned *err) {
  __shared__ RestShared S;
  if (failed_above(tb, level)) return;
  const int b = level % 3;
  const int nbl = min(tb.ctr[kCtrSplit + b], tb.max_blk), nwl = min(tb.ctr[kCtrSplit + 3 + b], tb.max_wrp);
  for (int bq = blockIdx.x; bq < nbl; bq += gridDim.x) split_below_big(X, T, tb, tb.split_blk[b][bq], S, err);
  int i = (int)((long long)nwl * blockIdx.x / gridDim.x);
  const int end = (int)((long long)nwl * (blockIdx.x + 1) / gridDim.x);
  while (i < end) {
    int n = 0, members = 0;
    for (;;) {
      const int count = min((int)blockDim.x, end - i);
      const int took = take_nodes(tb, tb.split_wrp[b] + i, count, n, members, S);
      i += took;
      if (took < count || i == end) break;
    }
    split_below(X, T, tb, n, S, err);
  }
}

// Centre and circulation of every node: sequential sums in ascending slot order
// (new_tree, tree.f90:124-152; the root's masked mean, tree.f90:50-54), plus the
// geometric distance of the opening test's correction (tree.f90:267-269).
constexpr int kSmallNode = 16;  // nodes up to this many members are summed by one thread

__device__ __forceinline__ void finish_node(TreeBuffers &tb, int id, bool root, double cx, double cy, double cz,
                                            double qx, double qy, double qz, const int *__restrict__ nxt,
                                            unsigned *err) {
  const int2 R = tb.nR[id];
  int4 I = tb.nI[id];
  const double4 P = tb.nP[id];
  const double w = tb.nA[id].w;
  if (R.y != 0) {
    cx = e_div(cx, (double)R.y);
    cy = e_div(cy, (double)R.y);
    cz = e_div(cz, (double)R.y);
  }
  const double hw = w / 2.;
  const double geo = e_sqrt(e_add(e_add(e_sq(e_sub(cx, e_add(P.x, hw))), e_sq(e_sub(cy, e_add(P.y, hw)))),
                                   e_sq(e_sub(cz, e_add(P.z, hw)))));
  // the centre only: the width (nA.w) is not written, since the split of this node may be
  // reading it at the same time (the depth-1 nodes are summed beside the level-1 split)
  double *a = reinterpret_cast<double *>(&tb.nA[id]);
  a[0] = cx;
  a[1] = cy;
  a[2] = cz;
  tb.nB[id] = make_double4(qx, qy, qz, geo);
  if (!root) {
    const int first = R.y > 0 ? tb.members[R.x] : 0;
    I.w = first ? nxt[first] : 0;
    tb.nI[id].w = I.w;  // the node's other links belong to the splits
    tb.nLeaf[id] = I.x == 1 ? first : 0;
    if (tb.nDepth[id] >= kMaxLevels && I.x > 1) atomicOr(err, DERR_TREE_DEPTH);
  }
}

// Nodes with at most kSmallNode members (most of them leaves): one thread each.
__global__ void k_node_sums_small(const double *__restrict__ X, const double *__restrict__ GI,
                                  const int *__restrict__ nxt, long long T, TreeBuffers tb, int nsys, unsigned *err) {
  if (failed_above(tb, INT_MAX)) return;
  const int n = tb.ctr[0];
  for (int id = nsys + blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
    const int2 R = tb.nR[id];
    if (R.y > kSmallNode) continue;
    const bool root = false;
    double cx = 0, cy = 0, cz = 0, qx = 0, qy = 0, qz = 0;
    for (int k = 0; k < R.y; ++k) {
      const int g = tb.members[R.x + k];
      const double x0 = __ldg(X + g), x1 = __ldg(X + T + g), x2 = __ldg(X + 2 * T + g);
      cx = e_add(cx, x0);
      cy = e_add(cy, x1);
      cz = e_add(cz, x2);
      if (!root) {
        qx = e_sub(e_add(qx, __ldg(GI + g)), x0);
        qy = e_sub(e_add(qy, __ldg(GI + T + g)), x1);
        qz = e_sub(e_add(qz, __ldg(GI + 2 * T + g)), x2);
      }
    }
    finish_node(tb, id, root, cx, cy, cz, qx, qy, qz, nxt, err);
  }
}

// Sequential sums of one node by one warp: the warp gathers 32 members' coordinates and
// ghosts (coalesced member reads) into shared memory; lanes 0-2 then add the three centre
// components and lanes 3-5 the three circulation components, each in ascending member order
// -- the reference loop's sequence of roundings.  A lane first moves its 32 operands into
// registers and then runs the dependent additions unrolled, so the chain proceeds at the
// latency of the additions alone; the next tile's loads are issued before them.
constexpr int kTilePad = 33;  // row stride: lanes 0-5 reading one column hit distinct banks

__device__ __forceinline__ void warp_node_sums(const double *__restrict__ X, const double *__restrict__ GI,
                                               long long T, const int *__restrict__ mem, int count, bool circ,
                                               double (*buf)[kTilePad], int lane, double &acc) {
  acc = 0;
  double v[6];
  auto gather = [&](int k0) {
    const int k = k0 + lane;
    if (k < count) {
      const int g = mem[k];
      v[0] = __ldg(X + g);
      v[1] = __ldg(X + T + g);
      v[2] = __ldg(X + 2 * T + g);
      if (circ) {
        v[3] = __ldg(GI + g);
        v[4] = __ldg(GI + T + g);
        v[5] = __ldg(GI + 2 * T + g);
      }
    }
  };
  gather(0);
  for (int k0 = 0; k0 < count; k0 += 32) {
    __syncwarp();
    if (k0 + lane < count) {
#pragma unroll
      for (int c = 0; c < 3; ++c) buf[c][lane] = v[c];
      if (circ)
#pragma unroll
        for (int c = 3; c < 6; ++c) buf[c][lane] = v[c];
    }
    __syncwarp();
    if (k0 + 32 < count) gather(k0 + 32);
    const int cnt = min(32, count - k0);
    // centre lanes 0-2: acc + x; circulation lanes 3-5: (acc + gi) - x.  With circulations
    // the centre lanes subtract +0 (which returns its operand, -0 included), so that the six
    // chains run as one instruction stream instead of two divergent ones in turn
    const int ncomp = circ ? 6 : 3;
    const bool sub = lane >= 3;
    const double *a = buf[lane < 6 ? lane : 0], *bq = buf[sub && lane < 6 ? lane - 3 : 0];
    if (lane < ncomp) {
      if (!circ) {
        for (int l = 0; l < cnt; ++l) acc = e_add(acc, a[l]);
      } else if (cnt == 32) {
        double r[32], q[32];
#pragma unroll
        for (int l = 0; l < 32; ++l) {
          r[l] = a[l];
          const double x = bq[l];
          q[l] = sub ? x : 0.0;
        }
#pragma unroll
        for (int l = 0; l < 32; ++l) acc = e_sub(e_add(acc, r[l]), q[l]);
      } else {
        for (int l = 0; l < cnt; ++l) {
          const double x = bq[l];
          acc = e_sub(e_add(acc, a[l]), sub ? x : 0.0);
        }
      }
    }
  }
}

// Nodes (roots excepted) with kSmallNode < members <= kBlockSumNode: one warp each.
__global__ void __launch_bounds__(128) k_node_sums_big(const double *__restrict__ X, const double *__restrict__ GI,
                                                       const int *__restrict__ nxt, long long T, TreeBuffers tb,
                                                       int nsys, unsigned *err) {
  __shared__ double sm[4][6][kTilePad];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  if (failed_above(tb, INT_MAX)) return;
  const int n = tb.ctr[0];
  // The warp's nodes are ids nsys + warp + j nwarps (consecutive ids, often one level's
  // nodes of similar size, go to different warps); their records are read 32 at a time and
  // the ones in this kernel's size range summed in turn.
  for (long long j0 = 0; nsys + warp + j0 * nwarps < n; j0 += 32) {
    const long long idl = nsys + warp + (j0 + lane) * nwarps;
    const int2 Rl = idl < n ? tb.nR[idl] : make_int2(0, 0);
    for (unsigned m = __ballot_sync(0xffffffffu, Rl.y > kSmallNode && Rl.y <= kBlockSumNode); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const int2 R = make_int2(__shfl_sync(0xffffffffu, Rl.x, l), __shfl_sync(0xffffffffu, Rl.y, l));
      double acc;
      warp_node_sums(X, GI, T, tb.members + R.x, R.y, true, sm[wl], lane, acc);
      const double cx = __shfl_sync(0xffffffffu, acc, 0), cy = __shfl_sync(0xffffffffu, acc, 1),
                   cz = __shfl_sync(0xffffffffu, acc, 2), qx = __shfl_sync(0xffffffffu, acc, 3),
                   qy = __shfl_sync(0xffffffffu, acc, 4), qz = __shfl_sync(0xffffffffu, acc, 5);
      if (lane == 0) finish_node(tb, (int)(nsys + warp + (j0 + l) * nwarps), false, cx, cy, cz, qx, qy, qz, nxt, err);
    }
  }
}

// Sequential sums of one large node by a block: warps 1.. stream member tiles into a ring of
// kSumDepth shared-memory tiles with 8-byte cp.async copies, kSumDepth - 1 tiles ahead of
// warp 0, whose lanes 0-2 (centre) and 3-5 (circulation) add each tile in member order.
constexpr int kSumTile = 512, kSumDepth = 4, kSumThreads = 256;
constexpr int kSumRow = kSumTile + 1;  // padded: lanes 0-5 reading one column hit distinct banks
constexpr size_t kSumSmem = (size_t)kSumDepth * 6 * kSumRow * sizeof(double);

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_depth() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kSumDepth - 2) : "memory");
}

__device__ void block_node_sums(const double *__restrict__ X, const double *__restrict__ GI, long long T,
                                const int *__restrict__ mem, int count, bool circ, double *sm, double &acc) {
  const int tid = threadIdx.x, lane = tid & 31;
  const bool producer = tid >= 32;
  const int ptid = tid - 32, np = kSumThreads - 32;
  const int ntiles = (count + kSumTile - 1) / kSumTile;
  const int ncomp = circ ? 6 : 3;
  auto issue = [&](int t) {  // producers: copies of tile t into its ring slot
    if (t < ntiles) {
      double *slot = sm + (size_t)(t % kSumDepth) * 6 * kSumRow;
      for (int e = ptid; e < kSumTile; e += np) {
        const int k = t * kSumTile + e;
        if (k >= count) break;
        const int g = mem[k];
        cp_async8(slot + e, X + g);
        cp_async8(slot + kSumRow + e, X + T + g);
        cp_async8(slot + 2 * kSumRow + e, X + 2 * T + g);
        if (circ) {
          cp_async8(slot + 3 * kSumRow + e, GI + g);
          cp_async8(slot + 4 * kSumRow + e, GI + T + g);
          cp_async8(slot + 5 * kSumRow + e, GI + 2 * T + g);
        }
      }
    }
    cp_async_commit();  // one group per tile, empty or not, so that the wait counts line up
  };
  acc = 0;
  if (producer) {
    for (int t = 0; t < kSumDepth - 1; ++t) issue(t);
    cp_async_wait_depth();  // tile 0 has landed
  }
  __syncthreads();
  for (int t = 0; t < ntiles; ++t) {
    if (producer) {
      issue(t + kSumDepth - 1);  // into the slot consumed in the previous round
      cp_async_wait_depth();     // tile t + 1 has landed
    } else if (lane < ncomp) {
      const double *slot = sm + (size_t)(t % kSumDepth) * 6 * kSumRow;
      // as in warp_node_sums: with circulations the centre lanes subtract +0, one stream
      const bool sub = lane >= 3;
      const double *a = slot + lane * kSumRow;
      const double *b = slot + (sub ? lane - 3 : 0) * kSumRow;
      const int cnt = min(kSumTile, count - t * kSumTile);
      if (!circ) {
        if (cnt == kSumTile) {
          for (int e0 = 0; e0 < kSumTile; e0 += 32) {
            double r[32];
#pragma unroll
            for (int l = 0; l < 32; ++l) r[l] = a[e0 + l];
#pragma unroll
            for (int l = 0; l < 32; ++l) acc = e_add(acc, r[l]);
          }
        } else {
          for (int l = 0; l < cnt; ++l) acc = e_add(acc, a[l]);
        }
      } else if (cnt == kSumTile) {
        for (int e0 = 0; e0 < kSumTile; e0 += 32) {
          double r[32], q[32];
#pragma unroll
          for (int l = 0; l < 32; ++l) {
            r[l] = a[e0 + l];
            const double x = b[e0 + l];
            q[l] = sub ? x : 0.0;
          }
#pragma unroll
          for (int l = 0; l < 32; ++l) acc = e_sub(e_add(acc, r[l]), q[l]);
        }
      } else {
        for (int l = 0; l < cnt; ++l) {
          const double x = b[l];
          acc = e_sub(e_add(acc, a[l]), sub ? x : 0.0);
        }
      }
    }
    __syncthreads();
  }
  if (producer) asm volatile("cp.async.wait_all;" ::: "memory");
}

// Non-root nodes with more than kBlockSumNode members (listed by the splits): one block each.
__global__ void __launch_bounds__(kSumThreads) k_node_sums_block(const double *__restrict__ X,
                                                                  const double *__restrict__ GI,
                                                                  const int *__restrict__ nxt, long long T,
                                                                  TreeBuffers tb, int part, unsigned *err) {
  // part 0: the big depth-1 nodes, listed by the roots' split (their member lists final),
  // summed beside the level splits (which read their width and write their first child,
  // fields the sums leave alone); part 1, after the levels: every other big node
  extern __shared__ double sm_dyn[];
  if (failed_above(tb, part == 0 ? 1 : INT_MAX)) return;
  const int snap = tb.ctr[kCtrBigSnap];
  const int nbig = part == 0 ? snap : min(tb.ctr[kCtrBig], tb.max_big);
  for (int b = blockIdx.x; b < nbig; b += gridDim.x) {
    const int id = tb.bigl[b];
    const bool early = b < snap && tb.nDepth[id] <= kSnapLevel;
    if (early != (part == 0)) continue;  // block-uniform
    const int2 R = tb.nR[id];
    double acc;
    block_node_sums(X, GI, T, tb.members + R.x, R.y, true, sm_dyn, acc);
    const double cx = __shfl_sync(0xffffffffu, acc, 0), cy = __shfl_sync(0xffffffffu, acc, 1),
                 cz = __shfl_sync(0xffffffffu, acc, 2), qx = __shfl_sync(0xffffffffu, acc, 3),
                 qy = __shfl_sync(0xffffffffu, acc, 4), qz = __shfl_sync(0xffffffffu, acc, 5);
    if (threadIdx.x == 0) finish_node(tb, id, false, cx, cy, cz, qx, qy, qz, nxt, err);
    __syncthreads();
  }
}

// Roots: the masked mean over live slots (tree.f90:50-54), circulation zero.  One block per
// system; launched beside the level splits (it reads only the root's member list, which
// the splits do not change).
__global__ void __launch_bounds__(kSumThreads) k_root_sums(const double *__restrict__ X, long long T,
                                                            TreeBuffers tb, int nsys, const int *__restrict__ nxt,
                                                            unsigned *err) {
  extern __shared__ double sm_dyn[];
  const int id = blockIdx.x;
  if (id >= nsys) return;
  const int2 R = tb.nR[id];
  double acc;
  block_node_sums(X, nullptr, T, tb.members + R.x, R.y, false, sm_dyn, acc);
  const double cx = __shfl_sync(0xffffffffu, acc, 0), cy = __shfl_sync(0xffffffffu, acc, 1),
               cz = __shfl_sync(0xffffffffu, acc, 2);
  if (threadIdx.x == 0) finish_node(tb, id, true, cx, cy, cz, 0.0, 0.0, 0.0, nxt, err);
}

// Estimate of each root's centre (the mean over live slots, tree.f90:50-52) by a blocked
// sum over `parts` blocks per system (k_root_partial, then k_root_approx adding the parts), and
// a bound on its distance to the reference's sequential sum: a sum of N terms in FP64 is within (N-1) u sum|x| of the exact one in either order, so the two means
// differ by at most 2 u (sum|x| + sum|y| + sum|z|) plus the roundings of the divisions.
__global__ void __launch_bounds__(256) k_root_partial(const double *__restrict__ X, long long T, TreeBuffers tb,
                                                      int nsys, int parts) {
  __shared__ double red[6][8];
  const int s = blockIdx.x / parts, part = blockIdx.x % parts;
  if (s >= nsys) return;
  const int2 R = tb.nR[s];
  const int per = (R.y + parts - 1) / parts;
  const int k0 = part * per, k1 = min(R.y, k0 + per);
  const int *mem = tb.members + R.x;
  double a[6] = {0, 0, 0, 0, 0, 0};
  for (int k = k0 + (int)threadIdx.x; k < k1; k += blockDim.x) {
    const int g = mem[k];
    for (int c = 0; c < 3; ++c) {
      const double v = __ldg(X + c * T + g);
      a[c] += v;
      a[3 + c] += fabs(v);
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c = 0; c < 6; ++c) {
    double v = a[c];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[c][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
    tb.root_part[(long long)blockIdx.x * 6 + threadIdx.x] = t;
  }
}

__global__ void k_root_approx(TreeBuffers tb, int nsys, int parts, double band_scale) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= nsys) return;
  double t[6] = {0, 0, 0, 0, 0, 0};
  for (int q = lane; q < parts; q += 32)
    for (int c = 0; c < 6; ++c) t[c] += tb.root_part[((long long)s * parts + q) * 6 + c];
  for (int c = 0; c < 6; ++c)
    for (int o = 16; o > 0; o >>= 1) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
  if (lane) return;
  const int n = tb.nR[s].y;
  const double dn = n > 0 ? (double)n : 1.0;
  const double cx = t[0] / dn, cy = t[1] / dn, cz = t[2] / dn;
  const double u = 1.2e-16;
  const double bound =
      band_scale * (2.0 * u * (t[3] + t[4] + t[5]) + 8.0 * u * (fabs(cx) + fabs(cy) + fabs(cz)) + 1e-300);
  tb.root_apx[s] = n > 0 ? make_double4(cx, cy, cz, bound) : make_double4(0, 0, 0, 0);
}

// The opening test of root `root` (tree.f90:264-278) for target xi and image shift s from
// the centre estimate: 0 the root is opened, 1 it is accepted (its circulation is zero, so
// the image adds nothing), 2 the estimate cannot tell.  The root's box is centred on the
// origin (corner -bsize/2, width bsize), so geo = |centre|.
__device__ __forceinline__ int root_decision(const TreeBuffers &tb, const SysConst &sc, int root, const double xi[3],
                                             const double s[3]) {
  const int4 I = tb.nI[root];
  if (I.x <= 1) return 2;  // empty or single-slot root: the exact path handles it
  if (sc.tree_extra_correction && sc.tree_theta > 1.1547) return 2;  // dist <= geo branch
  const double4 R = tb.root_apx[root];
  const double d0 = xi[0] - (R.x + s[0]), d1 = xi[1] - (R.y + s[1]), d2 = xi[2] - (R.z + s[2]);
  const double dist = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
  const double thr = sc.bsize / sc.tree_theta;
  double margin = dist - thr, pert = R.w;
  if (sc.tree_extra_correction) {
    margin -= sqrt(R.x * R.x + R.y * R.y + R.z * R.z);
    pert *= 2.0;
  }
  pert += 1e-12 * (dist + thr);
  if (margin > pert) return 1;
  if (margin < -pert) return 0;
  return 2;
}

__device__ __forceinline__ void defer_push(const TreeBuffers &tb, int g, unsigned *err) {
  const int q = atomicAdd(tb.defer_n, 1);
  if (q < kDeferCap) tb.defer[q] = g;
  else atomicOr(err, DERR_QUEUE);
}

// The opening test of a node (tree.f90:264-278) and the term of an accepted one (:289-308) in
// the reference's own operations, for the rare node whose squared distance lies within 1e-12 of
// the threshold's square, or whose operands lie outside the range of fp64.cuh's seeds.
__device__ __noinline__ bool accept_exact(double d2, double w, double geo, double theta0, bool corr) {
  const double dist = e_sqrt(d2);
  const double dg = corr ? e_sub(dist, geo) : dist;
  return (dg > 0. ? e_div(w, dg) : e_div(w, dist)) < theta0;
}
__device__ __noinline__ double3 node_term_exact(double v0, double v1, double v2, double c0, double c1, double c2,
                                                double dist, double qc, double two_pi) {
  const double vect[3] = {v0, v1, v2}, circ[3] = {c0, c1, c2};
  const double a = e_mul(dist, dist), b = e_mul(2.0, dot3(vect, circ)), c = dot3(circ, circ);
  const double D = term_d(a, b, c);
  double cr[3];
  cross3(vect, circ, cr);
  const double den = e_mul(two_pi, D);
  const double fac = e_sub(e_div(e_add(e_mul(2.0, c), b), e_sqrt(e_add(e_add(a, b), c))), e_div(b, e_sqrt(a)));
  return make_double3(e_mul(e_div(e_mul(cr[0], qc), den), fac), e_mul(e_div(e_mul(cr[1], qc), den), fac),
                      e_mul(e_div(e_mul(cr[2], qc), den), fac));
}

// tree_walk (tree.f90:250-316) for one image; accumulates into acc in preorder.
// `start` is the root, or the root's first child when the root is already known to be
// opened (its test then counted by the caller).
//
// Six of seven nodes visited are accepted, so the walk is a chain of loads, one distance and a
// term: the record of the node after this one's subtree is requested before this node is
// tested, and the test compares squares (no root, no quotient for an opened node; a band of
// 1e-12, far above the rounding of either form, goes to the reference's own test).  The
// distance's root serves the term too: sqrt(a) with a = dist*dist rounded is dist itself.
// 100,000 points: 4.40 ms, 32,768: 1.52 ms (6.95 and 2.48 ms with the IEEE operations one by one
// and no request ahead).  A lane per (target, sum) in blocks of their own, so that no sum waits
// for the other: 4.87 and 1.82 ms (the two sums of a block share their nodes in L1).
__device__ __forceinline__ void walk_fp64(const TreeBuffers &tb, int start, const SysConst &sc, const double xi[3],
                                          int gi_, int pi_, const int *__restrict__ prv, const double s[3], bool unshifted,
                                          double acc[3], unsigned long long &evals, unsigned long long &tests,
                                          bool &singular, bool &overrun) {
  if (start == kEnd) return;
  const double qc = sc.quant_circ, two_pi = sc.two_pi, theta0 = sc.tree_theta, inv_theta = 1.0 / sc.tree_theta;
  const bool corr = sc.tree_extra_correction;
  // (theta above 2/sqrt(3) with the correction: a node closer than its centre's offset can be
  // accepted, which no single threshold tells)
  const bool square = !(corr && theta0 > 1.1547);
  int node = start;
  int left = tb.ctr[0];  // a walk of a well-formed tree visits each node at most once
  unsigned ev = 0, te = 0;
  double4 A = ldg4(&tb.nA[node]), B = ldg4(&tb.nB[node]);
  int4 I = __ldg(&tb.nI[node]);
  for (;;) {
    if (--left < 0) {
      overrun = true;
      break;
    }
    const int nz = I.z;
    double4 An = make_double4(0, 0, 0, 0), Bn = An;
    int4 In = make_int4(0, kEnd, kEnd, 0);
    if (nz != kEnd) {
      An = ldg4(&tb.nA[nz]);
      Bn = ldg4(&tb.nB[nz]);
      In = __ldg(&tb.nI[nz]);
    }
    int next = nz;
    if (I.x != 0) {
      ++te;
      const double vect[3] = {e_sub(e_add(A.x, s[0]), xi[0]), e_sub(e_add(A.y, s[1]), xi[1]),
                              e_sub(e_add(A.z, s[2]), xi[2])};
      const double d2 = e_add(e_add(e_sq(vect[0]), e_sq(vect[1])), e_sq(vect[2]));
      bool take = I.x == 1;
      if (!take) {
        const double t1 = corr ? fma(A.w, inv_theta, B.w) : A.w * inv_theta;
        const double gap = fma(-t1, t1, d2);
        take = gap > 0.;
        if (!(fabs(gap) > 1e-12 * d2) || !square) take = accept_exact(d2, A.w, B.w, theta0, corr);
      }
      if (!take) {
        if (I.y != kEnd) next = I.y;
      } else {
        bool use = true;
        if (unshifted && I.x == 1) {  // the target's own segments are skipped
          const int j = __ldg(prv + I.w);
          use = !(j == gi_ || j == pi_);
        }
        if (use) {
          const double circ[3] = {B.x, B.y, B.z};
          const double b = e_mul(2.0, dot3(vect, circ));
          const double c = dot3(circ, circ);
          double ya;
          double dist = near_sqrt(d2, ya);
          const bool far = mid_range<true>(d2);
          if (!far) dist = e_sqrt(d2);
          const double a = e_mul(dist, dist);
          const double D = term_d(a, b, c);
          const double abc = e_add(e_add(a, b), c);
          if (I.x == 1 && dist < NV_EPS) {
            singular = true;
          } else if (!(D < NV_EPS)) {
            double tm[3];
            term_value(vect, circ, b, c, D, abc, dist, ya, qc, two_pi, tm);
            if (!(far && mid_range<false>(D) && mid_range<true>(abc))) {
              const double3 t = node_term_exact(vect[0], vect[1], vect[2], circ[0], circ[1], circ[2], dist, qc, two_pi);
              tm[0] = t.x;
              tm[1] = t.y;
              tm[2] = t.z;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) acc[k] = e_add(acc[k], tm[k]);
            ++ev;
          }
        }
      }
    }
    if (next == kEnd) break;
    if (next == nz) {
      A = An;
      B = Bn;
      I = In;
    } else {
      A = ldg4(&tb.nA[next]);
      B = ldg4(&tb.nB[next]);
      I = __ldg(&tb.nI[next]);
    }
  }
  evals += ev;
  tests += te;
}

// Local term, the unshifted image's tree sum ub0, the shifted images' sum ubs, mutual
// friction, in the reference's order of additions (timestep.f90:79-140).
__device__ void fp64_epilogue(const SysConst &sc, const SysDyn &dy, int g, const double *__restrict__ X,
                              const double *__restrict__ GI, const double *__restrict__ GB, double *__restrict__ U,
                              long long T, const double ub0[3], const double ubs[3]) {
  double xi[3], gi[3], gb[3], u[3], fdot[3];
  load3(X, T, g, xi);
  load3(GI, T, g, gi);
  load3(GB, T, g, gb);
  local_velocity(sc, xi, gi, gb, u, fdot);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], ub0[c]);
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], ubs[c]);
  if (sc.n_mirror)  // the mirrored trees' sum, walked before (k_tree_walk_mirror)
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = e_add(u[c], sc.umir[c * T + g]);
  mf_epilogue(sc, dy, xi, fdot, u, g);
  store3(U, T, g, u);
}

// tree_walk_mirror (tree.f90:321-392) for every mirror of target g, in mirror order, into
// acc: each node's centre and centre + circulation reflected in the wall; theta = width/dist
// (the reference computes the corrected angle and then overwrites it with this one); a leaf
// whose segment goes into the wall, and the target's own image as biot_savart_mirror skips
// it, add nothing; the accept test includes the root (its circulation is zero, so an accepted
// root adds nothing either).
__device__ void walk_mirror(const TreeBuffers &tb, int root, const SysConst &sc, const double xi[3], int g, int pi_,
                            int pin_g, const int *__restrict__ prv, double acc[3], unsigned long long &evals,
                            unsigned long long &tests, bool &singular, bool &overrun) {
  const double qc = sc.quant_circ, two_pi = sc.two_pi, theta0 = sc.tree_theta;
  for (int m = 0; m < sc.n_mirror; ++m) {
    const bool own = mirror_skips_own(sc, pin_g, m);
    int node = root;
    int left = tb.ctr[0];
    while (node != kEnd) {
      if (--left < 0) {
        overrun = true;
        break;
      }
      const double4 A = ldg4(&tb.nA[node]);
      const int4 I = __ldg(&tb.nI[node]);
      if (I.x == 0) {
        node = I.z;
        continue;
      }
      ++tests;
      const double4 B = ldg4(&tb.nB[node]);
      const double cent[3] = {A.x, A.y, A.z}, circ[3] = {B.x, B.y, B.z};
      double s[3], sgi[3];
      for (int c = 0; c < 3; ++c) {
        s[c] = reflect1(e_add(cent[c], circ[c]), sc.mirror[m][c], sc.box[c]);
        sgi[c] = reflect1(cent[c], sc.mirror[m][c], sc.box[c]);
      }
      const double dist = e_sqrt(e_add(e_add(e_sq(e_sub(xi[0], s[0])), e_sq(e_sub(xi[1], s[1]))), e_sq(e_sub(xi[2], s[2]))));
      const double theta = e_div(A.w, dist);
      if (I.x == 1 || theta < theta0) {
        node = (node == root) ? kEnd : I.z;
        if (I.x == 1) {
          const int j = __ldg(prv + I.w);
          if (pin_i(sc.pin[j])) continue;
          if (own && ((pin_b(pin_g) && g == j) || (pin_i(pin_g) && j == pi_))) continue;
          if (dist < NV_EPS) {
            singular = true;
            continue;
          }
        }
        const double vect[3] = {e_sub(s[0], xi[0]), e_sub(s[1], xi[1]), e_sub(s[2], xi[2])};
        const double dv[3] = {e_sub(sgi[0], s[0]), e_sub(sgi[1], s[1]), e_sub(sgi[2], s[2])};
        const double a = e_mul(dist, dist);
        const double b = e_mul(2.0, dot3(vect, dv));
        const double c = e_add(e_add(e_sq(e_sub(s[0], sgi[0])), e_sq(e_sub(s[1], sgi[1]))), e_sq(e_sub(s[2], sgi[2])));
        const double D = e_sub(e_mul(e_mul(4.0, a), c), e_mul(b, b));
        if (D < NV_EPS) continue;
        double cr[3];
        cross3(vect, dv, cr);
        const double den = e_mul(two_pi, D);
        const double fac = e_sub(e_div(e_add(e_mul(2.0, c), b), e_sqrt(e_add(e_add(a, b), c))), e_div(b, e_sqrt(a)));
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[k] = e_add(acc[k], e_mul(e_div(e_mul(cr[k], qc), den), fac));
        ++evals;
      } else {
        node = I.y != kEnd ? I.y : (node == root ? kEnd : I.z);
      }
    }
  }
}

// The mirror sums of every live target of the tree systems with solid walls (one thread
// each), written to umir for the FP64 walk's epilogue.  Runs after the roots' exact centres.
__global__ void k_tree_walk_mirror(const SysConst *__restrict__ scs, SysDyn *dyn, const int2 *__restrict__ work,
                                   const double *__restrict__ X, const int *__restrict__ nxt,
                                   const int *__restrict__ prv, long long T, TreeBuffers tb, unsigned *err) {
  const int2 w = work[blockIdx.x];
  const SysConst &sc = scs[w.x];
  if (!sc.n_mirror) return;
  const int g = w.y + threadIdx.x;
  const int k = g - sc.base;
  unsigned long long evals = 0, tests = 0;
  bool singular = false, overrun = false;
  if (!*err && k >= 1 && k <= dyn[w.x].pcount && k <= sc.cap && nxt[g] != 0) {
    double xi[3], acc[3] = {0, 0, 0};
    load3(X, T, g, xi);
    walk_mirror(tb, w.x, sc, xi, g, prv[g], sc.pin[g], prv, acc, evals, tests, singular, overrun);
    for (int c = 0; c < 3; ++c) sc.umir[c * T + g] = acc[c];
  }
  if (singular) atomicOr(err, DERR_SINGULAR);
  if (overrun) atomicOr(err, DERR_WALK);
  if (evals) atomicAdd(&dyn[w.x].tree_eval, evals);
  if (tests) atomicAdd(&dyn[w.x].tree_tests, tests);
}

// The tree sums of target g (timestep.f90:49-141 with tree_walk): over the unshifted image
// into ub0, then over the 26 shifts in order into ubs.  part 0 does both and the epilogue;
// part 1 only ub0, part 2 only ubs (the epilogue then runs where both are known), part 3 both
// without the epilogue -- each
// sum is the same chain of additions either way.  With `decided` the root's tests come from
// the centre estimate: a target for which any of them is too close to call is deferred
// whole (nothing counted; part 2 leaves the push to part 1), to be redone exactly.  Returns
// false for a deferred target.
__device__ bool fp64_target(const SysConst &sc, const SysDyn &dy, int sys, int g, const double *__restrict__ X,
                            const double *__restrict__ GI, const double *__restrict__ GB,
                            const int *__restrict__ prv, double *__restrict__ U, long long T, const TreeBuffers &tb,
                            bool decided, int part, double ub0[3], double ubs[3], unsigned long long &evals,
                            unsigned long long &tests, unsigned *err) {
  double xi[3];
  load3(X, T, g, xi);
  const double zero[3] = {0, 0, 0};
  int start[27];
  const int first = tb.nI[sys].y;
  unsigned long long t0 = 0;
  for (int m = 0; m <= sc.n_shift; ++m) {
    start[m] = sys;
    if (!decided) continue;
    const int d = root_decision(tb, sc, sys, xi, m == 0 ? zero : sc.shift[m - 1]);
    if (d == 2) {
      if (part != 2) defer_push(tb, g, err);
      return false;
    }
    start[m] = d == 1 ? kEnd : first;  // accepted: adds nothing; opened: walk the children
    ++t0;
  }
  if (part != 2) tests += t0;  // the root tests are counted once
  const int pi_ = prv[g];
  bool singular = false, overrun = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) ub0[c] = ubs[c] = 0.;
  if (part != 2) walk_fp64(tb, start[0], sc, xi, g, pi_, prv, zero, true, ub0, evals, tests, singular, overrun);
  if (part != 1)
    for (int m = 0; m < sc.n_shift; ++m)
      walk_fp64(tb, start[m + 1], sc, xi, g, pi_, prv, sc.shift[m], false, ubs, evals, tests, singular, overrun);
  if (singular) atomicOr(err, DERR_SINGULAR);
  if (overrun) atomicOr(err, DERR_WALK);
  if (part == 0) fp64_epilogue(sc, dy, g, X, GI, GB, U, T, ub0, ubs);
  return true;
}

// Plain FP64 tree walk, 64 targets per block.  With `split`, two threads per target (128
// per block): warps 0-1 sum the unshifted image (the deepest walk), warps 2-3 the 26 shifted
// ones, and the second thread adds the two sums in the reference's order once both are
// done -- for small systems, whose few blocks would leave most SMs idle.  Without, one
// thread per target does it all (64 per block).
__global__ void __launch_bounds__(128) k_tree_walk_fp64(const SysConst *__restrict__ scs, SysDyn *dyn,
                                                        const int2 *__restrict__ work, const double *__restrict__ X,
                                                        const double *__restrict__ GI, const double *__restrict__ GB,
                                                        const int *__restrict__ nxt, const int *__restrict__ prv,
                                                        double *__restrict__ U, long long T, TreeBuffers tb,
                                                        int split, unsigned *err) {
  __shared__ double s_ub0[3][64];
  const int2 w = work[blockIdx.x];
  const SysConst &sc = scs[w.x];
  const int t = threadIdx.x & 63, part = split ? 1 + (threadIdx.x >> 6) : 0;
  const int q = w.y + t - sc.base;  // position in the system's walk order
  const int g = q >= 1 && q <= sc.cap ? tb.perm[sc.base + q] : sc.base;
  const int k = g - sc.base;
  unsigned long long evals = 0, tests = 0;
  double ub0[3] = {0, 0, 0}, ubs[3] = {0, 0, 0};
  bool done = false;
  if (!*err && k >= 1 && k <= dyn[w.x].pcount && nxt[g] != 0 && q >= sc.walk_lo && q < sc.walk_hi)
    done = fp64_target(sc, dyn[w.x], w.x, g, X, GI, GB, prv, U, T, tb, true, part, ub0, ubs, evals, tests, err);
  if (part == 1)
    for (int c = 0; c < 3; ++c) s_ub0[c][t] = ub0[c];
  __syncthreads();
  if (part == 2 && done) {
    for (int c = 0; c < 3; ++c) ub0[c] = s_ub0[c][t];
    fp64_epilogue(sc, dyn[w.x], g, X, GI, GB, U, T, ub0, ubs);
  }
  // tree_eval (tree.f90:308): one atomic per warp
  unsigned long long tot = evals, tt = tests;
  for (int o = 16; o > 0; o >>= 1) {
    tot += __shfl_down_sync(0xffffffffu, tot, o);
    tt += __shfl_down_sync(0xffffffffu, tt, o);
  }
  if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&dyn[w.x].tree_eval, tot);
  if ((threadIdx.x & 31) == 0 && tt) atomicAdd(&dyn[w.x].tree_tests, tt);
}

// The targets with a deferred root test, after the exact root sums: again whole, by the exact
// FP64 walk (with `partial`, the mixed path, their sums go there).
__global__ void k_walk_fixup(const SysConst *__restrict__ scs, SysDyn *dyn, const int *__restrict__ sys_of,
                             const double *__restrict__ X, const double *__restrict__ GI,
                             const double *__restrict__ GB, const int *__restrict__ prv, double *__restrict__ U,
                             double *__restrict__ partial, long long T, TreeBuffers tb, unsigned *err) {
  const int n = min(*tb.defer_n, kDeferCap);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int g = tb.defer[e], s = sys_of[g];
    const SysConst &sc = scs[s];
    unsigned long long evals = 0, tests = 0;
    double ub0[3], ubs[3];
    fp64_target(sc, dyn[s], s, g, X, GI, GB, prv, U, T, tb, false, partial ? 3 : 0, ub0, ubs, evals, tests, err);
    if (partial)
      for (int c = 0; c < 3; ++c) partial[c * T + g] = ub0[c] + ubs[c];
    if (evals) atomicAdd(&dyn[s].tree_eval, evals);
    if (tests) atomicAdd(&dyn[s].tree_tests, tests);
  }
}

// Squared distance from x to the cell [P, P + w]^3 (0 inside).
__device__ __forceinline__ double cube_dist2(const double x[3], const double4 P, double w) {
  const double p[3] = {P.x, P.y, P.z};
  double d2 = 0.;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double lo = p[c] - x[c], hi = x[c] - (p[c] + w);
    const double d = fmax(fmax(lo, hi), 0.);
    d2 += d * d;
  }
  return d2;
}

// An upper bound on the distance the closest-point walk settles on: the distance of a leaf
// that walk accepts and counts, or 100.  A node whose cell holds the target is opened by the
// walk (its centroid lies in the same cell, so width/dist >= 1/sqrt(3) > .5), so every child
// of such a node is reached; a child that is a single point is accepted, and below such a
// child the walk's own opening test decides what is reached.  Any accepted leaf's distance,
// formed as the walk forms it, is at least the walk's final closestd.  The search follows
// the cells that hold the target down from the root, takes the nearest counted leaf child on
// the way, and then walks, with the reference's opening test, the subtree of the deepest
// node on that path that holds at least kBoundNode points (a few dozen visits): warps whose
// targets all get a bound near their final closestd prune the rest of their walks alike.
constexpr int kBoundNode = 16;

__device__ double closest_bound(const TreeBuffers &tb, const SysConst &sc, int root, const double xi[3], int g,
                                int ni, int pi_, const int *__restrict__ prv) {
  double best = 100.;
  auto counted = [&](int j) { return j != g && j != ni && j != pi_ && !pinned_at(sc, j); };
  auto dist_to = [&](const double4 &A) {
    return e_sqrt(e_add(e_add(e_sq(e_sub(xi[0], A.x)), e_sq(e_sub(xi[1], A.y))), e_sq(e_sub(xi[2], A.z))));
  };
  {  // the root's cell must hold the target too (it always does between enforce_boundary calls)
    const double4 P = ldg4(&tb.nP[root]);
    const double w = tb.nA[root].w;
    if (!(xi[0] >= P.x && xi[0] < P.x + w && xi[1] >= P.y && xi[1] < P.y + w && xi[2] >= P.z && xi[2] < P.z + w))
      return best;
  }
  int node = root, deep = root;
  for (int depth = 0; depth <= kMaxLevels && node != kEnd; ++depth) {
    const int4 I = __ldg(&tb.nI[node]);
    if (I.x <= 1 || I.y == kEnd) break;
    if (I.x >= kBoundNode) deep = node;
    const int stop = I.z;  // the node after the last child's subtree
    int next = kEnd;
    for (int c = I.y; c != kEnd && c != stop;) {
      const int4 Ic = __ldg(&tb.nI[c]);
      if (Ic.x == 1) {
        if (counted(__ldg(prv + Ic.w))) best = fmin(best, dist_to(ldg4(&tb.nA[c])));
      } else if (Ic.x > 1 && next == kEnd) {
        const double4 P = ldg4(&tb.nP[c]);
        const double w = tb.nA[c].w;
        if (xi[0] >= P.x && xi[0] < P.x + w && xi[1] >= P.y && xi[1] < P.y + w && xi[2] >= P.z && xi[2] < P.z + w)
          next = c;
      }
      c = Ic.z;
    }
    node = next;
  }
  // the walk below `deep` (opened: it holds the target), with the reference's opening test
  const int4 Id = __ldg(&tb.nI[deep]);
  if (Id.x <= 1) return best;
  int left = tb.ctr[0];  // (a malformed tree only loosens the bound; the main walk reports it)
  for (int n = Id.y; n != kEnd && n != Id.z && --left >= 0;) {
    const int4 I = __ldg(&tb.nI[n]);
    if (I.x == 0) {
      n = I.z;
      continue;
    }
    const double4 A = ldg4(&tb.nA[n]);
    const double dist = dist_to(A);
    if (I.x == 1 || e_div(A.w, dist) < .5) {
      if (I.x == 1 && counted(__ldg(prv + I.w))) best = fmin(best, dist);
      n = I.z;
    } else {
      n = I.y != kEnd ? I.y : I.z;
    }
  }
  return best;
}

// pclose_tree + closest_tree (tree.f90:190-244): theta = width/dist < .5, no shift, no
// correction; the candidate is prv(first member's infront at build time) with the links of
// now (after pinsert).  Subtrees whose cells lie farther than min(cd, closest_bound) are
// skipped: they hold no leaf or node that could still change closest or closestd.
template <bool kPrefetch>
__global__ void k_closest_tree(const SysConst *__restrict__ scs, const SysDyn *__restrict__ dyn,
                               const int *__restrict__ sys_of, const double *__restrict__ X,
                               const int *__restrict__ nxt, const int *__restrict__ prv, int *__restrict__ cl,
                               double *__restrict__ CD, long long T, TreeBuffers tb, unsigned *err) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T || *err) return;
  const long long g = tb.perm[t];  // the walk order: neighbouring threads, neighbouring targets
  const int s = sys_of[g];
  const SysConst &sc = scs[s];
  if (!sc.use_tree || (dyn[s].itime % sc.recon_shots) != 0) return;
  const int k = (int)(g - sc.base);
  if (k < 1 || k > dyn[s].pcount) return;
  double cd = 100.;
  const int ni = nxt[g];
  if (ni == 0) {
    CD[g] = cd;
    return;
  }
  if (pinned_at(sc, (int)g)) {  // pinned points are not tested (tree.f90:198-199)
    CD[g] = cd;
    return;
  }
  const int pi_ = prv[g];
  int best = cl[g];
  double xi[3];
  load3(X, T, (int)g, xi);
  // The reference forms dist = sqrt(d2) and theta = width/dist at every node.  Both are
  // correctly rounded, so theta < .5 and dist < cd can differ from d2 > 4 width^2 and
  // d2 < cd^2 only when d2 lies within a few ulps of the bound: outside a 1e-12 band the
  // squared comparison decides, inside it the reference's own expressions do.
  constexpr double kBand = 1e-12;
  double cd2 = cd * cd;
  // slack of the subtree skip below: covers the rounding of the centroids (sums of up to
  // 2^24 positions) and of the distances
  const double margin = 1e-8 * sc.bsize;
  const double bound = closest_bound(tb, sc, s, xi, (int)g, ni, pi_, prv);
  int node = s;
  double4 A = ldg4(&tb.nA[node]);
  int4 I = __ldg(&tb.nI[node]);
  int left = tb.ctr[0];  // a walk of a well-formed tree visits each node at most once
  for (;;) {
    if (--left < 0) {
      atomicOr(err, DERR_WALK);
      break;
    }
    // kPrefetch (few targets, latency-bound): the records of both possible successors (next
    // in preorder past the subtree, first child) are requested before this node is decided,
    // so their loads overlap the test; with a full GPU the extra loads cost more than that
    const int nz = I.z, ny = I.y;
    double4 Az = make_double4(0, 0, 0, 0), Ay = Az;
    int4 Iz = make_int4(0, kEnd, kEnd, 0), Iy = Iz;
    if (kPrefetch && nz != kEnd) {
      Az = ldg4(&tb.nA[nz]);
      Iz = __ldg(&tb.nI[nz]);
    }
    if (kPrefetch && ny != kEnd) {
      Ay = ldg4(&tb.nA[ny]);
      Iy = __ldg(&tb.nI[ny]);
    }
    bool down = false;  // to the first child; else past the subtree
    if (I.x != 0) {
      const double d2 = e_add(e_add(e_sq(e_sub(xi[0], A.x)), e_sq(e_sub(xi[1], A.y))), e_sq(e_sub(xi[2], A.z)));
      bool acc = I.x == 1;
      if (!acc) {
        const double w4 = 4.0 * A.w * A.w;
        if (d2 > w4 * (1 + kBand)) acc = true;
        else if (d2 >= w4 * (1 - kBand)) acc = e_div(A.w, e_sqrt(d2)) < .5;
      }
      if (acc) {
        bool closer;
        if (d2 < cd2 * (1 - kBand)) closer = true;
        else if (d2 > cd2 * (1 + kBand)) closer = false;
        else closer = e_sqrt(d2) < cd;
        if (closer) {
          const int j = prv[I.w];
          if (I.x > 1) {
            best = 0;
          } else if (j != (int)g && ni != j && pi_ != j && !pinned_at(sc, j)) {  // pinned j: nothing
            best = j;
            cd = e_sqrt(d2);
            cd2 = cd * cd;
          }
        }
      } else if (ny != kEnd &&
                 !(node != s && cube_dist2(xi, ldg4(&tb.nP[node]), A.w) >
                               (fmin(cd, bound) + margin) * (fmin(cd, bound) + margin))) {
        down = true;
      }
      // (an opened node whose cell lies farther than cd: every member of this node lies in
      // its cell -- the splits drop points outside the children's cells -- so every
      // centroid in its subtree is farther than cd: none is closer, now or later (cd only
      // shrinks), and none changes best or cd.  Its subtree is skipped.)
    }
    const int next = down ? ny : nz;
    if (next == kEnd) break;
    if (kPrefetch) {
      A = down ? Ay : Az;
      I = down ? Iy : Iz;
    } else {
      A = ldg4(&tb.nA[next]);
      I = __ldg(&tb.nI[next]);
    }
    node = next;
  }
  cl[g] = best;
  CD[g] = cd;
}

// Mixed-precision node records: FP64 centre with the squared acceptance distance, FP32
// circulation.  The opening test of tree_walk (tree.f90:266-278) accepts a node when
//   dist - geo > 0 and width/(dist - geo) < theta0   <=>  dist > geo + width/theta0, or
//   dist - geo <= 0 and width/dist < theta0          <=>  geo >= dist > width/theta0,
// (without the correction: dist > width/theta0); comparing squared distances in FP64 gives
// the same decisions except at exact ties.  The second branch needs geo > width/theta0,
// impossible for theta0 <= 2/sqrt(3) (geo <= sqrt(3)/2 width), so it is tested only above.
// Roots are skipped: their exact centre may still be summing (the walks take the roots'
// tests from the centre estimate).
// Relative half-width of the band around the opening threshold inside which the mixed
// walk's FP32 test defers to the FP64 one (the FP32 |r|^2 is within ~1e-6 of its value).
constexpr float kTestBand = 1e-5f;

__global__ void k_node_prep(TreeBuffers tb, int nsys, double theta0, int corr, const int *__restrict__ prv) {
  if (failed_above(tb, INT_MAX)) return;
  const int n = tb.ctr[0];
  for (int id = nsys + blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
    const double4 A = tb.nA[id], B = tb.nB[id];
    const double t0 = A.w / theta0;
    const double t1 = corr ? B.w + t0 : t0;
    tb.mx.C[id] = make_double4(A.x, A.y, A.z, t1 * t1);
    const float qx = (float)B.x, qy = (float)B.y, qz = (float)B.z;
    tb.mx.G[id] = make_double2(corr ? B.w * B.w : -1.0, t0 * t0);
    const float hx = (float)A.x, hy = (float)A.y, hz = (float)A.z;
    const int4 I = tb.nI[id];
    WalkNode wn;
    wn.a = make_float4(hx, hy, hz, (float)(t1 * t1));
    const float q2 = qx * qx + qy * qy + qz * qz;
    wn.b = make_float4((float)(A.x - hx), (float)(A.y - hy), (float)(A.z - hz), q2);
    wn.c = make_float4(qx, qy, qz, 0.f);
    wn.d = make_int4(I.x, I.y, tb.nKids[id], I.x == 1 ? prv[I.w] : I.w);
    tb.mx.W[id] = wn;
  }
}

// A leaf's record holds prv of its member, the start of the leaf's segment, for the walk's
// own-segment test; this refreshes it when points were relinked after the build.
__global__ void k_leaf_links(TreeBuffers tb, int nsys, const int *__restrict__ prv) {
  if (failed_above(tb, INT_MAX)) return;
  const int n = tb.ctr[0];
  for (int id = nsys + blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
    const int4 I = tb.nI[id];
    if (I.x == 1) tb.mx.W[id].d.w = prv[I.w];
  }
}

// Mixed tree walk: a block of W warps per group of 32 targets that are close in space
// (consecutive in the walk order), lane k of every warp holding target k, for all images
// at once.  An entry of the work list is (node, image, mask of the lanes whose walk reaches the
// node); the block takes up to 32 W entries a round, one per lane, and
//   1. each lane tests its entry's node against the box around the group's targets: most nodes
//      are accepted by every target or opened by every target, which settles 32 entries in one
//      pass over the lanes;
//   2. the entries in between are tested target by target, the lanes taking the reference's
//      opening decision each for its own target;
//   3. accepted nodes go to the term list with their lanes, the children of opened ones back
//      to the work list (a prefix sum over the block gives every entry its place, so that the
//      order, and with it every rounding, is the same in every run);
//   4. a full term list is summed: each warp takes 32 of its nodes, loads them (a lane a node)
//      into shared memory, two nodes side by side, and every lane adds its target's terms, two
//      in one packed instruction.
// So a node's record is loaded once per group, by lanes in parallel, and neither the loop over
// the nodes nor the tests diverge.  Which nodes a target accepts is the reference's choice
// (tree.f90:250-316), node by node; only the order of the additions is not.
//
// The opening test compares |r|^2 with t1^2.  r is formed in FP32 from the high and low parts
// of the image-shifted centre and of the target (|r_FP32 - r| <~ 2^-23 |r|), so |r|^2 in FP32
// is within 1e-6 of its value; outside a 1e-5 band around t1^2 the FP32 comparison gives the
// FP64 answer, inside it the FP64 test runs.  The box's distances are widened by 1e-6 of
// themselves and of the box, so that a verdict for the box holds for every target in it.
// FP32 terms are summed over one term list (at most 16 to a partial sum) and promoted to FP64;
// leaves within the near radius and ill-conditioned terms are evaluated in FP64.  Writes the
// target's sum over all images.
//
// Bound: latencies that 16 to 20 warps an SM, all that their shared memory lets reside, do not
// cover.  32,768 points: 16 warps active, 2.24 instructions a cycle of 4, 7.1 cycles between two
// of a warp, of them 1.8 fixed latencies, 1.0 at barriers and 1.2 for loads; ALU, FMA and XU at 38, 36
// and 27 % of their rates, DRAM at 0.2 %.  100,003 points: 1.39 ms; 1,048,576: 9.9 ms, 11.0 after
// some steps (2.27 and 14.1 ms for a warp stepping through the union of its targets' walks node
// by node).
// FP64 terms where they occur instead of from the queue: 1.59 ms at 100,000 points in place of
// 1.54 (both on the Morton order).
constexpr int walk_cap(int W) { return W == 8 ? 4096 : W == 4 ? 2048 : 1024; }  // work-list entries
// Entries kept free: taking one entry at a time (depth first), a list grows by at most this.
constexpr int kWalkReserve = 8 * kMaxLevels;

template <int W>
struct WalkShared {
  int node[walk_cap(W)];
  unsigned mask[walk_cap(W)];
  unsigned char image[walk_cap(W)];
  // the term list: at most 32 W - 1 entries left over and 32 W of a round
  int tnode[64 * W];
  unsigned tmask[64 * W];
  unsigned char timage[64 * W];
  // per warp: its round's centres (hi, threshold; lo, lanes), later its 32 terms' records
  union Warp {
    float4 centre[32][2];
    float pair[16 * 28];
  } warp[W];
  unsigned tlanes[W][32];  // per term: its lanes
  int2 info[W][32];        // per term: node, image << 5
  unsigned own[32];        // filter of the targets' own segments: bit (slot mod 1024)
  int2 queue[W][96];       // per warp: FP64 terms (node, image << 5 | lane), at most 31 + 64
  double result[W][3][32];
  double target[3][32];
  double shift[27][3];
  unsigned open[27], undecided[W];
  int wterms[W], wkids[W];
  double red[3][W][32];
};

// (The blocks an SM are those that the shared memory allows: 16 warps for W = 8, 20 for 4 and 2, 13
// for 1, so that the registers they leave are used: 32,768 points 486 us, 499 with 80 registers.)
template <int W>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : W == 1 ? 13 : 20 / W) k_tree_walk_mixed(
    const SysConst *__restrict__ scs, SysDyn *dyn, const int2 *__restrict__ work, const double *__restrict__ X,
    const int *__restrict__ nxt, const int *__restrict__ prv, double *__restrict__ partial, long long T,
    TreeBuffers tb, double near_factor, Fp32Guards gd, unsigned *err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WalkShared<W> &S = *reinterpret_cast<WalkShared<W> *>(smem_raw);
  __shared__ int s_abort;  // one thread reads the error word: blocks of this launch may set it meanwhile
  constexpr unsigned kAll = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int2 w = work[blockIdx.x];  // system, first position
  const SysConst &sc = scs[w.x];
  const int q = w.y + lane - sc.base;  // position in the system's walk order
  const int g = q >= 1 && q <= sc.cap ? tb.perm[sc.base + q] : sc.base;
  const int k = g - sc.base;
  // A walk range's ends fall on group boundaries (nv_set_walk_range): a group walks all its
  // targets or none, so its rounds and partial sums are the same as without a range.
  const bool valid = k >= 1 && k <= dyn[w.x].pcount && nxt[g] != 0 && q >= sc.walk_lo && q < sc.walk_hi;
  if (tid == 0) s_abort = (*err != 0);
  unsigned evals = 0, tests = 0, n64 = 0, nband = 0;
  double xi[3] = {0, 0, 0};
  int pi_ = 0;
  if (valid) {
    load3(X, T, g, xi);
    pi_ = prv[g];
  }
  const int n_img = 1 + sc.n_shift;
  if (wid == 0) {
    for (int c = 0; c < 3; ++c) S.target[c][lane] = xi[c];
    S.own[lane] = 0;
    __syncwarp();
    if (valid) {
      atomicOr(&S.own[(g >> 5) & 31], 1u << (g & 31));
      atomicOr(&S.own[(pi_ >> 5) & 31], 1u << (pi_ & 31));
    }
  }
  for (int i = tid; i < 3 * n_img; i += 32 * W) S.shift[i / 3][i % 3] = i < 3 ? 0.0 : sc.shift[i / 3 - 1][i % 3];
  __syncthreads();
  if (s_abort) return;
  // the root's test in every image from the centre estimate: accepted (nothing to add), opened
  // (the walk starts at its children) or undecided: the target is redone whole once the exact
  // centre is known
  {
    unsigned undec = 0;
    for (int m = wid; m < n_img; m += W) {
      const int rd = valid ? root_decision(tb, sc, w.x, xi, S.shift[m]) : 1;
      const unsigned open = __ballot_sync(kAll, rd == 0);
      undec |= __ballot_sync(kAll, rd == 2);
      if (lane == 0) S.open[m] = open;
    }
    if (lane == 0) S.undecided[wid] = undec;
  }
  __syncthreads();
  unsigned undec = 0;
#pragma unroll
  for (int v = 0; v < W; ++v) undec |= S.undecided[v];
  const unsigned live = __ballot_sync(kAll, valid) & ~undec;
  const bool mine = (live >> lane) & 1u;
  if (wid == 0) {
    if (valid && !mine) defer_push(tb, g, err);
    if (mine) tests += n_img;
  }
  const int first = tb.nI[w.x].y, n_kids = tb.nKids[w.x];
  int top = 0, nterm = 0;  // entries of the work list, of the term list (block-uniform)
  if (live) {  // the root's children in every image that some target opens
    for (int m = 0; m < n_img; ++m) {
      const unsigned open = S.open[m] & live;
      if (!open) continue;
      if (tid < n_kids) {
        S.node[top + tid] = first + tid;
        S.mask[top + tid] = open;
        S.image[top + tid] = (unsigned char)m;
      }
      top += n_kids;
    }
  }
  // the box around the live targets
  float bh[3], bl[3], bw[3];  // centre high and low, half width
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double lo = mine ? xi[c] : 1e300, hi = mine ? xi[c] : -1e300;
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(kAll, lo, o));
      hi = fmax(hi, __shfl_xor_sync(kAll, hi, o));
    }
    const double mid = 0.5 * (lo + hi);
    bh[c] = (float)mid;
    bl[c] = (float)(mid - (double)bh[c]);
    bw[c] = (float)(0.5 * (hi - lo)) * 1.000002f;
  }
  LaneTarget t;
  float xh[3], xl[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    xh[c] = (float)xi[c];
    xl[c] = (float)(xi[c] - (double)xh[c]);
    t.h[c] = pack2(-xh[c], -xh[c]);
    t.l[c] = pack2(-xl[c], -xl[c]);
  }
  const float near2 = (float)(near_factor * sc.delta * near_factor * sc.delta);
  const double gq64 = sc.quant_circ / (4.0 * NV_PI);
  const bool second = sc.tree_extra_correction && sc.tree_theta > 1.1547;
  double nx = 0., ny = 0., nz = 0.;  // FP64 terms and the promoted FP32 sums
  bool singular = false;
  // r and |r|^2 in FP64 as the FP64 walk forms them: (centre + shift) - target
  auto exact_r = [&](int cur, int m, double r[3]) -> double {
    const double4 C = ldg4(&tb.mx.C[cur]);
    r[0] = e_sub(e_add(C.x, S.shift[m][0]), xi[0]);
    r[1] = e_sub(e_add(C.y, S.shift[m][1]), xi[1]);
    r[2] = e_sub(e_add(C.z, S.shift[m][2]), xi[2]);
    return e_add(e_add(e_sq(r[0]), e_sq(r[1])), e_sq(r[2]));
  };
  // The terms that go to FP64 wait in a queue of the warp until there are 32, then a lane takes
  // one each, whoever's target it is for, and the targets' lanes add the results in queue order.
  int nq = 0;  // warp-uniform
  auto flush64 = [&]() {
    const int n = min(nq, 32);
    __syncwarp();
    double tm[3] = {0., 0., 0.};
    int to = -1;
    if (lane < n) {
      const int2 item = S.queue[wid][lane];
      to = item.y & 31;
      const int m = item.y >> 5;
      const double4 C = ldg4(&tb.mx.C[item.x]), B = ldg4(&tb.nB[item.x]);
      const double r[3] = {e_sub(e_add(C.x, S.shift[m][0]), S.target[0][to]),
                           e_sub(e_add(C.y, S.shift[m][1]), S.target[1][to]),
                           e_sub(e_add(C.z, S.shift[m][2]), S.target[2][to])};
      const double circ[3] = {B.x, B.y, B.z};
      // the reference's singularity check and skip decision in its own arithmetic
      // (tree.f90:289-303), the value from the cancellation-free form
      const double d2 = e_add(e_add(e_sq(r[0]), e_sq(r[1])), e_sq(r[2]));
      const double dist = e_sqrt(d2);
      const double a = e_mul(dist, dist);
      const double b = e_mul(2.0, dot3(r, circ));
      const double c = dot3(circ, circ);
      if (dist < NV_EPS) {
        singular = true;
        --evals;
      } else if (e_sub(e_mul(e_mul(4.0, a), c), e_mul(b, b)) < NV_EPS) {
        --evals;
      } else {
        term64_stable(r, circ, d2, gq64, tm);
        ++n64;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) S.result[wid][c][lane] = tm[c];
    const int2 left = lane < nq - 32 ? S.queue[wid][32 + lane] : make_int2(0, 0);
    const int2 left2 = lane < nq - 64 ? S.queue[wid][64 + lane] : make_int2(0, 0);
    __syncwarp();
    for (int i = 0; i < n; ++i) {
      const int l = __shfl_sync(kAll, to, i);
      if (l == lane) {
        nx += S.result[wid][0][i];
        ny += S.result[wid][1][i];
        nz += S.result[wid][2][i];
      }
    }
    if (lane < nq - 32) S.queue[wid][lane] = left;
    if (lane < nq - 64) S.queue[wid][32 + lane] = left2;
    nq -= n;
    __syncwarp();
  };
  // lanes of term (entry k of the warp's 32) into the queue
  auto push64 = [&](bool bad, int k) {
    const unsigned b = __ballot_sync(kAll, bad);
    if (bad) {
      const int2 inf = S.info[wid][k];
      S.queue[wid][nq + __popc(b & ((1u << lane) - 1u))] = make_int2(inf.x, inf.y | lane);
    }
    nq += __popc(b);
  };
  // a node's centre moved by the image's shift, FP32 high and low parts
  auto shifted = [&](const float4 &hi, const float4 &lo, int m, float h[3], float l[3]) {
    const float ch[3] = {hi.x, hi.y, hi.z}, cl[3] = {lo.x, lo.y, lo.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double v = (double)ch[c] + (double)cl[c] + S.shift[m][c];
      h[c] = (float)v;
      l[c] = (float)(v - (double)h[c]);
    }
  };
  // The terms of list entries [t0, t1): 32 to a warp, a partial FP32 sum of at most 16 each.
  const f32x2 kMinus = pack2(-1.f, -1.f), kAngle = pack2(gd.angle, gd.angle), kEndG = pack2(gd.end, gd.end);
  auto sum_terms = [&](int t0, int t1) {
    const int e = t0 + 32 * wid + lane;
    const int n = min(32, t1 - (t0 + 32 * wid));
    if (n <= 0) return;  // warp-uniform
    float *pr = S.warp[wid].pair;
    __syncwarp();
    {
      unsigned lanes = 0;
      int id = 0, m = 0, leaf = -1;
      float h[3] = {0, 0, 0}, l[3] = {0, 0, 0}, qx = 0, qy = 0, qz = 0, q2 = 0, near = 0;
      if (lane < n) {
        lanes = S.tmask[e];
        id = S.tnode[e];
        m = S.timage[e];
        const WalkNode *wn = tb.mx.W + id;
        const float4 A = __ldg(&wn->a), B = __ldg(&wn->b), Q = __ldg(&wn->c);
        const int4 D = __ldg(&wn->d);
        shifted(A, B, m, h, l);
        qx = Q.x;
        qy = Q.y;
        qz = Q.z;
        q2 = B.w;
        if (D.x == 1) {
          near = near2;  // near leaves in FP64
          if (m == 0 && ((S.own[(D.w >> 5) & 31] >> (D.w & 31)) & 1u)) leaf = D.w;
        }
      }
      // the targets' own segments are skipped in the central image: a leaf that the filter
      // lets through is compared with every target's two
      for (unsigned hit = __ballot_sync(kAll, leaf >= 0); hit; hit &= hit - 1) {
        const int j = __ffs(hit) - 1, sl = __shfl_sync(kAll, leaf, j);
        const unsigned own = __ballot_sync(kAll, sl == g || sl == pi_);
        if (lane == j) {
          evals -= __popc(lanes & own);
          lanes &= ~own;
        }
      }
      const float v[14] = {h[0], h[1], h[2], l[0], l[1], l[2], qx, qy, qz, -qx, -qy, near, gd.line * q2, gd.end * q2};
      float *rec = pr + 28 * (lane >> 1) + (lane & 1);
#pragma unroll
      for (int c = 0; c < 14; ++c) rec[2 * c] = v[c];
      S.tlanes[wid][lane] = lanes;
      S.info[wid][lane] = make_int2(id, m << 5);
    }
    __syncwarp();
    f32x2 ux = pack2(0.f, 0.f), uy = ux, uz = ux;
    const int np = (n + 1) / 2;
    for (int p = 0; p < np; ++p) {
      const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(pr + 28 * p);
      const PairVec r = pair_vec(rec, t);
      const ulonglong2 v3 = rec[3], v4 = rec[4], v5 = rec[5], v6 = rec[6];
      const PairSeg d = {{v3.x}, {v3.y}, {v4.x}, {v4.y}, {v5.x}, {v5.y}};
      const f32x2 near = {v5.y}, line = {v6.x}, end = {v6.y};
      const uint2 lanes = *reinterpret_cast<const uint2 *>(&S.tlanes[wid][2 * p]);
      const PairGeo geo = pair_geo(r, d);
      const f32x2 cr2 = square2(geo.cx, geo.cy, geo.cz);
      const f32x2 sum = add2(geo.pp, geo.re), dif = fma2(geo.re, kMinus, geo.pp);
      // FP64 for a near leaf, a term the reference skips (4ac-b^2 = 4|r x circ|^2 < epsilon,
      // tree.f90:303) and where FP32 would cancel digits: the target near the segment's line,
      // near its far end, or under a wide angle (Fp32Guards)
      const f32x2 wide = mul2(geo.pp, kAngle), ea = mul2(r.a, kEndG);
      const f32x2 ln = mul2(line, pack2(fminf(lo2(r.a), lo2(geo.ee)), fminf(hi2(r.a), hi2(geo.ee))));
      constexpr float kSkip = 0.25f * (float)NV_EPS;
      const bool in0 = (lanes.x >> lane) & 1u, in1 = (lanes.y >> lane) & 1u;
      const bool bad0 = lo2(r.a) < lo2(near) || lo2(cr2) < lo2(ln) || lo2(cr2) < kSkip || lo2(geo.ee) < lo2(ea) ||
                        lo2(geo.ee) < lo2(end) || lo2(sum) < lo2(wide);
      const bool bad1 = hi2(r.a) < hi2(near) || hi2(cr2) < hi2(ln) || hi2(cr2) < kSkip || hi2(geo.ee) < hi2(ea) ||
                        hi2(geo.ee) < hi2(end) || hi2(sum) < hi2(wide);
      // pp + r.e = |r x circ|^2 / (pp - r.e) when r.e < 0 (no cancellation either way)
      const bool ob0 = lo2(geo.re) < 0.f, ob1 = hi2(geo.re) < 0.f;
      const f32x2 topf = mul2(geo.num, pack2(ob0 ? lo2(dif) : 1.f, ob1 ? hi2(dif) : 1.f));
      const f32x2 f = mul2(topf, pack2(rcp_fast(ob0 ? lo2(cr2) : lo2(sum)), rcp_fast(ob1 ? hi2(cr2) : hi2(sum))));
      const f32x2 fk = pack2(in0 && !bad0 ? lo2(f) : 0.f, in1 && !bad1 ? hi2(f) : 0.f);
      ux = fma2(fk, geo.cx, ux);
      uy = fma2(fk, geo.cy, uy);
      uz = fma2(fk, geo.cz, uz);
      if (__any_sync(kAll, (in0 && bad0) || (in1 && bad1))) {
        push64(in0 && bad0, 2 * p);
        push64(in1 && bad1, 2 * p + 1);
        while (nq >= 32) flush64();
      }
    }
    nx += gq64 * ((double)lo2(ux) + (double)hi2(ux));
    ny += gq64 * ((double)lo2(uy) + (double)hi2(uy));
    nz += gq64 * ((double)lo2(uz) + (double)hi2(uz));
    __syncwarp();
  };
  __syncthreads();
  // (no visit budget here, unlike the FP64 walks: an image's entries are distinct nodes, and the
  // build makes a tree)
  while (top > 0) {
    const int n = min(min(top, 32 * W), max(1, (walk_cap(W) - kWalkReserve - top) / 8));
    const int base = top - n;
    const int e = base + 32 * wid + lane;
    const bool have = 32 * wid + lane < n;
    int id = 0, m = 0, kids = 0, first_kid = 0;
    unsigned mask = 0, acc_lanes = 0, open_lanes = 0;
    bool split = false;
    if (have) {
      id = S.node[e];
      mask = S.mask[e];
      m = S.image[e];
      const WalkNode *wn = tb.mx.W + id;
      const int4 D = __ldg(&wn->d);
      const float4 A = __ldg(&wn->a), B = __ldg(&wn->b);
      kids = D.z;
      first_kid = D.y;
      tests += __popc(mask);  // (every node below a root has members)
      if (D.x == 1) {
        acc_lanes = mask;
      } else {
        float h[3], l[3];
        shifted(A, B, m, h, l);
        float dmin2 = 0.f, dmax2 = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float d = fabsf((h[c] - bh[c]) + (l[c] - bl[c]));
          const float lo = fmaxf(fmaf(d, 0.999999f, -bw[c]), 0.f), hi = fmaf(d, 1.000001f, bw[c]);
          dmin2 = fmaf(lo, lo, dmin2);
          dmax2 = fmaf(hi, hi, dmax2);
        }
        if (!second && dmin2 > A.w * (1.f + kTestBand)) {
          acc_lanes = mask;
        } else if (!second && dmax2 < A.w * (1.f - kTestBand)) {
          open_lanes = mask;
        } else {
          split = true;
          S.warp[wid].centre[lane][0] = make_float4(h[0], h[1], h[2], A.w);
          S.warp[wid].centre[lane][1] = make_float4(l[0], l[1], l[2], __uint_as_float(mask));
        }
      }
    }
    const unsigned todo = __ballot_sync(kAll, split);
    __syncwarp();
    for (unsigned rest = todo; rest; rest &= rest - 1) {
      const int j = __ffs(rest) - 1;
      const float4 H = S.warp[wid].centre[j][0], L = S.warp[wid].centre[j][1];
      const float rx = (H.x - xh[0]) + (L.x - xl[0]);
      const float ry = (H.y - xh[1]) + (L.y - xl[1]);
      const float rz = (H.z - xh[2]) + (L.z - xl[2]);
      const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
      const unsigned lanes = __float_as_uint(L.w);
      bool acc = d2 > H.w * (1.f + kTestBand);
      // near the threshold (or the second criterion): the FP64 test
      if (((lanes >> lane) & 1u) && (second || (!acc && !(d2 < H.w * (1.f - kTestBand))))) {
        ++nband;
        const int cur = S.node[base + 32 * wid + j];
        double r[3];
        const double d2e = exact_r(cur, S.image[base + 32 * wid + j], r);
        acc = d2e > tb.mx.C[cur].w;
        if (!acc && second) {
          const double2 G = tb.mx.G[cur];
          acc = d2e <= G.x && d2e > G.y;
        }
      }
      const unsigned al = __ballot_sync(kAll, acc) & lanes;
      if (lane == j) {
        acc_lanes = al;
        open_lanes = lanes & ~al;
      }
    }
    // places: accepted nodes behind the term list, opened nodes' children on the work list
    if (!open_lanes) kids = 0;
    evals += __popc(acc_lanes);
    const unsigned accb = __ballot_sync(kAll, acc_lanes != 0);
    int scan = kids;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kAll, scan, o);
      if (lane >= o) scan += v;
    }
    if (lane == 31) {
      S.wkids[wid] = scan;
      S.wterms[wid] = __popc(accb);
    }
    __syncthreads();
    int koff = base + scan - kids, toff = nterm + __popc(accb & ((1u << lane) - 1u)), ktot = 0, ttot = 0;
#pragma unroll
    for (int v = 0; v < W; ++v) {
      if (v < wid) {
        koff += S.wkids[v];
        toff += S.wterms[v];
      }
      ktot += S.wkids[v];
      ttot += S.wterms[v];
    }
    if (acc_lanes) {
      S.tnode[toff] = id;
      S.tmask[toff] = acc_lanes;
      S.timage[toff] = (unsigned char)m;
    }
    for (int c = 0; c < kids; ++c) {
      S.node[koff + c] = first_kid + c;
      S.mask[koff + c] = open_lanes;
      S.image[koff + c] = (unsigned char)m;
    }
    top = base + ktot;
    nterm += ttot;
    __syncthreads();
    if (nterm >= 32 * W) {
      nterm -= 32 * W;
      sum_terms(nterm, nterm + 32 * W);
      // (the next round's barrier comes before its writes to the term list)
    }
  }
  sum_terms(0, nterm);
  if (nq) flush64();
  S.red[0][wid][lane] = nx;
  S.red[1][wid][lane] = ny;
  S.red[2][wid][lane] = nz;
  if (singular) atomicOr(err, DERR_SINGULAR);
  __syncthreads();
  for (int c = wid; c < 3; c += W) {
    double v = 0.;
#pragma unroll
    for (int u = 0; u < W; ++u) v += S.red[c][u][lane];
    if (mine) partial[c * T + g] = v;
  }
  int v[4] = {(int)evals, (int)tests, (int)n64, (int)nband};  // (a lane's evals can be below zero)
#pragma unroll
  for (int c = 0; c < 4; ++c)
    for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(kAll, v[c], o);
  if (lane == 0) {
    if (v[0]) atomicAdd(&dyn[w.x].tree_eval, (unsigned long long)(long long)v[0]);
    if (v[1]) atomicAdd(&dyn[w.x].tree_tests, (unsigned long long)(long long)v[1]);
    if (v[2]) atomicAdd((unsigned long long *)&dyn[w.x].diag[8], (unsigned long long)(long long)v[2]);
    if (v[3]) atomicAdd((unsigned long long *)&dyn[w.x].diag[9], (unsigned long long)(long long)v[3]);
    if (v[0] != v[2]) atomicAdd((unsigned long long *)&dyn[w.x].diag[10], (unsigned long long)(long long)(v[0] - v[2]));
  }
}

int n_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

}  // namespace

int n_sms_host() { return n_sms(); }
const int *tree_iperm(nv_handle *h) { return h->tree ? h->tree->iperm : nullptr; }
const int *tree_perm(nv_handle *h) { return h->tree ? h->tree->perm : nullptr; }

void tree_alloc(nv_handle *h) {
  bool need = false;
  for (auto &s : h->sc) need = need || s.use_tree || s.sched_tree;
  if (!need) return;
  auto *tb = new TreeBuffers();
  const long long T = h->T;
  tb->max_nodes = (int)std::min<long long>(3 * T + h->nsys + 1024, (1LL << 31) - 1);
  tb->max_members = 24 * T + 1024;
  cudaMalloc(&tb->nA, (size_t)tb->max_nodes * sizeof(double4));
  cudaMalloc(&tb->nB, (size_t)tb->max_nodes * sizeof(double4));
  cudaMalloc(&tb->nP, (size_t)tb->max_nodes * sizeof(double4));
  cudaMalloc(&tb->nI, (size_t)tb->max_nodes * sizeof(int4));
  cudaMalloc(&tb->nR, (size_t)tb->max_nodes * sizeof(int2));
  cudaMalloc(&tb->nDepth, (size_t)tb->max_nodes * sizeof(int));
  cudaMalloc(&tb->nKids, (size_t)tb->max_nodes * sizeof(int));
  cudaMalloc(&tb->nLeaf, (size_t)tb->max_nodes * sizeof(int));
  cudaMalloc(&tb->members, (size_t)tb->max_members * sizeof(int));
  // each level holds at most T / (kBlockSumNode + 1) nodes above the block threshold
  tb->max_big = (int)std::min<long long>((long long)kMaxLevels * (T / (kBlockSumNode + 1) + 1) + 64, 1 << 30);
  cudaMalloc(&tb->bigl, (size_t)tb->max_big * sizeof(int));
  cudaMalloc(&tb->root_apx, (size_t)h->nsys * sizeof(double4));
  cudaMalloc(&tb->rdig, (size_t)T);
  cudaMalloc(&tb->rrank, (size_t)T * sizeof(int));
  cudaMalloc(&tb->root_rank, ((size_t)h->nsys + 1) * 9 * sizeof(int));
  cudaMalloc(&tb->root_mb, (size_t)h->nsys * 8 * sizeof(int));
  cudaMalloc(&tb->root_ok, (size_t)h->nsys * sizeof(int));
  pass_alloc(&tb->pass_state, &tb->pass_ctl, 9, T);
  tb->root_parts = std::max(1, std::min(64, 4096 / h->nsys));
  cudaMalloc(&tb->root_part, (size_t)h->nsys * tb->root_parts * 6 * sizeof(double));
  cudaMalloc(&tb->defer, (size_t)kDeferCap * sizeof(int));
  cudaMalloc(&tb->defer_n, sizeof(int));
  cudaMemset(tb->defer_n, 0, sizeof(int));
  cudaFuncSetAttribute(k_root_sums, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem);
  cudaFuncSetAttribute(k_node_sums_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem);
  if (h->precision == NV_PREC_MIXED) {
    cudaMalloc(&tb->mx.C, (size_t)tb->max_nodes * sizeof(double4));
    cudaMalloc(&tb->mx.W, (size_t)tb->max_nodes * sizeof(WalkNode));
    cudaMalloc(&tb->mx.G, (size_t)tb->max_nodes * sizeof(double2));
  }
  cudaMalloc(&tb->ctr, kCtrSize * sizeof(int));
  cudaMemset(tb->ctr, 0, kCtrSize * sizeof(int));
  tb->max_blk = (int)(T / (kBigNode + 1) + h->nsys + 64);
  tb->max_wrp = (int)(T / 2 + h->nsys + 64);
  for (int b = 0; b < 3; ++b) {
    cudaMalloc(&tb->split_blk[b], (size_t)tb->max_blk * sizeof(int));
    cudaMalloc(&tb->split_wrp[b], (size_t)tb->max_wrp * sizeof(int));
  }
  for (int b = 0; b < 2; ++b) {
    cudaMalloc(&tb->okey[b], (size_t)T * sizeof(unsigned long long));
    cudaMalloc(&tb->oval[b], (size_t)T * sizeof(int));
  }
  tb->perm = tb->oval[1];
  cudaMalloc(&tb->iperm, (size_t)T * sizeof(int));
  k_iota<<<grid_for(T, TB), TB, 0, h->stream>>>(tb->perm, T);  // a permutation before the first build
  int sb = 1;
  while ((1LL << sb) < h->nsys) ++sb;
  tb->key_bits = 34 + sb;
  cub::DeviceRadixSort::SortPairs(nullptr, tb->sort_bytes, tb->okey[0], tb->okey[1], tb->oval[0], tb->oval[1], (int)T,
                                  0, tb->key_bits);
  cudaMalloc(&tb->sort_tmp, std::max<size_t>(tb->sort_bytes, 16));
  double widest = 1.;  // box over segment length of the systems with a tree
  for (auto &s : h->sc)
    if ((s.use_tree || s.sched_tree) && s.delta > 0.) widest = std::max(widest, s.bsize / s.delta);
  tb->grid_levels = std::min(kMaxLevels, std::max(2, (int)std::ceil(std::log2(std::min(widest, 1e9))) + 3));
  h->tree = tb;
}

void tree_free(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb) return;
  void *ptrs[] = {tb->nA, tb->nB, tb->nP, tb->nI, tb->nR, tb->nDepth, tb->nLeaf, tb->nKids, tb->members, tb->bigl, tb->root_apx, tb->root_part, tb->defer, tb->defer_n,
                  tb->rdig, tb->rrank, tb->root_rank, tb->root_mb, tb->root_ok, tb->pass_state, tb->pass_ctl, tb->ctr,
                  tb->mx.C, tb->mx.W, tb->mx.G, tb->okey[0], tb->okey[1],
                  tb->oval[0], tb->oval[1], tb->iperm, tb->sort_tmp, tb->split_blk[0], tb->split_blk[1],
                  tb->split_blk[2], tb->split_wrp[0], tb->split_wrp[1], tb->split_wrp[2]};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  delete tb;
  h->tree = nullptr;
}

void launch_tree_build(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb) return;
  const long long T = h->T;
  k_root_lists<<<pass_blocks(T), kPassThreads, 0, h->stream>>>(h->d_sc, h->d_dyn, h->sys_of, h->x, h->nxt, *tb, h->nsys,
                                                               T, h->d_err);
  k_roots<<<grid_for(h->nsys, 64), 64, 0, h->stream>>>(h->d_sc, h->d_dyn, h->nsys, h->nxt, *tb, h->d_err);
  // the roots' estimates, the walk order and the roots' exact sums (one long sequential chain per
  // system) run on the side stream; the walks wait for the first two, the fix-up of deferred root tests
  // and the closest-point walk for the sums
  cudaEventRecord(h->fork_ev, h->stream);
  cudaStreamWaitEvent(h->side, h->fork_ev, 0);
  k_root_partial<<<h->nsys * tb->root_parts, 256, 0, h->side>>>(h->x, T, *tb, h->nsys, tb->root_parts);
  k_root_approx<<<grid_for(32LL * h->nsys, 128), 128, 0, h->side>>>(*tb, h->nsys, tb->root_parts, h->root_band_scale);
  k_order_keys<<<grid_for(T, TB), TB, 0, h->side>>>(h->d_sc, h->d_dyn, h->sys_of, h->x, h->nxt, tb->okey[0],
                                                    tb->oval[0], T);
  {
    size_t sb = tb->sort_bytes;
    cub::DeviceRadixSort::SortPairs(tb->sort_tmp, sb, tb->okey[0], tb->okey[1], tb->oval[0], tb->oval[1], (int)T, 0,
                                    tb->key_bits, h->side);
  }
  k_inv_perm<<<grid_for(T, TB), TB, 0, h->side>>>(tb->perm, tb->iperm, T);
  cudaEventRecord(h->sort_ev, h->side);
  k_root_sums<<<h->nsys, kSumThreads, kSumSmem, h->side>>>(h->x, T, *tb, h->nsys, h->nxt, h->d_err);
  cudaEventRecord(h->join_ev, h->side);
  const int sms = n_sms();
  k_root_scatter<<<grid_for(T, TB), TB, 0, h->stream>>>(h->sys_of, *tb, h->nsys, h->d_err);
  // the big depth-1 nodes' sums (the longest sequential chains after the roots') start as soon
  // as the roots' split has listed them and written their member lists, beside the levels
  cudaEventRecord(h->fork2_ev, h->stream);
  cudaStreamWaitEvent(h->side2, h->fork2_ev, 0);
  k_node_sums_block<<<sms, kSumThreads, kSumSmem, h->side2>>>(h->x, h->gi, h->nxt, T, *tb, 0, h->d_err);
  cudaEventRecord(h->join2_ev, h->side2);
  // A launch per level down to cells of about an eighth of delta, one for the rest (32,768 points,
  // 41 launches 172 us, now 9 in 122 us and the one in 2.8; 1,048,576 points, 10 and 22 us)
  for (int L = 1; L < tb->grid_levels; ++L)
    k_split_level<<<sms, kSplitThreads, 0, h->stream>>>(h->x, T, *tb, L, h->d_err);
  k_split_rest<<<sms, kSplitThreads, 0, h->stream>>>(h->x, T, *tb, tb->grid_levels, h->d_err);
  k_node_sums_block<<<sms, kSumThreads, kSumSmem, h->stream>>>(h->x, h->gi, h->nxt, T, *tb, 1, h->d_err);
  k_node_sums_big<<<sms * 8, 128, 0, h->stream>>>(h->x, h->gi, h->nxt, T, *tb, h->nsys, h->d_err);
  k_node_sums_small<<<sms * 8, 128, 0, h->stream>>>(h->x, h->gi, h->nxt, T, *tb, h->nsys, h->d_err);
  cudaStreamWaitEvent(h->stream, h->sort_ev, 0);
  cudaStreamWaitEvent(h->stream, h->join2_ev, 0);
  if (h->precision == NV_PREC_MIXED) {
    // theta0 and the correction flag are per system; a handle's systems share them when
    // any of them walks the tree (checked at creation)
    k_node_prep<<<sms * 4, 256, 0, h->stream>>>(*tb, h->nsys, h->sc[h->tree_sys0].tree_theta,
                                                h->sc[h->tree_sys0].tree_extra_correction, h->prv);
    tb->prep_epoch = h->links_epoch;
  }
  tb->built = true;
}

void join_root_sums(nv_handle *h) {
  if (h->tree) cudaStreamWaitEvent(h->stream, h->join_ev, 0);
}

void launch_walk_fixup(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb) return;
  join_root_sums(h);
  k_walk_fixup<<<n_sms(), 128, 0, h->stream>>>(h->d_sc, h->d_dyn, h->sys_of, h->x, h->gi, h->gb, h->prv, h->u,
                                               h->partial, h->T, *tb, h->d_err);
}

void launch_tree_walk(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb || h->n_work_tree == 0) return;
  if (h->any_mirror) {  // solid walls: the mirrored trees first, on the roots' exact centres
    join_root_sums(h);
    k_tree_walk_mirror<<<h->n_work_tree, 64, 0, h->stream>>>(h->d_sc, h->d_dyn, h->d_work_tree, h->x, h->nxt, h->prv,
                                                             h->T, *tb, h->d_err);
  }
  cudaMemsetAsync(tb->defer_n, 0, sizeof(int), h->stream);
  // two threads per target up to 20 blocks of targets an SM (automatic), or as
  // nv_set_walk_parts asks: 100,000 points 4.37 ms (4.58 with one), 262,144 points 5.85 ms (5.37)
  const int split = h->walk_parts == 0 ? h->n_work_tree < 20 * n_sms() : h->walk_parts > 1;
  k_tree_walk_fp64<<<h->n_work_tree, split ? 128 : 64, 0, h->stream>>>(
      h->d_sc, h->d_dyn, h->d_work_tree, h->x, h->gi, h->gb, h->nxt, h->prv, h->u, h->T, *tb, split, h->d_err);
}

namespace {
template <int W>
void launch_walk(nv_handle *h) {
  k_tree_walk_mixed<W><<<h->n_work_grp, 32 * W, sizeof(WalkShared<W>), h->stream>>>(
      h->d_sc, h->d_dyn, h->d_work_grp, h->x, h->nxt, h->prv, h->partial, h->T, *h->tree, h->near_factor, h->guards,
      h->d_err);
}
template <int W>
cudaError_t allow_walk() {
  return cudaFuncSetAttribute(k_tree_walk_mixed<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WalkShared<W>));
}
}  // namespace

cudaError_t tree_kernels_setup() {
  for (cudaError_t e : {allow_walk<1>(), allow_walk<2>(), allow_walk<4>(), allow_walk<8>()})
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

void launch_tree_walk_mixed(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb || h->n_work_grp == 0) return;
  if (tb->prep_epoch != h->links_epoch) {  // relinked since the build
    k_leaf_links<<<n_sms() * 4, 256, 0, h->stream>>>(*tb, h->nsys, h->prv);
    tb->prep_epoch = h->links_epoch;
  }
  cudaMemsetAsync(tb->defer_n, 0, sizeof(int), h->stream);
  switch (h->walk_parts_used) {
    case 1: launch_walk<1>(h); break;
    case 2: launch_walk<2>(h); break;
    case 4: launch_walk<4>(h); break;
    default: launch_walk<8>(h); break;
  }
}

void launch_closest_tree(nv_handle *h) {
  TreeBuffers *tb = h->tree;
  if (!tb) return;
  join_root_sums(h);
  // successor prefetch while the targets fill the GPU less than ~8 blocks per SM
  auto walk = h->T < 8LL * 128 * n_sms() ? k_closest_tree<true> : k_closest_tree<false>;
  walk<<<grid_for(h->T, 128), 128, 0, h->stream>>>(h->d_sc, h->d_dyn, h->sys_of, h->x, h->nxt, h->prv, h->closest,
                                                   h->closestd, h->T, *tb, h->d_err);
}

// Preorder dump of system `sys`'s tree (host side: download nodes, follow first_child/skip).
int tree_dump(nv_handle *h, int sys, void *buf, int cap, int *n) {
  TreeBuffers *tb = h->tree;
  if (!tb || !tb->built) return set_error(NV_ERR_STATE, "no tree has been built");
  cudaStreamSynchronize(h->stream);
  int nn = 0;
  NV_CUDA(cudaMemcpy(&nn, tb->ctr, sizeof(int), cudaMemcpyDeviceToHost));
  std::vector<double4> A(nn), B(nn), P(nn);
  std::vector<int4> I(nn);
  std::vector<int> D(nn), Lf(nn);
  NV_CUDA(cudaMemcpy(A.data(), tb->nA, nn * sizeof(double4), cudaMemcpyDeviceToHost));
  NV_CUDA(cudaMemcpy(B.data(), tb->nB, nn * sizeof(double4), cudaMemcpyDeviceToHost));
  NV_CUDA(cudaMemcpy(P.data(), tb->nP, nn * sizeof(double4), cudaMemcpyDeviceToHost));
  NV_CUDA(cudaMemcpy(I.data(), tb->nI, nn * sizeof(int4), cudaMemcpyDeviceToHost));
  NV_CUDA(cudaMemcpy(D.data(), tb->nDepth, nn * sizeof(int), cudaMemcpyDeviceToHost));
  NV_CUDA(cudaMemcpy(Lf.data(), tb->nLeaf, nn * sizeof(int), cudaMemcpyDeviceToHost));
  struct Rec {
    double pos[3], width, cent[3], circ[3];
    int32_t pcount, depth, leaf, first_next;
  };
  Rec *out = static_cast<Rec *>(buf);
  const int base = h->base[sys];
  int m = 0;
  for (int node = sys; node != kEnd;) {
    if (out && m < cap) {
      Rec &r = out[m];
      r.pos[0] = P[node].x; r.pos[1] = P[node].y; r.pos[2] = P[node].z;
      r.width = A[node].w;
      r.cent[0] = A[node].x; r.cent[1] = A[node].y; r.cent[2] = A[node].z;
      r.circ[0] = B[node].x; r.circ[1] = B[node].y; r.circ[2] = B[node].z;
      r.pcount = I[node].x;
      r.depth = D[node];
      r.leaf = Lf[node] ? Lf[node] - base : 0;
      r.first_next = I[node].w ? I[node].w - base : 0;
    }
    ++m;
    node = (I[node].x > 1 && I[node].y != kEnd) ? I[node].y : I[node].z;
  }
  *n = m;
  return NV_OK;
}
