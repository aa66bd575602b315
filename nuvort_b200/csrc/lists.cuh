// lists.cuh -- ordered lists of slots by one launch (a stable compaction into K lists).
#pragma once

#include "common.cuh"

// flags(g), for 0 <= g <= n, gives a word whose bits 0..K-1 say which lists slot g is in;
// put(g, k, p, word) is then called for every slot and list, p the number of list k's slots below
// g.  A block takes 1,024 consecutive slots (by a ticket, so that the blocks before it have
// started), counts its bits, and finds the sum of the blocks before it by looking back: every
// block publishes its own sum and, once known, its inclusive sum, each in one 64-bit word with
// the launch's epoch, so that nothing is cleared between launches (the last block to finish
// sets up the next).  One launch for what a flag kernel, a two-kernel scan and a scatter did in
// four per list.
constexpr int kPassThreads = 256, kPassItems = 4, kPassSlots = kPassThreads * kPassItems;
constexpr int kPassPolls = 1 << 22;  // polls of a predecessor before giving up

struct PassBuffers {
  unsigned long long *state;  // [K][blocks]
  unsigned *ctl;              // ticket, finished blocks, epoch
};
// The launch's epoch (below 2^30), the same to all its threads until they have called flags for
// their last slot.
__device__ __forceinline__ unsigned pass_epoch(const PassBuffers &L) { return *(const volatile unsigned *)&L.ctl[2]; }
inline int pass_blocks(long long n) { return (int)((n + kPassSlots) / kPassSlots); }  // slots 0..n
inline void pass_alloc(unsigned long long **state, unsigned **ctl, int K, long long n) {
  const size_t words = (size_t)K * pass_blocks(n);
  cudaMalloc(state, words * sizeof(unsigned long long));
  cudaMemset(*state, 0, words * sizeof(unsigned long long));
  cudaMalloc(ctl, 3 * sizeof(unsigned));
  cudaMemset(*ctl, 0, 3 * sizeof(unsigned));
}

template <int K, class F, class Put>
__device__ void ordered_pass(const PassBuffers &L, long long n, unsigned *err, F flags, Put put) {
  constexpr int kWarps = kPassThreads / 32;
  __shared__ int s_block, s_sum[K][kWarps], s_base[K];
  __shared__ unsigned s_epoch;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) {
    s_epoch = *(volatile unsigned *)&L.ctl[2];
    s_block = (int)atomicAdd(&L.ctl[0], 1u);
  }
  __syncthreads();
  const int b = s_block, nb = gridDim.x;
  const unsigned epoch = s_epoch;
  const long long g0 = (long long)b * kPassSlots + wid * (32 * kPassItems) + lane;
  unsigned m[K][kPassItems], f[kPassItems];
#pragma unroll
  for (int it = 0; it < kPassItems; ++it) {
    const long long g = g0 + 32 * it;
    f[it] = g <= n ? flags(g) : 0u;
#pragma unroll
    for (int k = 0; k < K; ++k) m[k][it] = __ballot_sync(0xffffffffu, (f[it] >> k) & 1u);
  }
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      int v = 0;
#pragma unroll
      for (int it = 0; it < kPassItems; ++it) v += __popc(m[k][it]);
      s_sum[k][wid] = v;
    }
  __syncthreads();
  for (int k = wid; k < K; k += kWarps) {  // a warp per list: its bits before this block
    volatile unsigned long long *st = L.state + (long long)k * nb;
    auto word = [&](unsigned flag, int v) {
      return (unsigned long long)((epoch << 2) | flag) << 32 | (unsigned long long)(unsigned)v;
    };
    int own = 0;
    for (int w = 0; w < kWarps; ++w) own += s_sum[k][w];
    if (lane == 0) st[b] = word(b == 0 ? 2u : 1u, own);
    int before = 0;
    bool ok = true;
    for (int j = b - 1; j >= 0 && ok; j -= 32) {
      const int q = j - lane;
      unsigned long long v = word(2u, 0);  // before the first block: an inclusive sum of 0
      int polls = 0;
      for (;;) {
        if (q >= 0) v = st[q];
        const unsigned tag = (unsigned)(v >> 32);
        const bool ready = (tag >> 2) == (epoch & 0x3fffffffu) && (tag & 3u);
        if (__all_sync(0xffffffffu, ready)) break;
        if (++polls > kPassPolls) {
          ok = false;
          break;
        }
      }
      const unsigned incl = __ballot_sync(0xffffffffu, ((unsigned)(v >> 32) & 3u) == 2u);
      const int stop = incl ? __ffs(incl) - 1 : 31;
      int x = lane <= stop ? (int)(unsigned)v : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      before += x;
      if (incl) break;
    }
    if (lane == 0) {
      if (!ok) {
        atomicOr(err, DERR_TIMEOUT);
        before = 0;
      }
      if (b > 0) st[b] = word(2u, before + own);
      s_base[k] = before;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    int off = s_base[k];
    for (int w = 0; w < wid; ++w) off += s_sum[k][w];
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) {
      const long long g = g0 + 32 * it;
      const int p = off + __popc(m[k][it] & ((1u << lane) - 1u));
      if (g <= n) put(g, k, p, f[it]);
      off += __popc(m[k][it]);
    }
  }
  if (tid == 0 && atomicAdd(&L.ctl[1], 1u) == (unsigned)nb - 1) {  // every block has taken its ticket and epoch
    L.ctl[0] = 0;
    L.ctl[1] = 0;
    L.ctl[2] = (epoch + 1) & 0x3fffffffu;
  }
}

// The slots with bit k in ascending order in list[k], the number of them below g in pos[k][g].
template <int K>
struct Lists {
  int *pos[K], *list[K];
  PassBuffers buf;
};
template <int K, class F>
__device__ __forceinline__ void ordered_lists(const Lists<K> &L, long long n, unsigned *err, F flags) {
  ordered_pass<K>(L.buf, n, err, flags, [&](long long g, int k, int p, unsigned word) {
    L.pos[k][g] = p;
    if ((word >> k) & 1u) L.list[k][p] = (int)g;
  });
}
