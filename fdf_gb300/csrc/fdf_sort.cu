// fdf_sort.cu -- per-step re-sort of the particles by cell (a counting sort).
//
//   1. the locate kernel histograms the new cell keys (count[c], integer atomics,
//      warp-aggregated: exact and order-independent);
//   2. an exclusive scan turns count[0..Nc+1) into cell_start[0..Nc+1]: cell c
//      owns sorted slots [cell_start[c], cell_start[c+1]); bucket Nc holds the LOST
//      particles the initial setup keeps, and removed particles get no slot;
//   3. each particle takes slot cell_start[key] + its rank within its cell, which the
//      histogram atomic of step 1 returned;
//   4. each cell's slots are then ordered by (PID, previous slot) in the plain form, so
//      the final order -- and every later sum -- is the same on every run, whatever
//      order the atomics took, and does not depend on the history of the swarm: sorted
//      order is (cell, PID), the order the oracle uses for the face deposits, which makes
//      those sums comparable bit for bit.  The precision forms order each cell's slots by
//      previous slot alone (a stable counting sort: the same on every run for the same
//      input, and no gather of the PIDs), as does the standalone sort.
#include "fdf_internal.cuh"
#include "fdf_counters.cuh"

#include <algorithm>

namespace {

// ---- exclusive scan of a u32 array (reduce -> scan of block sums -> scan with offsets) ----
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_BLOCK = SCAN_THREADS * SCAN_ITEMS;   // 8192 values per block
constexpr int SUMS_PER_THREAD = 16;                      // up to 16384 blocks -> 134M values

__device__ __forceinline__ unsigned int block_exclusive_scan(unsigned int v, unsigned int *total) {
  __shared__ unsigned int warp_tot[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    unsigned int t = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    warp_tot[lane] = t;  // inclusive
  }
  __syncthreads();
  unsigned int warp_prefix = wid ? warp_tot[wid - 1] : 0u;
  if (total) *total = warp_tot[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

// Loads SCAN_ITEMS (= 8) consecutive values as two 16-B vectors when the block is
// fully inside and the base is aligned, element by element otherwise.
__device__ __forceinline__ void load8(const unsigned int *__restrict__ in, long long base, long long count,
                                      unsigned int v[SCAN_ITEMS]) {
  if (base + SCAN_ITEMS <= count && ((reinterpret_cast<size_t>(in + base) & 15) == 0)) {
    const uint4 a = *reinterpret_cast<const uint4 *>(in + base);
    const uint4 b = *reinterpret_cast<const uint4 *>(in + base + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int q = 0; q < SCAN_ITEMS; ++q) v[q] = (base + q < count) ? in[base + q] : 0u;
  }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const unsigned int *__restrict__ in, long long count,
                                                             unsigned int *__restrict__ sums) {
  long long base = (long long)blockIdx.x * SCAN_BLOCK + (long long)threadIdx.x * SCAN_ITEMS;
  unsigned int v[SCAN_ITEMS], t = 0;
  load8(in, base, count, v);
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) t += v[q];
  unsigned int tot;
  block_exclusive_scan(t, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(unsigned int *sums, int nsums) {
  int base = threadIdx.x * SUMS_PER_THREAD;
  unsigned int v[SUMS_PER_THREAD], t = 0;
#pragma unroll
  for (int q = 0; q < SUMS_PER_THREAD; ++q) { v[q] = (base + q < nsums) ? sums[base + q] : 0u; t += v[q]; }
  unsigned int ex = block_exclusive_scan(t, nullptr);
#pragma unroll
  for (int q = 0; q < SUMS_PER_THREAD; ++q) {
    if (base + q < nsums) sums[base + q] = ex;
    ex += v[q];
  }
}

// out = exclusive scan of in (out == in allowed).  DIRECT: sums holds the blocks' own sums and each
// block adds up those before it, which spares the launch that scans them; clear: `in` is left zero
// (the histogram of the next step).
template <bool DIRECT>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(unsigned int *in, unsigned int *out, long long count,
                                                            const unsigned int *__restrict__ sums, int clear) {
  long long base = (long long)blockIdx.x * SCAN_BLOCK + (long long)threadIdx.x * SCAN_ITEMS;
  unsigned int v[SCAN_ITEMS], t = 0;
  load8(in, base, count, v);
  unsigned int before;
  if (DIRECT) {
    unsigned int part = 0;
    for (int q = threadIdx.x; q < (int)blockIdx.x; q += SCAN_THREADS) part += sums[q];
    block_exclusive_scan(part, &before);
  } else {
    before = sums[blockIdx.x];
  }
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) t += v[q];
  unsigned int ex = block_exclusive_scan(t, nullptr) + before;
  unsigned int o[SCAN_ITEMS];
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) { o[q] = ex; ex += v[q]; }
  if (base + SCAN_ITEMS <= count && ((reinterpret_cast<size_t>(in + base) | reinterpret_cast<size_t>(out + base)) & 15) == 0) {
    *reinterpret_cast<uint4 *>(out + base) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4 *>(out + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
    if (clear) {
      *reinterpret_cast<uint4 *>(in + base) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4 *>(in + base + 4) = make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
#pragma unroll
    for (int q = 0; q < SCAN_ITEMS; ++q)
      if (base + q < count) {
        out[base + q] = o[q];
        if (clear) in[base + q] = 0u;
      }
  }
}

// Slot of every kept particle: cell_start[key] + its rank among the particles of the same
// key, which the locate kernels took from their histogram atomics.  Each thread handles
// FDF_SCATTER_ITEMS particles (strided by the block, so every load stays coalesced) and issues
// all their loads before their stores: the cell_start gather depends on the key, so a thread
// with one particle waits two load latencies for one store (sort stage per 64M-particle step:
// 0.78 ms with one particle per thread, 0.66 with 2, 0.61 with 4, 0.63 with 8).
#ifndef FDF_SCATTER_ITEMS
#define FDF_SCATTER_ITEMS 4
#endif
// The last block folds the counters' flush rows instead (the walk has ended): a launch of its own
// took 13 us at the end of every step, this runs beside the slots.
__global__ void __launch_bounds__(256) k_scatter_slots(const unsigned int *__restrict__ keys,
                                                      const unsigned int *__restrict__ rank, DevCounters *cnt,
                                                      unsigned int sentinel, int keep_lost,
                                                      const unsigned int *__restrict__ cell_start,
                                                      unsigned int *__restrict__ perm) {
  if (blockIdx.x == gridDim.x - 1) {
    fold_counts(cnt);
    return;
  }
  constexpr int IT = FDF_SCATTER_ITEMS;
  const long long n = cnt->n_sorted;
  const long long base = (long long)blockIdx.x * IT * blockDim.x + threadIdx.x;
  unsigned int key[IT], start[IT], rk[IT];
  bool keep[IT];
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    const long long s = base + (long long)q * blockDim.x;
    key[q] = s < n ? keys[s] : 0xffffffffu;   // sentinel: a LOST particle kept at the end; above: removed
    keep[q] = key[q] < sentinel || (key[q] == sentinel && keep_lost);
  }
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    const long long s = base + (long long)q * blockDim.x;
    start[q] = keep[q] ? cell_start[key[q]] : 0u;
    rk[q] = keep[q] ? rank[s] : 0u;
  }
#pragma unroll
  for (int q = 0; q < IT; ++q)
    if (keep[q]) perm[start[q] + rk[q]] = (unsigned int)(base + (long long)q * blockDim.x);
}

// Orders every cell's slots by (PID, previous slot), or by previous slot alone: the keys are then
// the slots themselves, one 32-bit word per entry and no gather.  One thread per cell; a cell's
// entries decide who works on it:
//   up to 8    its thread: a 19-comparator sorting network in registers (two or four cells per
//              thread, their loads issued first, measured no faster);
//   9 to 32    its warp, one lane per entry (two cells at a time up to 16): a bitonic network of
//              shuffles, the next cells' entries already loading;
//   33 to 128  its warp, in shared memory;
//   above      its block, together: in shared memory (up to SEG_SHARED entries) or in place in
//              global memory.
// (A thread's own insertion sort in global memory, which the cells above 8 took before, is a chain of
// dependent loads.  Sort stage per step, before -> now: 64M particles, 4.5 per cell, by slot
// 0.51 -> 0.45 ms, by PID 1.28 -> 1.17 ms; 32M particles, 27 per cell, 0.49 -> 0.34 and
// 1.60 -> 0.65 ms.)
constexpr int SEG_NET = 8, SEG_WARP = 128, SEG_SHARED = 1024;

// The key of slot v: its PID and then the slot, or the slot alone.
template <bool PID>
struct SlotKey {
  long long pid;
  unsigned int slot;
  __device__ __forceinline__ bool after(const SlotKey &o) const { return pid > o.pid || (pid == o.pid && slot > o.slot); }
};
template <>
struct SlotKey<false> {
  unsigned int slot;
  __device__ __forceinline__ bool after(const SlotKey &o) const { return slot > o.slot; }
};
template <bool PID>
__device__ __forceinline__ SlotKey<PID> slot_key(unsigned int v, const long long *__restrict__ pid) {
  SlotKey<PID> k;
  if constexpr (PID) k.pid = __ldg(pid + v);
  k.slot = v;
  return k;
}

template <bool PID>
__device__ __forceinline__ SlotKey<PID> last_key() {   // sorts after every slot's (slots are below 2^31)
  SlotKey<PID> k;
  if constexpr (PID) k.pid = 0x7fffffffffffffffLL;
  k.slot = 0xffffffffu;
  return k;
}

// Ascending bitonic sort of the n items that get(i) reads and set(i, item) writes, by `many` threads
// of which this is number `me`: the form whose comparators all point the same way, so that the
// items past n of the next power of two need not exist.
template <typename Get, typename Set, typename Sync>
__device__ __forceinline__ void bitonic(unsigned int n, unsigned int me, unsigned int many, Get get, Set set,
                                        Sync sync) {
  unsigned int P = 1;
  while (P < n) P <<= 1;
  auto exchange = [&](unsigned int i, unsigned int j) {
    if (j >= n) return;
    const auto x = get(i), y = get(j);
    if (x.after(y)) {
      set(i, y);
      set(j, x);
    }
  };
  for (unsigned int h = 2; h <= P; h <<= 1) {
    for (unsigned int t = me; t < P / 2; t += many) {   // mirrored halves of each h items
      const unsigned int o = t & (h / 2 - 1), q = 2 * (t - o);
      exchange(q + o, q + h - 1 - o);
    }
    sync();
    for (unsigned int d = h / 4; d >= 1; d >>= 1) {
      for (unsigned int t = me; t < P / 2; t += many) {
        const unsigned int o = t & (d - 1), q = 2 * (t - o);
        exchange(q + o, q + o + d);
      }
      sync();
    }
  }
}
template <typename Get, typename Set>
__device__ __forceinline__ void block_bitonic(unsigned int n, Get get, Set set) {
  bitonic(n, threadIdx.x, blockDim.x, get, set, [] { __syncthreads(); });
}

// One key per lane, ascending within each group of W lanes.
template <int W, bool PID>
__device__ __forceinline__ void lane_bitonic(SlotKey<PID> &k, int lane) {
#pragma unroll
  for (int h = 2; h <= W; h <<= 1)
#pragma unroll
    for (int d = h >> 1; d > 0; d >>= 1) {
      SlotKey<PID> o;
      o.slot = __shfl_xor_sync(0xffffffffu, k.slot, d);
      if constexpr (PID) o.pid = __shfl_xor_sync(0xffffffffu, k.pid, d);
      const bool up = h == W || (lane & h) == 0, low = (lane & d) == 0;
      if constexpr (PID) {
        if (k.after(o) == (up == low)) k = o;   // equal keys only among the padding
      } else {
        k.slot = up == low ? min(k.slot, o.slot) : max(k.slot, o.slot);
      }
    }
}

// The cells of `todo` (a lane mask; each lane holds its own cell's start s0 and length L <= W),
// 32 / W at a time.
template <int W, bool PID>
__device__ __forceinline__ void order_lanes(unsigned int todo, unsigned int s0, unsigned int L, int lane,
                                            const long long *__restrict__ pid, unsigned int *__restrict__ perm) {
  const int group = lane / W, at = lane % W;
  unsigned int q0 = 0u, n = 0u, v = 0u;
  // takes this group's next cell out of `todo` and starts loading its entries
  auto take = [&](unsigned int &q, unsigned int &m, unsigned int &e) {
    unsigned int mine = 0u;
#pragma unroll
    for (int g = 0; g < 32 / W; ++g) {
      if (g == group) mine = todo;
      todo &= todo - 1u;   // 0 stays 0
    }
    const int who = mine ? __ffs((int)mine) - 1 : 0;
    q = __shfl_sync(0xffffffffu, s0, who);
    m = __shfl_sync(0xffffffffu, L, who);
    if (!mine) m = 0u;
    e = at < (int)m ? perm[q + at] : 0u;
  };
  take(q0, n, v);
  while (__any_sync(0xffffffffu, n != 0u)) {
    SlotKey<PID> k = at < (int)n ? slot_key<PID>(v, pid) : last_key<PID>();
    const unsigned int w0 = q0, wn = n, was = v;
    take(q0, n, v);
    lane_bitonic<W, PID>(k, lane);
    if (at < (int)wn && k.slot != was) perm[w0 + at] = k.slot;
  }
}

template <bool PID>
__global__ void __launch_bounds__(256, FDF_ORDER_MIN_BLOCKS) k_order_segments(const unsigned int *__restrict__ cell_start,
                                                                             int nseg,
                                                                             const long long *__restrict__ pid,
                                                                             unsigned int *__restrict__ perm) {
  using Key = SlotKey<PID>;
  __shared__ unsigned int big[256][2], nbig;
  __shared__ Key item[SEG_SHARED];
  static_assert(SEG_SHARED == 8 * SEG_WARP, "one warp's part each, or the block's");
  const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  unsigned int s0 = 0u, L = 0u;
  if (c < nseg) {
    s0 = cell_start[c];
    L = cell_start[c + 1] - s0;
  }
  if (L >= 2u && L <= (unsigned int)SEG_NET) {
    Key k[SEG_NET];
    bool sorted = true;
#pragma unroll
    for (int e = 0; e < SEG_NET; ++e) {
      k[e] = last_key<PID>();
      if (e < (int)L) {
        k[e] = slot_key<PID>(perm[s0 + e], pid);
        if (e > 0 && k[e - 1].after(k[e])) sorted = false;
      }
    }
    if (!sorted) {
      auto cx = [&](int a, int b) {
        const Key x = k[a], y = k[b];
        if constexpr (PID) {
          const bool sw = x.after(y);
          k[a] = sw ? y : x;
          k[b] = sw ? x : y;
        } else {
          k[a].slot = min(x.slot, y.slot);
          k[b].slot = max(x.slot, y.slot);
        }
      };
      cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
      cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
      cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
      cx(2, 4); cx(3, 5);
      cx(1, 4); cx(3, 6);
      cx(1, 2); cx(3, 4); cx(5, 6);
#pragma unroll
      for (int e = 0; e < SEG_NET; ++e)
        if (e < (int)L) perm[s0 + e] = k[e].slot;
    }
  }
  const unsigned int w16 = __ballot_sync(0xffffffffu, L > (unsigned int)SEG_NET && L <= 16u);
  const unsigned int w32 = __ballot_sync(0xffffffffu, L > 16u && L <= 32u);
  if (w16) order_lanes<16, PID>(w16, s0, L, lane, pid, perm);
  if (w32) order_lanes<32, PID>(w32, s0, L, lane, pid, perm);
  for (unsigned int todo = __ballot_sync(0xffffffffu, L > 32u && L <= (unsigned int)SEG_WARP); todo; todo &= todo - 1u) {
    const int who = __ffs((int)todo) - 1;
    const unsigned int q0 = __shfl_sync(0xffffffffu, s0, who), n = __shfl_sync(0xffffffffu, L, who);
    Key *mine = item + (threadIdx.x >> 5) * SEG_WARP;
    for (unsigned int e = lane; e < n; e += 32) mine[e] = slot_key<PID>(perm[q0 + e], pid);
    __syncwarp();
    bitonic(n, (unsigned int)lane, 32u, [&](unsigned int i) { return mine[i]; },
            [&](unsigned int i, const Key &x) { mine[i] = x; }, [] { __syncwarp(); });
    for (unsigned int e = lane; e < n; e += 32) perm[q0 + e] = mine[e].slot;
    __syncwarp();
  }
  if (threadIdx.x == 0) nbig = 0u;
  if (!__syncthreads_or(L > (unsigned int)SEG_WARP)) return;
  if (L > (unsigned int)SEG_WARP) {
    const unsigned int at = atomicAdd(&nbig, 1u);   // any order: each cell is sorted by itself
    big[at][0] = s0;
    big[at][1] = L;
  }
  __syncthreads();
  const unsigned int many = nbig;
  for (unsigned int q = 0; q < many; ++q) {
    const unsigned int q0 = big[q][0], n = big[q][1];
    if (n <= (unsigned int)SEG_SHARED) {
      for (unsigned int e = threadIdx.x; e < n; e += blockDim.x) item[e] = slot_key<PID>(perm[q0 + e], pid);
      __syncthreads();
      block_bitonic(n, [&](unsigned int i) { return item[i]; }, [&](unsigned int i, const Key &v) { item[i] = v; });
      for (unsigned int e = threadIdx.x; e < n; e += blockDim.x) perm[q0 + e] = item[e].slot;
      __syncthreads();
    } else {
      block_bitonic(n, [&](unsigned int i) { return slot_key<PID>(perm[q0 + i], pid); },
                    [&](unsigned int i, const Key &v) { perm[q0 + i] = v.slot; });
    }
  }
}

// The LOST particles that the initial setup and the staged calls keep: one bucket, which may hold a
// few percent of the swarm, ordered like the cells' slots but by the whole GPU.  Chunks of
// LOST_CHUNK entries are sorted in shared memory, then neighbouring runs are merged, twice as long
// each time, between perm and `other` (both indexed like perm): every entry finds its rank in the
// partner run by binary search.  Only the device knows how many there are, so the merges are one
// launch with a barrier of the grid between them (cooperative: one block per SM, all resident): with none
// LOST it costs 2 us at any capacity, where a launch for each merge that the capacity allowed took
// 2.5 us each (removing the LOST of a million slots 153 us against 117 without them).  (A single thread's
// insertion sort took 0.40 s for the 20,000 LOST of 1M particles on the sinusoidal 64x64x1024 grid,
// 0.94 s for the 78,000 of 6M on 96x96x1536.)
constexpr int LOST_CHUNK = 2048, LOST_THREADS = 1024;

// Polls of a barrier before it is given up (seconds; the longest merge, of 2^29 entries, takes a tenth).
constexpr unsigned int LOST_WAIT_LIMIT = 1u << 24;

// Barrier number m of this launch: false (in every thread of the block) when the wait ran out.
__device__ __forceinline__ bool lost_barrier(unsigned int *arrived, int m) {
  __shared__ unsigned int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived + m, 1u);
    unsigned int it = 0;
    while (*reinterpret_cast<volatile unsigned int *>(arrived + m) < gridDim.x && it < LOST_WAIT_LIMIT) ++it;
    ok = it < LOST_WAIT_LIMIT ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  return ok != 0u;
}

template <bool PID>
__global__ void __launch_bounds__(LOST_THREADS, 1) k_order_lost(const unsigned int *__restrict__ bucket,
                                                              const long long *__restrict__ pid, unsigned int *perm,
                                                              unsigned int *other, DevCounters *cnt) {
  using Key = SlotKey<PID>;
  __shared__ Key item[LOST_CHUNK];
  const unsigned int s0 = bucket[0], L = bucket[1] - s0;
  if (L <= 1u) return;
  int merges = 0;
  for (unsigned long long r = LOST_CHUNK; r < L; r <<= 1) ++merges;
  unsigned int *to = merges & 1 ? other : perm, *from = perm;   // the last merge ends in perm
  for (unsigned int c0 = blockIdx.x * LOST_CHUNK; c0 < L; c0 += gridDim.x * LOST_CHUNK) {
    const unsigned int n = min(L - c0, (unsigned int)LOST_CHUNK);
    for (unsigned int e = threadIdx.x; e < n; e += blockDim.x) item[e] = slot_key<PID>(perm[s0 + c0 + e], pid);
    __syncthreads();
    block_bitonic(n, [&](unsigned int i) { return item[i]; }, [&](unsigned int i, const Key &v) { item[i] = v; });
    for (unsigned int e = threadIdx.x; e < n; e += blockDim.x) to[s0 + c0 + e] = item[e].slot;
    __syncthreads();
  }
  if (merges == 0) return;
  const unsigned int stride = gridDim.x * blockDim.x;
  unsigned int run = LOST_CHUNK;
  for (int m = 0; m < merges; ++m, run <<= 1) {
    if (!lost_barrier(cnt->lost_arrived, m)) {
      if (threadIdx.x == 0) atomicOr(&cnt->err, (unsigned int)ERRBIT_SORT_TIMEOUT);
      return;
    }
    from = to;
    to = from == perm ? other : perm;
    for (unsigned int p = blockIdx.x * blockDim.x + threadIdx.x; p < L; p += stride) {
      const unsigned int v = from[s0 + p];
      const Key k = slot_key<PID>(v, pid);
      const unsigned int own = p / run * run, pair = own / (2 * run) * (2 * run);
      unsigned int lo = own == pair ? min(own + run, L) : pair, base = lo;
      unsigned int hi = own == pair ? min(lo + run, L) : own;
      while (lo < hi) {   // the partner's entries before k: keys are distinct (slots differ)
        const unsigned int mid = lo + (hi - lo) / 2;
        if (k.after(slot_key<PID>(from[s0 + mid], pid))) lo = mid + 1;
        else hi = mid;
      }
      to[s0 + pair + (p - own) + (lo - base)] = v;
    }
  }
  // the last block to come here has every block past every barrier: it clears their counts
  if (threadIdx.x == 0 && atomicAdd(cnt->lost_arrived + LOST_BARRIERS, 1u) == gridDim.x - 1) {
    for (int m = 0; m <= LOST_BARRIERS; ++m) cnt->lost_arrived[m] = 0u;
  }
}

template <bool PID>
void order_lost(const unsigned int *bucket, const long long *pid, unsigned int *perm, unsigned int *other, int n_cap,
                DevCounters *cnt, int num_sms, cudaStream_t s) {
  const long long chunks = ((long long)n_cap + LOST_CHUNK - 1) / LOST_CHUNK;
  const unsigned int blocks = (unsigned int)std::min<long long>(std::max<long long>(chunks, 1), num_sms);
  void *args[] = {&bucket, &pid, &perm, &other, &cnt};
  cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_order_lost<PID>), dim3(blocks), dim3(LOST_THREADS), args, 0,
                              s);   // errors through cudaGetLastError
}

// count[cell[s]] += 1 for 0 <= cell[s] < ncells (warp-aggregated integer atomics)
__global__ void __launch_bounds__(256) k_cell_histogram(const int *__restrict__ cell, long long n, long long ncells,
                                                       unsigned int *__restrict__ count) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  unsigned int key = 0xffffffffu;
  if (s < n) {
    const int c = cell[s];
    if (c >= 0 && (long long)c < ncells) key = (unsigned int)c;
  }
  const unsigned int peers = __match_any_sync(0xffffffffu, key);
  if (key != 0xffffffffu && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
    atomicAdd(count + key, (unsigned int)__popc(peers));
}

// count[cell[s]] += 1 as above, and rank[s] = the count before it: a second pass then places the slots
// without atomics.  Each thread handles SORT_ITEMS slots (strided by the block), whose atomics are
// all in flight before the first result is used; equal neighbours of a warp share one (ids as a step
// leaves them come in runs; finding every equal pair of the warp by matching costs more than it saves).
// 16M ids in 4M cells, nearly sorted: 125 us and 111 us for the placing, against 145 us for the histogram
// and 305 us for the slots from a second pass of atomics.
constexpr int SORT_ITEMS = 4;
__global__ void __launch_bounds__(256) k_cell_rank(const int *__restrict__ cell, long long n, long long ncells,
                                                  unsigned int *__restrict__ count, unsigned int *__restrict__ rank) {
  const long long base = (long long)blockIdx.x * SORT_ITEMS * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  unsigned int key[SORT_ITEMS], r[SORT_ITEMS];
  int leader[SORT_ITEMS];
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q) {
    const long long s = base + (long long)q * blockDim.x;
    const int c = s < n ? cell[s] : -1;
    key[q] = c >= 0 && (long long)c < ncells ? (unsigned int)c : 0xffffffffu;
  }
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q) {
    const unsigned int before = __shfl_up_sync(0xffffffffu, key[q], 1);
    const unsigned int heads = __ballot_sync(0xffffffffu, lane == 0 || key[q] != before);
    const unsigned int upto = 0xffffffffu >> (31 - lane), later = heads & ~upto;
    leader[q] = 31 - __clz((int)(heads & upto));
    r[q] = 0u;
    if (leader[q] == lane && key[q] != 0xffffffffu)
      r[q] = atomicAdd(count + key[q], (unsigned int)((later ? __ffs((int)later) - 1 : 32) - lane));
  }
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q) {
    const long long s = base + (long long)q * blockDim.x;
    const unsigned int first = __shfl_sync(0xffffffffu, r[q], leader[q]);
    if (key[q] != 0xffffffffu) rank[s] = first + (unsigned int)(lane - leader[q]);
  }
}

// A tile of TILE ids at a time, for ids nearly in order (a step's ids are: a particle moves a few cells): a block
// whose ids span fewer than TILE_BINS cells counts them in shared memory and adds its counts to count[] cell
// by cell -- neighbouring lanes on neighbouring words, one request where k_cell_rank makes 32.  A block whose ids
// span more merges runs of equal neighbours in a warp, as k_cell_rank does.
//   RANK: rank[s] as k_cell_rank makes it, from the counts before the block's and the id's place in the block.
//   COUNT, then SLOTS (count: the cells' cursors, cell_start before): the second pass counts again and writes the
//   slots, so that nothing is kept per id between the passes and the scratch is a word per cell.
// Bound by the latency of their phases: 32 registers (an id and its place share a word) and four blocks an SM.
// The whole sort, with RANK and with COUNT and SLOTS: 16M nearly sorted ids in 4M cells 191 and 174 us (each call
// after a synchronisation, which gives the scratch back: 408 and 333), 32M in 1M 663 and 628 (1011 and 788), 64M in
// 14M 635 and 542 (1217 and 778); 16M in no order 393 and 397 (608 and 555); but 8M nearly sorted 100 and 104 (251
// and 267), in no order 190 and 201, 4M 64 and 74, 111 and 128: so COUNT and SLOTS from TILE_CURSORS ids on,
// where the ranks take 32 MB, the pool's remapping begins to tell and the ids no longer stay in L2.
// Against k_cell_rank: from three ids per cell on, where a tile of ids in order spans 2731 cells and leaves the
// rest of the bins for its disorder, and from 3M ids, half a wave of blocks: 3.2M nearly sorted by 64 and by 4096
// cells 62 and 80 us against 67 and 93, 6M 80 and 116 against 93 and 137; 6M in no order 142 against 140.
// One atomic per id where a tile spans too much took 16M ids in runs of 8 and 32 at random 298 and 424 us, now
// 180 and 218; one id in 8192 far off 249, now 157.
constexpr int TILE_THREADS = 512, TILE_ITEMS = 16, TILE = TILE_THREADS * TILE_ITEMS, TILE_BINS = 12224;
constexpr long long TILE_MIN = 3 << 20, TILE_CURSORS = 8 << 20;
enum { COUNT, RANK, SLOTS };
template <int WHAT>
__global__ void __launch_bounds__(TILE_THREADS, 4) k_cell_tile(const int *__restrict__ cell, long long n, long long ncells,
                                                             unsigned int *__restrict__ count,
                                                             unsigned int *__restrict__ out) {
  // an id's rank (RANK) or place (SLOTS)
  auto put = [&](long long s, unsigned int at) {
    if (WHAT == RANK) out[s] = at;
    else out[at] = (unsigned int)s;
  };
  __shared__ unsigned int bin[TILE_BINS];
  __shared__ unsigned int span[2];
  const long long base = (long long)blockIdx.x * TILE + threadIdx.x;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) { span[0] = 0xffffffffu; span[1] = 0u; }
  unsigned int key[TILE_ITEMS], lo = 0xffffffffu, hi = 0u;
#pragma unroll
  for (int q = 0; q < TILE_ITEMS; ++q) {
    const long long s = base + q * TILE_THREADS;
    const int c = s < n ? cell[s] : -1;
    key[q] = c >= 0 && (long long)c < ncells ? (unsigned int)c : 0xffffffffu;
  }
#pragma unroll
  for (int q = 0; q < TILE_ITEMS; ++q) {
    lo = min(lo, key[q]);
    if (key[q] != 0xffffffffu) hi = max(hi, key[q]);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  __syncthreads();
  if (lane == 0) { atomicMin(&span[0], lo); atomicMax(&span[1], hi); }
  __syncthreads();
  lo = span[0];
  hi = span[1];
  if (lo == 0xffffffffu) return;   // no id of the block has a cell
  const unsigned int bins = hi - lo + 1u;
  if (bins <= (unsigned int)TILE_BINS) {
    for (unsigned int b = threadIdx.x; b < bins; b += TILE_THREADS) bin[b] = 0u;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TILE_ITEMS; ++q)   // from here on the bin and, above it, the id's place in it
      if (key[q] != 0xffffffffu) {
        key[q] -= lo;
        const unsigned int place = atomicAdd(&bin[key[q]], 1u);
        if (WHAT != COUNT) key[q] |= place << 16;
      }
    __syncthreads();
#pragma unroll 8
    for (unsigned int b = threadIdx.x; b < bins; b += TILE_THREADS) {
      const unsigned int c = bin[b];
      if (c != 0u) {
        const unsigned int before = atomicAdd(count + lo + b, c);
        if (WHAT != COUNT) bin[b] = before;
      }
    }
    if (WHAT == COUNT) return;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TILE_ITEMS; ++q)
      if (key[q] != 0xffffffffu) put(base + q * TILE_THREADS, bin[key[q] & 0xffffu] + (key[q] >> 16));
    return;
  }
  constexpr int IN_FLIGHT = 4;
#pragma unroll
  for (int h = 0; h < TILE_ITEMS; h += IN_FLIGHT) {
    unsigned int at[IN_FLIGHT];
    int leader[IN_FLIGHT];
#pragma unroll
    for (int q = 0; q < IN_FLIGHT; ++q) {
      const unsigned int k = key[h + q], before = __shfl_up_sync(0xffffffffu, k, 1);
      const unsigned int heads = __ballot_sync(0xffffffffu, lane == 0 || k != before);
      const unsigned int upto = 0xffffffffu >> (31 - lane), later = heads & ~upto;
      leader[q] = 31 - __clz((int)(heads & upto));
      at[q] = 0u;
      if (leader[q] == lane && k != 0xffffffffu)
        at[q] = atomicAdd(count + k, (unsigned int)((later ? __ffs((int)later) - 1 : 32) - lane));
    }
    if (WHAT != COUNT) {
#pragma unroll
      for (int q = 0; q < IN_FLIGHT; ++q) {
        const unsigned int first = __shfl_sync(0xffffffffu, at[q], leader[q]);
        if (key[h + q] != 0xffffffffu) put(base + (h + q) * TILE_THREADS, first + (unsigned int)(lane - leader[q]));
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_cell_place(const int *__restrict__ cell, long long n, long long ncells,
                                                   const unsigned int *__restrict__ cell_start,
                                                   const unsigned int *__restrict__ rank,
                                                   unsigned int *__restrict__ perm) {
  const long long base = (long long)blockIdx.x * SORT_ITEMS * blockDim.x + threadIdx.x;
  int c[SORT_ITEMS];
  unsigned int at[SORT_ITEMS];
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q) {
    const long long s = base + (long long)q * blockDim.x;
    c[q] = s < n ? cell[s] : -1;
    if ((long long)c[q] >= ncells) c[q] = -1;
  }
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q)
    at[q] = c[q] >= 0 ? cell_start[c[q]] + rank[base + (long long)q * blockDim.x] : 0u;
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; ++q)
    if (c[q] >= 0) perm[at[q]] = (unsigned int)(base + (long long)q * blockDim.x);
}

// slot of every particle with a valid cell (warp-aggregated cursors, the cells' starts before)
__global__ void __launch_bounds__(256) k_cell_slots(const int *__restrict__ cell, long long n, long long ncells,
                                                   unsigned int *__restrict__ cursor, unsigned int *__restrict__ perm) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  unsigned int key = 0xffffffffu;
  if (s < n) {
    const int c = cell[s];
    if (c >= 0 && (long long)c < ncells) key = (unsigned int)c;
  }
  const unsigned int peers = __match_any_sync(0xffffffffu, key);
  if (key == 0xffffffffu) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  const unsigned int rank = __popc(peers & ((1u << lane) - 1u));
  unsigned int base = 0;
  if (lane == leader) base = atomicAdd(cursor + key, (unsigned int)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  perm[base + rank] = (unsigned int)s;
}

}  // namespace

size_t scan_scratch_words(long long count) { return (size_t)((count + SCAN_BLOCK - 1) / SCAN_BLOCK) + 1; }

long long scan_max_count() { return (long long)SCAN_BLOCK * SCAN_THREADS * SUMS_PER_THREAD; }

// Blocks of a scan whose offsets each block adds up itself, half of the sums on average: up to here (33M
// values, 34 MB of sums read from L2 in all) the launch saved outweighs that.  A sort of 1000 ids, which is
// its scan: 73 us against 75 with three launches in 8M cells, 100 against 103 in 14M, 153 against 158 in 24M,
// 223 against 227 in 33M.
constexpr long long SCAN_DIRECT = 4096;

static int exclusive_scan(unsigned int *in, unsigned int *out, long long count, unsigned int *sums, int clear,
                          cudaStream_t s) {
  const long long blocks = std::max<long long>((count + SCAN_BLOCK - 1) / SCAN_BLOCK, 1);
  k_scan_reduce<<<(unsigned)blocks, SCAN_THREADS, 0, s>>>(in, count, sums);
  if (blocks <= SCAN_DIRECT) {
    k_scan_apply<true><<<(unsigned)blocks, SCAN_THREADS, 0, s>>>(in, out, count, sums, clear);
    return 2;
  }
  k_scan_sums<<<1, SCAN_THREADS, 0, s>>>(sums, (int)blocks);
  k_scan_apply<false><<<(unsigned)blocks, SCAN_THREADS, 0, s>>>(in, out, count, sums, clear);
  return 3;
}

int exclusive_scan_u32(unsigned int *data, long long count, unsigned int *sums, cudaStream_t s) {
  return exclusive_scan(data, data, count, sums, 0, s);
}

int scan_histogram(unsigned int *hist, unsigned int *cell_start, long long count, unsigned int *sums, cudaStream_t s) {
  return exclusive_scan(hist, cell_start, count, sums, 1, s);
}

void launch_scatter_slots(const unsigned int *keys, const unsigned int *rank, int n_cap, DevCounters *cnt,
                          unsigned int sentinel, int keep_lost, const unsigned int *cell_start, unsigned int *perm,
                          cudaStream_t s) {
  const int th = 256, per_block = th * FDF_SCATTER_ITEMS;
  int blocks = (n_cap + per_block - 1) / per_block;
  k_scatter_slots<<<blocks + 1, th, 0, s>>>(keys, rank, cnt, sentinel, keep_lost, cell_start, perm);
}

int launch_order_segments(const unsigned int *cell_start, int ncells, const long long *pid, unsigned int *perm,
                          unsigned int *lost_scratch, int n_cap, DevCounters *cnt, int num_sms, cudaStream_t s) {
  const int th = 256, blocks = (ncells + th - 1) / th;
  if (pid) k_order_segments<true><<<blocks, th, 0, s>>>(cell_start, ncells, pid, perm);
  else k_order_segments<false><<<blocks, th, 0, s>>>(cell_start, ncells, nullptr, perm);
  if (!lost_scratch) return 1;
  if (pid) order_lost<true>(cell_start + ncells, pid, perm, lost_scratch, n_cap, cnt, num_sms, s);
  else order_lost<false>(cell_start + ncells, nullptr, perm, lost_scratch, n_cap, cnt, num_sms, s);
  return 2;
}

static bool by_tiles(long long n, long long ncells) { return n >= TILE_MIN && n >= 3 * ncells; }

bool cell_sort_on_cursors(long long n, long long ncells) { return by_tiles(n, ncells) && n >= TILE_CURSORS; }

// Stable counting sort of particle slots by cell id, on caller-provided scratch: sums
// [scan_scratch_words(ncells + 1)] and either rank [n] (and no cursor), for sizes where cell_sort_on_cursors does
// not hold, or cursor [ncells] (the slots then come from a second pass of atomics).  cell_start [ncells + 1] is
// both the histogram and (after the scan) the output.
void cell_sort_on_scratch(const int *cell, long long n, long long ncells, unsigned int *perm,
                          unsigned int *cell_start, unsigned int *rank, unsigned int *cursor, unsigned int *sums,
                          cudaStream_t s) {
  const int th = 256;
  const unsigned int blocks = (unsigned int)std::max<long long>((n + th - 1) / th, 1);
  const unsigned int blocks_items = (blocks + SORT_ITEMS - 1) / SORT_ITEMS, tiles = (unsigned int)((n + TILE - 1) / TILE);
  const bool tiled = by_tiles(n, ncells);
  cudaMemsetAsync(cell_start, 0, 4ull * (ncells + 1), s);
  if (tiled && rank) k_cell_tile<RANK><<<tiles, TILE_THREADS, 0, s>>>(cell, n, ncells, cell_start, rank);
  else if (tiled) k_cell_tile<COUNT><<<tiles, TILE_THREADS, 0, s>>>(cell, n, ncells, cell_start, nullptr);
  else if (rank) k_cell_rank<<<blocks_items, th, 0, s>>>(cell, n, ncells, cell_start, rank);
  else k_cell_histogram<<<blocks, th, 0, s>>>(cell, n, ncells, cell_start);
  exclusive_scan_u32(cell_start, ncells + 1, sums, s);
  if (cursor) cudaMemcpyAsync(cursor, cell_start, 4ull * ncells, cudaMemcpyDeviceToDevice, s);
  if (rank) k_cell_place<<<blocks_items, th, 0, s>>>(cell, n, ncells, cell_start, rank, perm);
  else if (tiled) k_cell_tile<SLOTS><<<tiles, TILE_THREADS, 0, s>>>(cell, n, ncells, cursor, perm);
  else k_cell_slots<<<blocks, th, 0, s>>>(cell, n, ncells, cursor, perm);
  launch_order_segments(cell_start, (int)ncells, nullptr, perm, nullptr, 0, nullptr, 0, s);
}
