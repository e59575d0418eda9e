// Sampling on the device: a cluster of eight thread blocks per row of logits.
//
// The chain is the reference's (crates/engine/decode/src/sampler.rs:234-362): penalties ->
// greedy? -> top-k -> top-p -> min-p -> temperature -> softmax -> inverse-CDF draw.  Candidates
// are ordered by (logit descending, token id ascending); every filter keeps a prefix of that
// order, so the surviving set is "all tokens whose order key is >= a threshold".  Thresholds are
// found by radix selection over a 64-bit key (32 bits of order-preserving logit, 32 bits of
// inverted id): by count for top-k, by accumulated probability mass for top-p and for the draw.
// Nothing is sorted there and no size is limited.
//
// That selection reads a row some twenty times.  Almost every row needs far less:
// the filters leave a few tokens.  So the blocks of a row first count its logits in bins of 1/64
// below its maximum (one reading for the maximum, one for the bins), which bounds the tokens that
// can survive, gather those (a third reading) into the first block's shared memory, sort them there
// and finish the chain on the sorted list.  A row whose bound is above CAP tokens (no filter, or a
// flat distribution) goes the general way, every block with its slice of the row.  (In the first
// block alone, 64 rows took 12 to 30 % longer than a grid of one block per row, whose blocks do not
// share SMs.)  What bounds the short way: the three readings, from L2 behind the head's product.  64
// rows of 151,936 logits with the four mixes of options of a server: 1,248 us with one block per row,
// 45 us so (one row: 25 us).
// A small top-k (what a server's rows mostly have) needs no bins: the k-th largest of the largest logits
// of 128 groups of a block's threads bounds its k largest tokens, and the second reading gathers what
// reaches the highest of the blocks' bounds, some 350 tokens: the call with the tokens back on the host,
// 64 rows, 125 -> 118 us.
#include "common.cuh"

#include <cooperative_groups.h>
#include <limits.h>

namespace {
namespace cg = cooperative_groups;

constexpr int THREADS = 512;
constexpr int BINS = 2048;         // of 1/64 below the row's maximum; the last holds all that is lower
constexpr float PER_UNIT = 64.0f;
constexpr int CAP = 2048;          // tokens that the first block of a row can sort
constexpr int MAX_BLOCKS = 8;      // blocks of a row (a portable cluster)
constexpr int GROUPS = 128;        // of a block's threads, whose largest logits bound a small top-k
constexpr int FEW = 64;            // the largest such k

__device__ __forceinline__ uint32_t float_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // larger float -> larger key
}
__device__ __forceinline__ uint64_t order_key(float v, int id) {
  return ((uint64_t)float_key(v) << 32) | (uint32_t)(~(uint32_t)id);  // ties: lower id first
}
__device__ __forceinline__ uint64_t id_key(float, int id) { return (uint32_t)(~(uint32_t)id); }

struct Shared {
  float red[33];
  float hist_f[256], all_f[256];     // of this block's slice; in the first block also of the row
  int hist_i[256], all_i[256];
  unsigned long long prefix;
  float carry_f;
  int carry_i;
};

// All threads of a row's blocks.  (The block's barrier first: threads leave the loops over the
// logits one by one, and the cluster's barrier counts whole warps.)
__device__ __forceinline__ void row_sync(const cg::cluster_group& cluster) {
  __syncthreads();
  cluster.sync();
}

// A row as its blocks see it: this one has the ids [begin, end).
struct Row {
  const float* logits;
  int begin, end, blocks, rank;
};

// Radix selection, most significant byte first, by all blocks of a row.  Elements take part when
// their order key is >= low.  BY_MASS = false: the `target`-th largest key (target counts from 1).
// BY_MASS = true: walking keys downwards, the first key at which the accumulated mass
// w = exp((l - M) * inv_t) reaches the target (`>=` when inclusive, `>` otherwise); if it never does,
// the smallest key with non-zero mass.  ID_ORDER walks by ascending token id instead of by logit.
template <bool BY_MASS, bool ID_ORDER>
__device__ uint64_t radix_select(const cg::cluster_group& cluster, const Row& row, uint64_t low, float M, float inv_t,
                                 float target_f, int target_i, bool inclusive, Shared& s) {
  const int top_byte = ID_ORDER ? 3 : 7;
  if (threadIdx.x == 0) { s.prefix = 0; s.carry_f = 0.f; s.carry_i = 0; }
  __syncthreads();
  for (int b = top_byte; b >= 0; --b) {
    for (int i = threadIdx.x; i < 256; i += THREADS) { s.hist_f[i] = 0.f; s.hist_i[i] = 0; }
    __syncthreads();
    const uint64_t prefix = s.prefix;
    const int shift = 8 * b;
    for (int i = row.begin + threadIdx.x; i < row.end; i += THREADS) {
      const float l = row.logits[i];
      if (order_key(l, i) < low) continue;
      const uint64_t k = ID_ORDER ? id_key(l, i) : order_key(l, i);
      if (b < top_byte && (k >> (shift + 8)) != (prefix >> (shift + 8))) continue;
      const int bin = (int)((k >> shift) & 255u);
      if (BY_MASS) {
        const float w = expf((l - M) * inv_t);
        if (w > 0.f) { atomicAdd(&s.hist_f[bin], w); atomicAdd(&s.hist_i[bin], 1); }
      } else {
        atomicAdd(&s.hist_i[bin], 1);
      }
    }
    row_sync(cluster);
    if (row.rank == 0) {
      for (int i = threadIdx.x; i < 256; i += THREADS) {
        float f = 0.f;
        int n = 0;
        for (int p = 0; p < row.blocks; ++p) {
          const Shared* peer = cluster.map_shared_rank(&s, p);
          if (BY_MASS) f += peer->hist_f[i];
          n += peer->hist_i[i];
        }
        s.all_f[i] = f, s.all_i[i] = n;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        int chosen = -1, last_nonempty = -1;
        if (BY_MASS) {
          float cum = s.carry_f;
          for (int bin = 255; bin >= 0; --bin) {
            if (s.all_i[bin] == 0) continue;
            last_nonempty = bin;
            const float next = cum + s.all_f[bin];
            // at the last byte a bin is one element: apply the crossing rule exactly there;
            // before it, descend into the first bin whose end reaches the target
            const bool hit = inclusive ? (next >= target_f) : (next > target_f);
            if (hit) { chosen = bin; break; }
            cum = next;
          }
          // never reached (rounding): stay on the smallest keys that carry mass; the carry is
          // left as it was, so the finer levels do not reach the target either
          if (chosen < 0) chosen = last_nonempty < 0 ? 0 : last_nonempty;
          else s.carry_f = cum;
        } else {
          int cum = s.carry_i;
          for (int bin = 255; bin >= 0; --bin) {
            if (s.all_i[bin] == 0) continue;
            last_nonempty = bin;
            if (cum + s.all_i[bin] >= target_i) { chosen = bin; break; }
            cum += s.all_i[bin];
          }
          if (chosen < 0) chosen = last_nonempty < 0 ? 0 : last_nonempty;
          else s.carry_i = cum;
        }
        const uint64_t next = prefix | ((uint64_t)chosen << shift);
        for (int p = 0; p < row.blocks; ++p) cluster.map_shared_rank(&s, p)->prefix = next;
      }
    }
    row_sync(cluster);
  }
  const uint64_t found = s.prefix;
  __syncthreads();
  return found;
}

// The mass of the elements with order keys >= low, in every block of the row.
__device__ float row_mass(const cg::cluster_group& cluster, const Row& row, uint64_t low, float M, float inv_t,
                          Shared& s) {
  float z = 0.f;
  for (int i = row.begin + threadIdx.x; i < row.end; i += THREADS) {
    const float l = row.logits[i];
    if (order_key(l, i) >= low) z += expf((l - M) * inv_t);
  }
  z = warp_sum(z);
  if ((threadIdx.x & 31) == 0) s.red[threadIdx.x >> 5] = z;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < THREADS / 32 ? s.red[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) s.red[32] = t;
  }
  row_sync(cluster);
  float all = 0.f;
  for (int p = 0; p < row.blocks; ++p) all += cluster.map_shared_rank(&s, p)->red[32];
  row_sync(cluster);
  return all;
}

// The whole chain by radix selection, for all blocks of a row: any number of survivors.
__device__ void sample_general(const cg::cluster_group& cluster, const Row& row, int V, float M, float temp, int k, float p,
                               float mp, double u, int* out, Shared& s) {
  uint64_t low = 0;
  bool sorted = false;
  if (k > 0 && k < V) {
    low = radix_select<false, false>(cluster, row, 0, M, 1.f, 0.f, k, true, s);
    sorted = true;
  }
  if (p < 1.0f && !(k == 1)) {
    const float Z = row_mass(cluster, row, low, M, 1.f, s);
    const uint64_t t = radix_select<true, false>(cluster, row, low, M, 1.f, p * Z, 0, true, s);
    low = t > low ? t : low;
    sorted = true;
  }
  if (mp > 0.f) {
    const float floor_logit = M + logf(mp);
    const uint64_t t = (uint64_t)float_key(floor_logit) << 32;  // every id at or above the floor
    low = t > low ? t : low;
  }
  const float inv_t = 1.0f / temp;
  const float Z = row_mass(cluster, row, low, M, inv_t, s);
  const float target = (float)(u * (double)Z);
  const uint64_t pick = sorted ? radix_select<true, false>(cluster, row, low, M, inv_t, target, 0, false, s)
                               : radix_select<true, true>(cluster, row, low, M, inv_t, target, 0, false, s);
  if (row.rank == 0 && threadIdx.x == 0) *out = (int)(~(uint32_t)(pick & 0xffffffffu));
}

// f(logit, id) for the ids [begin, end) of a row, in batches of four 16-byte loads per thread where
// the row allows it (the loads of a batch are in flight together: f may touch shared memory, which
// the compiler does not move loads across).
template <typename F>
__device__ __forceinline__ void for_each_logit(const float* row, int begin, int end, F f) {
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {        // begin is a multiple of four
    constexpr int BATCH = 4;
    const int whole = begin + ((end - begin) & ~3);
    for (int i0 = begin + 4 * threadIdx.x; i0 < whole; i0 += 4 * THREADS * BATCH) {
      float4 v[BATCH];
#pragma unroll
      for (int j = 0; j < BATCH; ++j)
        if (i0 + 4 * THREADS * j < whole) v[j] = __ldg(reinterpret_cast<const float4*>(row + i0 + 4 * THREADS * j));
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        const int i = i0 + 4 * THREADS * j;
        if (i < whole) f(v[j].x, i), f(v[j].y, i + 1), f(v[j].z, i + 2), f(v[j].w, i + 3);
      }
    }
    begin = whole;
  }
  for (int i = begin + threadIdx.x; i < end; i += THREADS) f(__ldg(row + i), i);
}

// The bin of a logit: monotone in the logit (the difference and the scaling by a power of two
// round monotonically).  What is not a number sorts below everything and goes to the last bin.
__device__ __forceinline__ int bin_of(float l, float M) {
  const float d = (M - l) * PER_UNIT;
  return d < (float)BINS ? (int)d : BINS - 1;
}

struct Control {
  int cut;            // the last bin whose tokens are gathered, or -1: the general way
  int n;              // how many tokens that are
  unsigned taken;     // slots of the list given out so far
};

struct ListShared {
  Control control;
  unsigned long long best[MAX_BLOCKS], warp_best[THREADS / 32];
  double part[THREADS / 32];
  int part_i[THREADS / 32];
  int crossing;
  uint32_t group_best[GROUPS], block_bound, bound[MAX_BLOCKS];
  union {
    struct { alignas(16) int count[BINS]; alignas(16) float mass[BINS]; } bins;
    unsigned long long list[CAP];
    Shared general;
  };
};

// Exclusive prefix over the block of one value per thread; `total` gets the sum.
template <typename T>
__device__ __forceinline__ T block_prefix(T v, T* part, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T run = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T up = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += up;
  }
  __syncthreads();
  if (lane == 31) part[warp] = run;
  __syncthreads();
  T before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) {
    if (w < warp) before += part[w];
    total += part[w];
  }
  return before + run - v;
}

// The keys of `list` [n] in descending order; the list has room for the next power of two.
__device__ void sort_descending(unsigned long long* list, int n) {
  int size = 1;
  while (size < n) size <<= 1;
  for (int i = n + threadIdx.x; i < size; i += THREADS) list[i] = 0;
  __syncthreads();
  for (int k = 2; k <= size; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < size / 2; t += THREADS) {
        const int a = 2 * t - (t & (j - 1)), b = a + j;
        const unsigned long long x = list[a], y = list[b];
        if ((x < y) == ((a & k) == 0)) list[a] = y, list[b] = x;
      }
      __syncthreads();
    }
}

// The first place of the sorted list at which the running sum of weight(i) reaches the target
// (`>=` when inclusive, `>` otherwise) given by target_of(sum of all weights); the last place with
// a weight when none does, -1 when there is none.  Thread t holds PER adjacent places.
template <typename W, typename G>
__device__ int crossing_place(int n, bool inclusive, W weight, G target_of, ListShared& s) {
  constexpr int PER = CAP / THREADS;
  float w[PER];
  double mine = 0;
  int last = -1;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int i = threadIdx.x * PER + e;
    w[e] = i < n ? weight(i) : 0.f;
    if (w[e] > 0.f) last = i;
    mine += (double)w[e];
  }
  double total;
  double cum = block_prefix(mine, s.part, total);
  const float target = target_of(total);
  if (threadIdx.x == 0) s.crossing = INT_MAX;
  __syncthreads();
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    cum += (double)w[e];
    if (w[e] > 0.f && (inclusive ? (float)cum >= target : (float)cum > target)) {
      atomicMin(&s.crossing, threadIdx.x * PER + e);
      break;
    }
  }
  __syncthreads();
  int place = s.crossing;
  if (place == INT_MAX) {
    __syncthreads();
    if (threadIdx.x == 0) s.crossing = -1;
    __syncthreads();
    if (last >= 0) atomicMax(&s.crossing, last);
    __syncthreads();
    place = s.crossing;
  }
  __syncthreads();
  return place;
}

__device__ __forceinline__ float logit_of_key(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// One cluster of blocks per row (grid: blocks of a row, rows).
__global__ void __launch_bounds__(THREADS) sample_kernel(
    const float* __restrict__ logits, long long ld, int V, const float* __restrict__ temperature,
    const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
    const double* __restrict__ uniform, int* __restrict__ out, const int* __restrict__ status,
    int* __restrict__ status_out) {
  __shared__ ListShared s;
  cg::cluster_group cluster = cg::this_cluster();
  const int blocks = gridDim.x, rank = blockIdx.x, r = blockIdx.y;
  // the library's status words travel to the host with the tokens: whoever reads the tokens
  // learns in the same copy whether a kernel of the step gave up a wait or met a bad token id
  if (status != nullptr && r == 0 && rank == 0 && threadIdx.x < 4) status_out[threadIdx.x] = status[threadIdx.x];
  const float* row = logits + (size_t)r * ld;
  const int slice = ((V + blocks - 1) / blocks + 3) & ~3;
  const int begin = min(V, rank * slice), end = min(V, begin + slice);

  const float temp = temperature[r];
  const int k = top_k[r];
  const bool by_count = k > 0 && k < V, few = by_count && k <= FEW && temp > 0.f;

  // ---- the largest order key of the row (the arg max, lowest id among equals)
  uint64_t b = 0;
  for_each_logit(row, begin, end, [&](float l, int i) {
    const uint64_t k = order_key(l, i);
    b = k > b ? k : b;
  });
  for (int i = threadIdx.x; i < BINS; i += THREADS) s.bins.count[i] = 0, s.bins.mass[i] = 0.f;
  if (threadIdx.x == 0) s.control.taken = 0;
  if (few) {
    // The largest logits of 128 groups of threads: the k-th largest of them is a bound below which no
    // token of the k largest can lie (at least k of this block's reach it), and the highest of the
    // blocks' bounds is one for the row.
    static_assert(THREADS == 4 * GROUPS, "four threads to a group");
    uint32_t mine = (uint32_t)(b >> 32);
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) mine = max(mine, __shfl_xor_sync(0xffffffffu, mine, o));
    if ((threadIdx.x & 3) == 0) s.group_best[threadIdx.x >> 2] = mine;
    __syncthreads();
    if (threadIdx.x < GROUPS) {
      const uint32_t key = s.group_best[threadIdx.x];
      int above = 0, equal = 0;
      for (int i = 0; i < GROUPS; ++i) {
        const uint32_t other = s.group_best[i];
        above += other > key, equal += other == key;
      }
      if (above < k && above + equal >= k) s.block_bound = key;      // (one value, whoever writes it)
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t k = __shfl_xor_sync(0xffffffffu, b, o);
    b = k > b ? k : b;
  }
  if ((threadIdx.x & 31) == 0) s.warp_best[threadIdx.x >> 5] = b;
  row_sync(cluster);                     // every block of the row has started
  // each block hands its best to all of them
  if (threadIdx.x < blocks) {
    for (int w = 0; w < THREADS / 32; ++w) b = s.warp_best[w] > b ? s.warp_best[w] : b;
    cluster.map_shared_rank(&s, threadIdx.x)->best[rank] = b;
    if (few) cluster.map_shared_rank(&s, threadIdx.x)->bound[rank] = s.block_bound;
  }
  row_sync(cluster);
  uint64_t best = 0;
  for (int i = 0; i < blocks; ++i) best = s.best[i] > best ? s.best[i] : best;

  const int best_id = (int)(~(uint32_t)(best & 0xffffffffu));
  const float M = row[best_id];
  if (!(temp > 0.f) || !isfinite(M)) {  // greedy: first maximum wins
    if (rank == 0 && threadIdx.x == 0) out[r] = best_id;
    return;                             // every block of the row alike
  }
  const float p = top_p[r], mp = min_p[r], inv_t = 1.0f / temp;
  const bool by_mass = p < 1.0f && k != 1;
  const float floor_logit = mp > 0.f ? M + logf(mp) : -INFINITY;
  ListShared* first = cluster.map_shared_rank(&s, 0);

  double mass_all = 0;                   // of the row, where the bins tell it (by_mass && !by_count)
  int n = 0;                             // tokens in the first block's list
  bool listed = false;
  if (few && isfinite(inv_t) && floor_logit <= M) {
    // ---- a small top-k: the tokens that reach the bound, some 45 a block (no counting in bins)
    uint32_t bound = 0;
    for (int i = 0; i < blocks; ++i) bound = max(bound, s.bound[i]);
    for_each_logit(row, begin, end, [&](float l, int i) {
      if (float_key(l) >= bound) {
        const unsigned at = atomicAdd(&first->control.taken, 1u);
        if (at < CAP) first->list[at] = order_key(l, i);
      }
    });
    row_sync(cluster);
    n = (int)first->control.taken;
    listed = n <= CAP;
    if (listed && rank != 0) return;     // (the first block waits for these readers at its end)
    if (!listed) {                       // many equal logits: the bins, as for any other row
      row_sync(cluster);
      for (int i = threadIdx.x; i < BINS; i += THREADS) s.bins.count[i] = 0, s.bins.mass[i] = 0.f;
      if (threadIdx.x == 0) s.control.taken = 0;
      row_sync(cluster);
    }
  }
  if (!listed) {
    // ---- how many tokens (and how much of the mass) lie in which bin
    // (a peaked row has nearly all of its tokens in the last bin: those are counted per thread)
    int deep = 0;
    float deep_mass = 0.f;
    for_each_logit(row, begin, end, [&](float l, int) {
      const int bin = bin_of(l, M);
      float w = 0.f;
      if (by_mass && !by_count) {
        w = expf(l - M);
        w = w > 0.f ? w : 0.f;             // no number, no mass
      }
      if (bin == BINS - 1) {
        ++deep;
        deep_mass += w;
      } else {
        atomicAdd(&s.bins.count[bin], 1);
        if (w > 0.f) atomicAdd(&s.bins.mass[bin], w);
      }
    });
    if (deep) atomicAdd(&s.bins.count[BINS - 1], deep);
    if (deep_mass > 0.f) atomicAdd(&s.bins.mass[BINS - 1], deep_mass);
    row_sync(cluster);
    constexpr int PER = BINS / THREADS;
    if (rank == 0) {
      int count[PER], n = 0;
      double mass[PER], m = 0;
#pragma unroll
      for (int e = 0; e < PER; ++e) count[e] = 0, mass[e] = 0;
      for (int i = 0; i < blocks; ++i) {
        const ListShared* peer = cluster.map_shared_rank(&s, i);
        static_assert(PER == 4, "a thread's bins are one 16-byte load");
        const int4 c = *reinterpret_cast<const int4*>(peer->bins.count + threadIdx.x * PER);
        count[0] += c.x, count[1] += c.y, count[2] += c.z, count[3] += c.w;
        if (by_mass && !by_count) {
          const float4 w = *reinterpret_cast<const float4*>(peer->bins.mass + threadIdx.x * PER);
          mass[0] += (double)w.x, mass[1] += (double)w.y, mass[2] += (double)w.z, mass[3] += (double)w.w;
        }
      }
#pragma unroll
      for (int e = 0; e < PER; ++e) n += count[e], m += mass[e];
      int n_all;
      int before = block_prefix(n, s.part_i, n_all);
      double m_before = block_prefix(m, s.part, mass_all);
      if (threadIdx.x == 0) s.control.cut = BINS - 1, s.control.n = n_all;
      __syncthreads();
      // the first bin behind which nothing can survive: the k-th token's or the one in which the
      // mass is reached, and the floor's.  With both top-k and top-p the mass is that of all k
      // tokens, so the floor may not hide any of them.
      const float target = p * (float)mass_all;
      const int floor_bin = mp > 0.f && !(by_count && by_mass) ? bin_of(floor_logit, M) : BINS - 1;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int bin = threadIdx.x * PER + e;
        before += count[e];
        m_before += mass[e];
        bool hit = bin == floor_bin;
        if (by_count) hit = hit || before >= k;
        else if (by_mass) hit = hit || (count[e] > 0 && (float)m_before >= target);
        if (hit) { atomicMin(&s.control.cut, bin); break; }
      }
      __syncthreads();
      const int cut = s.control.cut;
      __syncthreads();                     // (all have read it: the thread that owns the cut writes the word)
      if (cut / PER == (int)threadIdx.x) {
        // `before` stands at the cut for this thread: it left its loop there
        const bool list = before <= CAP && isfinite(inv_t) && floor_logit <= M;
        for (int i = 0; i < blocks; ++i) {
          Control* c = &cluster.map_shared_rank(&s, i)->control;
          c->cut = list ? cut : -1;
          c->n = before;
        }
      }
    }
    row_sync(cluster);                        // the first block is done with the bins as well
    const int cut = s.control.cut;
    n = s.control.n;
    if (cut < 0) {
      sample_general(cluster, Row{row, begin, end, blocks, rank}, V, M, temp, k, p, mp, uniform[r], out + r, s.general);
      return;
    }

    // ---- those tokens into the first block's list
    for_each_logit(row, begin, end, [&](float l, int i) {
      if (bin_of(l, M) <= cut) {
        const unsigned at = atomicAdd(&first->control.taken, 1u);
        if (at < CAP) first->list[at] = order_key(l, i);
      }
    });
    row_sync(cluster);
    if (rank != 0) return;
  }
  const bool sorted = by_count || by_mass;
  if (!sorted) {                         // the draw walks by ascending id: id first, logit second
    for (int i = threadIdx.x; i < n; i += THREADS) s.list[i] = (s.list[i] << 32) | (s.list[i] >> 32);
    __syncthreads();
  }
  sort_descending(s.list, n);
  const uint32_t floor_key = float_key(floor_logit);
  auto key_at = [&](int i) { return (uint32_t)(sorted ? s.list[i] >> 32 : s.list[i]); };
  int m = by_count ? min(k, n) : n;
  if (by_mass) {
    const int place = crossing_place(
        m, true, [&](int i) { return expf(logit_of_key(key_at(i)) - M); },
        [&](double sum) { return p * (float)(by_count ? sum : mass_all); }, s);
    m = place < 0 ? m : place + 1;
  }
  const int place = crossing_place(
      m, false,
      [&](int i) {
        const uint32_t key = key_at(i);
        return key >= floor_key ? expf((logit_of_key(key) - M) * inv_t) : 0.f;
      },
      [&](double sum) { return (float)(uniform[r] * (double)(float)sum); }, s);
  if (threadIdx.x == 0) {
    const unsigned long long e = s.list[place < 0 ? 0 : place];
    out[r] = (int)~(uint32_t)(sorted ? e : e >> 32);
  }
  cluster.sync();                        // (the other blocks have read its count, or left)
}

// For every (row, token, count) of the penalty windows: a positive logit is divided by the
// repeat penalty, another multiplied; then count * frequency + presence is subtracted
// (sampler.rs:486-507).
__global__ void penalty_kernel(float* __restrict__ logits, long long ld, const int* __restrict__ triples,
                               int n, const float* __restrict__ repeat, const float* __restrict__ freq,
                               const float* __restrict__ presence, const int* __restrict__ inflight_src,
                               const int* __restrict__ drawn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = triples[3 * i], tok = triples[3 * i + 1];
  int count = triples[3 * i + 2];
  // the token that the step before is still drawing for this row counts once more
  if (inflight_src && inflight_src[r] >= 0 && drawn[inflight_src[r]] == tok) ++count;
  float* l = logits + (size_t)r * ld + tok;
  float v = *l;
  v = v <= 0.f ? v * repeat[r] : v / repeat[r];
  v -= (float)count * freq[r] + presence[r];
  *l = v;
}

// Rows whose window gets a token that the host does not know yet (the step before is still
// drawing it; drawn[inflight_src[row]] will hold it in stream order): when no triple of the row
// names that token, it has been seen once.  One thread per row walks the triples.
__global__ void penalty_inflight_kernel(float* __restrict__ logits, long long ld, int V,
                                        const int* __restrict__ triples, int n, int rows,
                                        const float* __restrict__ repeat, const float* __restrict__ freq,
                                        const float* __restrict__ presence,
                                        const int* __restrict__ inflight_src, const int* __restrict__ drawn) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows || inflight_src[r] < 0) return;
  const int tok = drawn[inflight_src[r]];
  if (tok < 0 || tok >= V) return;
  for (int i = 0; i < n; ++i)
    if (triples[3 * i] == r && triples[3 * i + 1] == tok) return;      // counted by its triple
  float* l = logits + (size_t)r * ld + tok;
  float v = *l;
  v = v <= 0.f ? v * repeat[r] : v / repeat[r];
  v -= 1.0f * freq[r] + presence[r];
  *l = v;
}
}  // namespace

LLM_EXPORT int llm_sample(const float* logits, long long ld, int rows, int V,
                          const float* temperature, const int* top_k, const float* top_p,
                          const float* min_p, const double* uniform, int* out, const int* status,
                          int* status_out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0) return LLM_ERR_ARGUMENT;
  // a row of a small vocabulary is one block's work: its readings take less than the cluster's
  // barriers
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = V >= 8192 ? MAX_BLOCKS : 1;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = THREADS;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  for (int r = 0; r < rows; r += 65535) {                // rows lie along the grid's y
    const size_t at = (size_t)r;
    cfg.gridDim = dim3(attr[0].val.clusterDim.x, rows - r < 65535 ? rows - r : 65535);
    const int rc = (int)cudaLaunchKernelEx(&cfg, sample_kernel, logits + at * ld, ld, V, temperature + at,
                                           top_k + at, top_p + at, min_p + at, uniform + at, out + at,
                                           r ? (const int*)nullptr : status, status_out);
    if (rc) return rc;
  }
  return launch_status();
}

// triples: n (row, token, count) of the tokens in the rows' penalty windows.  inflight_src (may be
// null): per row of `rows`, the index in `drawn` of a token that enters the row's window but is
// still being drawn by the step before (-1: none); rows with penalties switched off must have -1.
LLM_EXPORT int llm_apply_penalties(float* logits, long long ld, int V, const int* triples, int n,
                                   const float* repeat, const float* freq, const float* presence,
                                   const int* inflight_src, const int* drawn, int rows,
                                   cudaStream_t stream) {
  if (n > 0)
    penalty_kernel<<<(n + 127) / 128, 128, 0, stream>>>(logits, ld, triples, n, repeat, freq, presence,
                                                        inflight_src, drawn);
  if (inflight_src && rows > 0)
    penalty_inflight_kernel<<<(rows + 63) / 64, 64, 0, stream>>>(logits, ld, V, triples, n, rows, repeat, freq,
                                                               presence, inflight_src, drawn);
  return launch_status();
}
