// The persistent tcgen05 matrix product on CTA pairs (tcgen05 cta_group::2) for many rows:
//     C[t][n] (=|+=) sum_k X[t][k] * W[n][k],   tiles of 256 weight rows x 256 tokens per pair.
// Two CTAs on neighbouring SMs (a cluster of two) share one tile.  Each loads HALF of both
// operands into its own shared memory (its 128 weight rows, its 128 tokens: 32 KB per stage instead
// of the 48 KB a lone CTA needs for half the tile), the leader CTA issues one
// tcgen05.mma.cta_group::2 of 256 x 256 x 16 that reads both halves from both CTAs, and each CTA
// ends up with the accumulator of its own 128 weight rows x 256 tokens in its own tensor memory.
// A third less shared-memory fill per flop is what the lone-CTA kernel lacked: its tensor pipe
// waited for operands.
//
//   warp 0     TMA producer of this CTA's halves, running ahead across tiles through a ring of stages
//              (both CTAs' loads count their bytes on the LEADER's barrier of the stage)
//   warp 1     leader CTA only: waits until a stage is full in both CTAs, issues the MMAs, and commits
//              them to the stage's "empty" barrier in both CTAs (tcgen05.commit ... multicast::cluster)
//   warps 2-5  epilogue of one of two accumulators (2 x 256 TMEM columns) while the next tile is
//              multiplied: TMEM -> registers -> shared memory in chunks of 32 tokens -> TMA store or
//              TMA add-reduction; the leader learns from both CTAs when an accumulator is drained
//
// The grouped form (GROUPED): X's rows lie in tiles of bn rows, tile i multiplied with matrix
// tile_group[i] of W (a feed-forward of routed experts, the tokens sorted by expert).  Neighbouring
// tiles of one matrix are taken together, up to 256 rows, and the MMA is as wide as what was
// taken (N = bn, 2 bn, ... 256), so that only the padding of an expert's last bn rows is multiplied for
// nothing.  1,501 tokens with two of eight experts of 6,144 x 4,096, lone CTAs with tiles of 128 rows ->
// pairs: up with its squared rectifier 241 -> 163 us (one kernel instead of two), gated 183 -> 164, down
// 165 -> 165 (3,072 tokens: 299 -> 288).  (Dealing the pieces by length, the longest first, took 199 us:
// a matrix's pieces then are not neighbours in time and its rows come from memory twice.)
//
// Epilogues: store, residual add, squared rectifier, gated silu(g) * u with gate and up rows
// interleaved in blocks of 16.  The output must be reachable by TMA.  Every wait is bounded: a CTA that gives up sets
// *status and walks to the final cluster barrier, where its peer (whose own waits run out in
// turn) meets it before tensor memory is freed.  No load is multicast.
#include "tcgen05.cuh"

int g_llm_pair = 1;           // 0: the dispatcher keeps to the one-CTA kernels (for comparisons)
int g_llm_pair_ksplits = 0;   // > 0: this many ranges of K in the adding epilogue (for measurements)

namespace {

constexpr int BN = 256;          // tokens per pair tile
constexpr int HALF_N = 128;      // tokens this CTA loads
constexpr int CH = 32;           // tokens per epilogue chunk

constexpr int MAX_SMALL = 512;   // tiles of bn rows that the grouped form takes

template <int STAGES, int FEAT, typename TC, bool GROUPED>
struct alignas(1024) PairStorage {
  uint8_t a[STAGES][TILE_M * TILE_K * 2];      // this CTA's 128 weight rows
  uint8_t b[STAGES][HALF_N * TILE_K * 2];      // this CTA's 128 tokens
  alignas(128) TC out[2][CH * FEAT];
  uint64_t full[STAGES];        // leader's: the bytes of both CTAs' halves are counted here
  uint64_t empty[STAGES];       // both: the MMAs that read this stage are done
  uint64_t acc_full[2];         // both: the tile's MMAs are done
  uint64_t acc_empty[2];        // leader: both CTAs have drained the accumulator
  uint32_t tmem_base;
  int dead;
  int n_list;                                      // grouped form: what is multiplied together,
  int list[GROUPED ? MAX_SMALL : 1];               // first tile + (tiles << 16),
  int group[GROUPED ? MAX_SMALL : 1];              // and every tile's matrix
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_local(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// arrive on the barrier at the same shared-memory offset in CTA `cta` of the pair
__device__ __forceinline__ void mbar_arrive_in(uint64_t* bar, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(cta));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// bounded wait on a barrier that the other CTA (or an MMA commit from it) arrives on
__device__ __forceinline__ bool mbar_wait_pair(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  long long start = 0;
  for (uint32_t i = 0;; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (i == 0) start = clock64();
    else if (clock64() - start > WAIT_CYCLES) return false;
  }
}
// the shared::cluster address of `p` as CTA `cta` of the pair holds it
__device__ __forceinline__ uint32_t in_cta(const void* p, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(p)), "r"(cta));
  return remote;
}
// TMA tile load into this CTA's shared memory whose bytes are counted on a barrier that may be the
// other CTA's (`bar_cluster`: a shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float relu_squared(float z) {
  const float r = fmaxf(z, 0.f);
  return r * r;
}
// when the MMAs issued so far are done, arrive on the barrier at this offset in both CTAs
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  const uint16_t both = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(both)
      : "memory");
}

// the grouped form's operands: n_small tiles of bn rows, tile i with matrix tile_group[i] (negative:
// left out), matrices group_rows rows of W apart; row_scale (clamped epilogue): a factor per row of X
struct Grouping {
  const int* tile_group;
  int bn, n_small, group_rows;
  const float* row_scale;
  int in_order;      // LAST_TOKENS: a matrix tile's last tokens follow its whole tiles (see launch)
  int k_up;          // the ranges of K: range ks begins at its share of the blocks of K, rounded down (0) or up (1)
};

// What a tile holds: 256 tokens always; 256 or, at the end of T, fewer; or the grouped form's pieces.
// (A variant of its own for the first: with a width read at run time it lost 1 % on prompts of 2,048
// and 8,192 tokens.)
enum Form : int { WHOLE_TILES = 0, LAST_TOKENS = 1, GROUPED_TILES = 2 };

// map_x: boxes of 128 tokens, map_xs: of 64
template <int STAGES, int EPI, typename TC, int FORM>
__global__ void __launch_bounds__(192, 1) gemm_pair_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
    const __grid_constant__ CUtensorMap map_xs, const __grid_constant__ CUtensorMap map_c, int T, int N, int K, int half,
    int m_tiles, int n_tiles, int ksplits, float act_limit, int* __restrict__ status, const Grouping grouping) {
  constexpr bool GATED = gated_epilogue(EPI), GROUPED = FORM == GROUPED_TILES;
  constexpr int FEAT = GATED ? 64 : TILE_M;     // output features of this CTA per tile
  // EPI_TWO_SUMS: the accumulators hold the sums over the first and the second half of K of one tile,
  // which are added where they are read: the bits of a product whose halves were added in memory,
  // without the additions (a tile's epilogue then has no next tile beside it)
  constexpr int SUMS = EPI == EPI_TWO_SUMS ? 2 : 1;
  extern __shared__ uint8_t raw[];
  auto& sm = *reinterpret_cast<PairStorage<STAGES, FEAT, TC, GROUPED>*>(
      (reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int nkb = (K + TILE_K - 1) / TILE_K;
  // A work item is a tile and one of `ksplits` ranges of K (more than one only with the adding
  // epilogue, whose partial sums meet in memory).
  int works = m_tiles * n_tiles * ksplits;
  // float32 accumulator, bf16 A and B, both K-major, M = 256 over the pair; N as the tile has tokens
  constexpr uint32_t idesc_0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((2 * TILE_M) >> 4) << 24);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.full[s], 1);          // the leader's producer, expecting the bytes of both CTAs
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.acc_full[b], 1);
      mbar_init(&sm.acc_empty[b], 8);     // four epilogue warps in each CTA
    }
    sm.dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  pair_sync();               // both CTAs' barriers exist before either signals the other
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  pdl_trigger();             // after the allocation, as in the one-CTA kernel
  if (GROUPED) {
    // (the tiles' matrices come from a kernel before this one, and the weights depend on them)
    pdl_wait();
    for (int i = threadIdx.x; i < grouping.n_small; i += 192) sm.group[i] = grouping.tile_group[i];
    __syncthreads();
    if (threadIdx.x == 0) {
      const int most = BN / grouping.bn;
      int n = 0, len = 0, last = -1;
      for (int i = 0; i < grouping.n_small; ++i) {
        const int g = sm.group[i];
        if (g >= 0) {
          if (g == last && len < most) ++len, sm.list[n - 1] += 1 << 16;
          else len = 1, sm.list[n++] = i | (1 << 16);
        }
        last = g;
      }
      sm.n_list = n;
    }
    __syncthreads();
    n_tiles = sm.n_list;
    works = m_tiles * n_tiles;
  }
  // the tile and the range of K of a work item: items of whole tiles before those of the last tokens
  const int n_whole = GROUPED ? 0 : FORM == WHOLE_TILES ? m_tiles * n_tiles : m_tiles * (T / BN);
  auto item = [&](int work, int& tile, int& ks) {
    if (GROUPED) {
      tile = work, ks = 0;
    } else if (FORM == WHOLE_TILES) {
      tile = work % n_whole, ks = work / n_whole;
    } else if (grouping.in_order) {
      // (dealt one place further in every round, so that the short items do not all meet the same pairs)
      const int all = m_tiles * n_tiles, round = work / n_pairs, base = round * n_pairs;
      const int at = base + (work - base + round) % min(n_pairs, works - base);
      ks = at / all, tile = at % all;
    } else if (work < n_whole * ksplits) {
      tile = work % n_whole, ks = work / n_whole;
    } else {
      const int rest = work - n_whole * ksplits;
      tile = n_whole + rest % m_tiles, ks = rest / m_tiles;
    }
  };
  auto range_start = [&](int ks) {
    return (int)(((long long)ks * nkb + (grouping.k_up ? ksplits - 1 : 0)) / ksplits);
  };
  // a tile's place among the tiles of weight rows, its first row of X, its rows, and the row of W
  // where its matrix starts
  auto place = [&](int tile, int& m, int& t0, int& n, int& w0) {
    if (GROUPED) {
      const int e = sm.list[tile % n_tiles], i = e & 0xffff;
      m = tile / n_tiles, t0 = i * grouping.bn, n = (e >> 16) * grouping.bn, w0 = sm.group[i] * grouping.group_rows;
    } else if (FORM == WHOLE_TILES) {
      m = tile / n_tiles, t0 = (tile % n_tiles) * BN, n = BN, w0 = 0;
    } else {
      // the whole tiles of tokens first, then, if T is not a multiple of 256, the last tokens, with
      // an MMA as wide as they are (in steps of 32)
      const int whole = T / BN;
      w0 = 0;
      if (grouping.in_order) {
        m = tile / n_tiles, t0 = (tile % n_tiles) * BN;
        n = T - t0 >= BN ? BN : (T - t0 + 31) & ~31;
      } else if (tile < n_whole) m = tile / whole, t0 = (tile % whole) * BN, n = BN;
      else m = tile - n_whole, t0 = whole * BN, n = (T - t0 + 31) & ~31;
    }
  };

  if (warp == 0 && lane == 0) {
    // ------------------------------------------------------------------ producer (both CTAs)
    // Both CTAs' loads count their bytes on the LEADER's barrier of the stage; only the leader's
    // producer arrives there, expecting the bytes of both (the other CTA's bytes may be counted
    // before that arrival: the count is signed).
    uint32_t full_addr[STAGES];
    for (int s = 0; s < STAGES; ++s) full_addr[s] = in_cta(&sm.full[s], 0);
    // A tile of up to 128 tokens brings half a box of them (both operands come from the L2 at some 10
    // TB/s over all pairs, which is what holds this kernel; several smaller boxes cost the TMA unit
    // more than they save: 165 -> 181 us for the grouped products above).
    auto load_w = [&](int s, int row0, int k, int n) {
      const int b_rows = FORM == WHOLE_TILES || n > HALF_N ? HALF_N : HALF_N / 2;
      if (leader) mbar_expect_tx(&sm.full[s], 2 * (uint32_t)((TILE_M + b_rows) * TILE_K * 2));
      tma_load_2d_pair(sm.a[s], &map_w, k, row0, full_addr[s]);
    };
    auto load_x = [&](int s, int t0, int k, int n) {
      tma_load_2d_pair(sm.b[s], FORM == WHOLE_TILES || n > HALF_N ? &map_x : &map_xs, k, t0, full_addr[s]);
    };
    long long it = 0;
    bool ok = true;
    bool first = true;
    for (int work = pair; work < works && ok; work += n_pairs) {
      int tile, ks, m, t0, n, w0;
      item(work, tile, ks);
      place(tile, m, t0, n, w0);
      const int kb0 = range_start(ks), kb1 = range_start(ks + 1);
      const int f0 = m * (2 * FEAT) + (int)rank * FEAT;          // first output feature
      const int row0 = w0 + (GATED ? 2 * f0 : f0);               // first weight row
      t0 += (int)rank * (n >> 1);                                // (this CTA's half of the tokens)
      int kb = kb0;
      if (!GROUPED && first) {
        // weights do not depend on earlier kernels: fetch a ring of them before waiting
        const int head = min(kb1 - kb0, STAGES);
        for (int i = 0; i < head; ++i) load_w(i, row0, (kb0 + i) * TILE_K, n);
        pdl_wait();
        for (int i = 0; i < head; ++i) load_x(i, t0, (kb0 + i) * TILE_K, n);
        it = head;
        kb = kb0 + head;
        first = false;
      }
      for (; kb < kb1; ++kb, ++it) {
        const int s = (int)(it % STAGES);
        ok = mbar_wait_pair(&sm.empty[s], (uint32_t)((it / STAGES) & 1) ^ 1);
        if (!ok) { atomicExch(status, 1); sm.dead = 1; break; }
        load_w(s, row0, kb * TILE_K, n);
        load_x(s, t0, kb * TILE_K, n);
      }
    }
    // A producer gives up only after a wait of about two seconds, far longer than any load it
    // still has in flight needs to land; the final barrier of the pair comes after that.
  } else if (warp == 1 && lane == 0 && leader) {
    // ------------------------------------------------------------------ leader: MMA issuer
    long long it = 0;
    int local = 0;
    bool ok = true;
    for (int work = pair; work < works && ok; work += n_pairs, ++local) {
      int tile, ks, m, t0, n, w0;
      item(work, tile, ks);
      place(tile, m, t0, n, w0);
      const uint32_t idesc = idesc_0 | ((uint32_t)(n >> 3) << 17);
#pragma unroll 1
      for (int sum = 0; sum < SUMS && ok; ++sum) {
        const int kb0 = SUMS == 2 ? sum * ((nkb + 1) / 2) : range_start(ks);
        const int kb1 = SUMS == 2 ? (sum ? nkb : (nkb + 1) / 2) : range_start(ks + 1);
        const int buf = SUMS == 2 ? sum : local & 1, use = SUMS == 2 ? local : local >> 1;
        ok = mbar_wait_pair(&sm.acc_empty[buf], (uint32_t)(use & 1) ^ 1);
        if (!ok) { atomicExch(status, 2); sm.dead = 1; break; }
        tc_fence_after();
        const uint32_t acc = tmem + (uint32_t)buf * BN;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = (int)(it % STAGES);
          ok = mbar_wait_pair(&sm.full[s], (uint32_t)((it / STAGES) & 1));
          if (!ok) { atomicExch(status, 2); sm.dead = 1; break; }
          tc_fence_after();
          const uint64_t da = smem_desc(smem_u32(sm.a[s]));
          const uint64_t db = smem_desc(smem_u32(sm.b[s]));
#pragma unroll
          for (int k = 0; k < TILE_K / UMMA_K; ++k)
            pair_mma(acc, da + (uint64_t)(k * UMMA_K * 2 >> 4), db + (uint64_t)(k * UMMA_K * 2 >> 4), idesc,
                     (kb > kb0 || k > 0) ? 1u : 0u);
          pair_commit(&sm.empty[s]);
        }
        if (ok) pair_commit(&sm.acc_full[buf]);
      }
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (both CTAs)
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const bool issuer = warp == 2 && lane == 0;
    pdl_wait();
    int local = 0;
    int chunk_no = 0;
    for (int work = pair; work < works; work += n_pairs, ++local) {
      int tile, ks, m, t0, n_cols, w0;
      item(work, tile, ks);
      place(tile, m, t0, n_cols, w0);
      const int n0 = m * (2 * FEAT) + (int)rank * FEAT;
      const int buf = SUMS == 2 ? 0 : local & 1, use = SUMS == 2 ? local : local >> 1;
      bool ok = mbar_wait_pair(&sm.acc_full[buf], (uint32_t)(use & 1));
      if (SUMS == 2 && ok) ok = mbar_wait_pair(&sm.acc_full[1], (uint32_t)(use & 1));
      if (!ok) { if (lane == 0) atomicExch(status, 3); sm.dead = 1; }
      // the four warps decide together whether to go on
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (sm.dead) break;
      tc_fence_after();
      const uint32_t acc = tmem + (uint32_t)buf * BN + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < n_cols; c += CH, ++chunk_no) {
        TC* stage_out = sm.out[chunk_no & 1];
        // the store that last used this buffer (two chunks ago) must have read it
        if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
        for (int h = 0; h < CH / 16; ++h) {
          uint32_t v[16];
          tmem_ld16(acc + (uint32_t)(c + h * 16), v);
          if (SUMS == 2) {
            uint32_t second[16];
            tmem_ld16(acc + (uint32_t)(BN + c + h * 16), second);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(second[j]));
          } else {
            tmem_ld_wait();
          }
          if (GATED) {
            const int f = q * 16 + (lane & 15);
            const int col0 = h * 16 + (lane < 16 ? 0 : 8);
            float r[8];
            if (EPI == EPI_CLAMPED) {
              float sc[8];
#pragma unroll
              for (int i = 0; i < 8; ++i)
                sc[i] = GROUPED && grouping.row_scale ? grouping.row_scale[min(t0 + c + col0 + i, T - 1)] : 1.f;
              clamped_columns<TC>(v, lane, act_limit, sc, r);
            } else {
              gated_columns<TC>(v, lane, r);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) stage_out[(col0 + i) * FEAT + f] = from_f32<TC>(r[i]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float z = __uint_as_float(v[j]);
              if (EPI == EPI_RELU2) z = relu_squared(z);
              stage_out[(h * 16 + j) * FEAT + row] = from_f32<TC>(z);
            }
          }
        }
        if (c + CH >= n_cols) {           // this accumulator has been read completely
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            for (int b = buf; b < buf + SUMS; ++b) {
              if (leader) mbar_arrive_local(&sm.acc_empty[b]);
              else mbar_arrive_in(&sm.acc_empty[b], 0);
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (issuer) {
          const uint32_t src = smem_u32(stage_out);
          if (EPI == EPI_ACCUM)
            asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
                         ::"l"(&map_c), "r"(src), "r"(n0), "r"(t0 + c) : "memory");
          else
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                         ::"l"(&map_c), "r"(src), "r"(n0), "r"(t0 + c) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  // Neither CTA may go while the other can still read its shared memory, signal its barriers or
  // write its tensor memory.
  tc_fence_before();
  __syncwarp();
  pair_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// The last tokens of a T that is not a multiple of 256 make shorter items where they are at most half a
// tile and there are fewer than four whole ones.  A pair's time for a tile falls with its tokens only
// where the box of tokens does too (up to 128: see load_w), and the variant with a width read at run time
// loses about 1 % on the whole tiles, which four or more of them make more than the padding.  The four
// products of a layer, padded -> narrow, us: Qwen3-0.6B widths 600 / 840 tokens 60 -> 58 / 67 -> 64, 4B 163 ->
// 156 / 194 -> 192, 8B 220 -> 218 / 322 -> 321 (its matrices of 100 and 200 MB follow their tiles, see below:
// 780 tokens 311 -> 317, 896 329 -> 324).  Tried wider: with 129 to 255 tokens left 0.6B widths 641 / 720 / 900 /
// 1,020 tokens 563 / 566 / 648 / 661 -> 597 / 580 / 634 / 667 (twelve layers), beyond four tiles 1,280 and
// 2,060 789 / 908 -> 790 / 911: nothing.
bool short_tail(int T) { return T < 4 * BN && T % BN != 0 && T % BN <= BN / 2; }
// Dealt last, the short items even out the pairs, but they meet every weight a second time: fine
// while the weights stay in the L2 (some 48 MB), else they follow their tiles (600 tokens 1,199 ->
// 1,187 us, 1,100 tokens 1,869 -> 1,858).
bool tail_in_order(int N, int K) { return (long long)N * K * 2 > 48LL << 20; }

// What a product in s ranges of K takes, in blocks of K of a whole tile: a work item costs its 64-wide
// blocks of K plus about six blocks' worth of start and epilogue (fitted to measured times of seven
// shapes), an item of last tokens less where they are dealt last.
double rounds_cost(int N, int K, int T, int pairs, int s) {
  const bool tail = short_tail(T) && !tail_in_order(N, K);
  const int m_tiles = (N + 2 * TILE_M - 1) / (2 * TILE_M), nkb = (K + TILE_K - 1) / TILE_K;
  const int whole = m_tiles * (tail ? T / BN : (T + BN - 1) / BN) * s, rest = tail ? m_tiles * s : 0;
  const int first = (whole + pairs - 1) / pairs, all = (whole + rest + pairs - 1) / pairs;
  return first * ((double)nkb / s + 6.0) + (all - first) * ((double)nkb / s * (0.25 + 0.75 * (T % BN) / BN) + 5.0);
}

// The adding epilogue lets K be cut.  With few tiles to a pair the last round of tiles leaves
// most pairs idle (160 tiles on 74 pairs: three rounds for the work of 2.2), and with fewer
// tiles than pairs some never work.  K is cut into the number of ranges, each of at least eight
// blocks, for which the rounds of whole tiles cost least.  (Narrow last tiles do not enter: how often a
// sum is cut decides its rounding, and one range alone gives the same bits every time.)
int cheapest_cut(int m_tiles, int T, int nkb, int pairs) {
  const int tiles = m_tiles * ((T + BN - 1) / BN);
  int ksplits = 1;
  double best = 0;
  for (int s = 1; s <= 8 && nkb / s >= 8; ++s) {
    const int rounds = (tiles * s + pairs - 1) / pairs;
    const double cost = rounds * ((double)nkb / s + 6.0);
    if (s == 1 || cost < best * 0.99) best = cost, ksplits = s;
  }
  return ksplits;
}

int pair_sm_count() {
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (sm_count <= 0) sm_count = 148;
  }
  return sm_count;
}

template <int STAGES, int EPI, typename TC, int FORM>
constexpr int pair_smem() {
  return (int)sizeof(PairStorage<STAGES, gated_epilogue(EPI) ? 64 : TILE_M, TC, FORM == GROUPED_TILES>) + 1024;
}

// As many pairs as the device holds at once (an SM without a free neighbour stays empty), at most one
// per two SMs; negative: a CUDA error, 0: no pair of this kernel fits.
template <int STAGES, int EPI, typename TC, int FORM>
int resident_pairs() {
  static int pairs = 0;
  if (pairs) return pairs;
  auto kernel = gemm_pair_kernel<STAGES, EPI, TC, FORM>;
  constexpr int smem = pair_smem<STAGES, EPI, TC, FORM>();
  static_assert(smem <= 227 * 1024, "the stages and output chunks fit one SM");
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return -(int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(192);
  cfg.gridDim = dim3(pair_sm_count() & ~1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    return 0;
  }
  return pairs = n < pair_sm_count() / 2 ? n : pair_sm_count() / 2;
}

template <int STAGES, int EPI, typename TC, int FORM>
int launch_form(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mxs, const CUtensorMap& mc, int T, int N,
           int K, int half, int* status, cudaStream_t stream, float act_limit = 0.f,
           const Grouping& grouping = Grouping(), int ranges = 0) {
  constexpr bool GATED = gated_epilogue(EPI), GROUPED = FORM == GROUPED_TILES;
  constexpr int FEAT = GATED ? 64 : TILE_M;
  auto kernel = gemm_pair_kernel<STAGES, EPI, TC, FORM>;
  const int most = resident_pairs<STAGES, EPI, TC, FORM>();
  if (most <= 0) return most < 0 ? -most : LLM_ERR_UNSUPPORTED;
  const int limit = GATED ? half : N;
  const int m_tiles = (limit + 2 * FEAT - 1) / (2 * FEAT), n_tiles = GROUPED ? grouping.n_small : (T + BN - 1) / BN;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = pair_smem<STAGES, EPI, TC, FORM>();
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  int ksplits = 1;
  if (EPI == EPI_ACCUM) {
    const int nkb = (K + TILE_K - 1) / TILE_K;
    ksplits = ranges > 0 ? ranges : cheapest_cut(m_tiles, T, nkb, most);
    if (g_llm_pair_ksplits > 0 && nkb / g_llm_pair_ksplits >= 1) ksplits = g_llm_pair_ksplits;
  }
  const int works = m_tiles * n_tiles * ksplits;
  const int pairs = works < most ? works : most;
  cfg.gridDim = dim3(2 * pairs);
  // directly behind the rotation kernel the pair kernel starts only when that kernel is done
  cfg.numAttrs = (g_llm_pdl && !g_llm_after_rotation) ? 2 : 1;
  g_llm_after_rotation = 0;
  return (int)cudaLaunchKernelEx(&cfg, kernel, mw, mx, mxs, mc, T, N, K, half, m_tiles, n_tiles, ksplits, act_limit, status,
                                 grouping);
}

template <int STAGES, int EPI, typename TC>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mxs, const CUtensorMap& mc, int T, int N,
           int K, int half, int* status, cudaStream_t stream, float act_limit = 0.f, int ranges = 0) {
  Grouping g = Grouping();
  g.k_up = ranges > 0;
  if (short_tail(T)) {
    g.in_order = tail_in_order(N, K);
    return launch_form<STAGES, EPI, TC, LAST_TOKENS>(mw, mx, mxs, mc, T, N, K, half, status, stream, act_limit, g,
                                                     ranges);
  }
  return launch_form<STAGES, EPI, TC, WHOLE_TILES>(mw, mx, mxs, mc, T, N, K, half, status, stream, act_limit, g,
                                                   ranges);
}
}  // namespace

// How a 32-bit product of many rows with few tiles, for which the caller asked for a split of K, is
// made soonest: 0 without additions in memory on pairs, 1 the output cleared and ranges of K added into
// it on pairs, 2 the same on lone CTAs with tiles of 128 x 128 in `splits` ranges.  In units of one
// 64-wide block of K of a pair's tile (0.39 us): clearing is a launch and a pass over the output (2.5
// us, then 3 TB/s with the additions' own traffic); a lone CTA's block is 1.4 units with two CTAs to an SM.
// Two sums that are added into zeros commute, so a product that is asked for in two ranges gives the
// same bits every time, and keeps them in all three ways (two sums in the first, the same two ranges in
// the second).  Three or more have no order in memory, so how many there are is free.
// Measured, lone CTAs against the choice made here, with weights from memory: 2,048 x 1,024 x 3,072
// (rows x N x K) 39.6 -> 27.4 us (ranges of K), 777 x 4,096 x 1,024 29.7 -> 20.5 (two sums; one sum 19.5,
// two ranges added in memory 26.6), 1,501 x 4,096 x 4,096 70.5 -> 57.3 (two ranges; one sum 56.3, two sums
// 61.5); 513 x 1,024 x 1,024 stays on lone CTAs (15.4 against 18.4 on pairs).
LLM_EXPORT int llm_pair_store_way(int T, int N, int K, int splits) {
  const int pairs = g_llm_pair ? resident_pairs<5, EPI_STORE, float, WHOLE_TILES>() : 0;
  if (pairs <= 0) return 2;
  const int nkb = (K + TILE_K - 1) / TILE_K;
  const int m_tiles = (N + 2 * TILE_M - 1) / (2 * TILE_M);
  const double clear = (2.5 + (double)T * N * 4 / 3e6) / 0.39;
  // (two sums leave no accumulator for the next tile: every round but the last waits for its epilogue)
  const int rounds = (m_tiles * ((T + BN - 1) / BN) + pairs - 1) / pairs;
  const double whole = rounds_cost(N, K, T, pairs, 1) + (splits == 2 ? 6.0 * (rounds - 1) : 0.0);
  const int s = splits == 2 ? 2 : cheapest_cut(m_tiles, T, nkb, pairs);
  const double cut = s == 1 ? 1e30 : rounds_cost(N, K, T, pairs, s);
  const long long lone = (long long)((N + TILE_M - 1) / TILE_M) * ((T + 127) / 128) * splits;
  const double alone = (double)((lone + 2 * pair_sm_count() - 1) / (2 * pair_sm_count())) * (1.4 * nkb / splits + 6.0) + clear;
  if (alone < whole && alone < cut + clear) return 2;
  return cut + clear < whole ? 1 : 0;
}

// The pair kernel for bfloat16 X [T][K], W [N][K]; modes 0, 1, 3 and 4 of llm_gemm_tcgen05 (no K
// split but in mode 1, in `ranges` ranges or, for 0, as many as are soonest, and in mode 0 with 32-bit C
// as two sums for ranges = 2; the gated form only with interleaved rows).  Returns LLM_ERR_UNSUPPORTED when the output
// cannot be written by TMA or the mode is not one of these: the caller then uses the one-CTA kernel.
LLM_EXPORT void llm_set_pair_ksplits(int n) { g_llm_pair_ksplits = n; }
LLM_EXPORT void llm_set_pair(int on) { g_llm_pair = on ? 1 : 0; }

int llm_gemm_tcgen05_pair(const void* X, const void* W, void* C, int c_dtype, int T, int N, int K, int lda,
                          int ldw, int ldc, int mode, int half, float limit, int ranges, int* status, cudaStream_t stream) {
  if (!g_llm_pair) return LLM_ERR_UNSUPPORTED;
  if (mode != 0 && mode != 1 && mode != 3 && mode != 4) return LLM_ERR_UNSUPPORTED;
  const int esize = c_dtype == LLM_F32 ? 4 : 2;
  if (((uintptr_t)C & 15) || ((size_t)ldc * esize) % 16) return LLM_ERR_UNSUPPORTED;
  CUtensorMap mw, mx, mxs, mc;
  if (!llm_tensor_map(W, N, K, ldw, TILE_M, TILE_K, 0, &mw)) return LLM_ERR_UNSUPPORTED;
  if (!llm_tensor_map(X, T, K, lda, HALF_N, TILE_K, 0, &mx)) return LLM_ERR_UNSUPPORTED;
  mxs = mx;      // (read for narrow last tokens alone)
  if (short_tail(T) && !llm_tensor_map(X, T, K, lda, HALF_N / 2, TILE_K, 0, &mxs)) return LLM_ERR_UNSUPPORTED;
  const int out_cols = mode >= 3 ? half : N;
  if (!llm_tensor_map(C, T, out_cols, ldc, CH, mode >= 3 ? 64 : TILE_M, c_dtype == LLM_F32 ? 2 : 1, &mc))
    return LLM_ERR_UNSUPPORTED;
  if (mode == 0) {
    if (c_dtype == LLM_F32 && ranges == 2)
      return launch<5, EPI_TWO_SUMS, float>(mw, mx, mxs, mc, T, N, K, half, status, stream);
    if (c_dtype == LLM_F32) return launch<5, EPI_STORE, float>(mw, mx, mxs, mc, T, N, K, half, status, stream);
    if (c_dtype == LLM_BF16) return launch<6, EPI_STORE, bf16>(mw, mx, mxs, mc, T, N, K, half, status, stream);
  } else if (mode == 1) {
    if (c_dtype == LLM_F32) return launch<5, EPI_ACCUM, float>(mw, mx, mxs, mc, T, N, K, half, status, stream, 0.f, ranges);
  } else {
    if (N != 2 * half || half % 16) return LLM_ERR_ARGUMENT;
    if (mode == 4)
      return c_dtype == LLM_BF16 ? launch<6, EPI_CLAMPED, bf16>(mw, mx, mxs, mc, T, N, K, half, status, stream, limit)
                                 : LLM_ERR_UNSUPPORTED;
    if (c_dtype == LLM_BF16) return launch<6, EPI_GATED, bf16>(mw, mx, mxs, mc, T, N, K, half, status, stream);
    if (c_dtype == LLM_F32) return launch<6, EPI_GATED, float>(mw, mx, mxs, mc, T, N, K, half, status, stream);
  }
  return LLM_ERR_UNSUPPORTED;
}

// The grouped product of llm_gemm_tcgen05_grouped on CTA pairs: tile i of bn rows of X (32, 64 or 128)
// with matrix tile_group[i] of W, at most 512 tiles.  mode 0: C f32; 3 and 4: the gated forms with
// interleaved rows, C bf16 [T][half]; 5: C = max(X W_g^T, 0)^2, bf16.
LLM_EXPORT int llm_gemm_tcgen05_grouped_pair(const void* X, const void* W, void* C, int c_dtype, int T, int N, int K,
                                             int lda, int ldw, int ldc, int mode, int half, int bn, int groups,
                                             const int* tile_group, float limit, const float* row_scale, int* status,
                                             cudaStream_t stream) {
  if (T <= 0 || N <= 0 || groups <= 0) return 0;
  if (!tile_group || (mode != 0 && mode != 3 && mode != 4 && mode != 5)) return LLM_ERR_ARGUMENT;
  const bool gated = mode == 3 || mode == 4;
  if (gated && (N != 2 * half || half % 16)) return LLM_ERR_ARGUMENT;
  if (bn != 32 && bn != 64 && bn != 128) return LLM_ERR_UNSUPPORTED;
  if (K <= 0 || K % 8 || lda % 8 || ldw % 8 || (((uintptr_t)X | (uintptr_t)W) & 15)) return LLM_ERR_UNSUPPORTED;
  if ((long long)groups * N > 0x7fffffffLL || (mode == 0) != (c_dtype == LLM_F32)) return LLM_ERR_UNSUPPORTED;
  const int esize = c_dtype == LLM_F32 ? 4 : 2;
  if (((uintptr_t)C & 15) || ((size_t)ldc * esize) % 16) return LLM_ERR_UNSUPPORTED;
  Grouping g = Grouping();
  g.tile_group = tile_group, g.bn = bn, g.n_small = (T + bn - 1) / bn, g.group_rows = N, g.row_scale = row_scale;
  if (g.n_small > MAX_SMALL) return LLM_ERR_UNSUPPORTED;
  CUtensorMap mw, mx, mxs, mc;
  if (!llm_tensor_map(W, (long long)groups * N, K, ldw, TILE_M, TILE_K, 0, &mw)) return LLM_ERR_UNSUPPORTED;
  if (!llm_tensor_map(X, T, K, lda, HALF_N, TILE_K, 0, &mx)) return LLM_ERR_UNSUPPORTED;
  if (!llm_tensor_map(X, T, K, lda, HALF_N / 2, TILE_K, 0, &mxs)) return LLM_ERR_UNSUPPORTED;
  if (!llm_tensor_map(C, T, gated ? half : N, ldc, CH, gated ? 64 : TILE_M, c_dtype == LLM_F32 ? 2 : 1, &mc))
    return LLM_ERR_UNSUPPORTED;
  if (mode == 0) return launch_form<5, EPI_STORE, float, GROUPED_TILES>(mw, mx, mxs, mc, T, N, K, half, status, stream, 0.f, g);
  if (mode == 3) return launch_form<6, EPI_GATED, bf16, GROUPED_TILES>(mw, mx, mxs, mc, T, N, K, half, status, stream, 0.f, g);
  if (mode == 4) return launch_form<6, EPI_CLAMPED, bf16, GROUPED_TILES>(mw, mx, mxs, mc, T, N, K, half, status, stream, limit, g);
  return launch_form<6, EPI_RELU2, bf16, GROUPED_TILES>(mw, mx, mxs, mc, T, N, K, half, status, stream, 0.f, g);
}
