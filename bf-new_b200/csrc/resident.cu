// Frontier searches outside the grid-wide kernels: one lane (net) of a batch is
// relaxed by one thread-block cluster whose shared memories hold all of the
// net's distances; larger whole-graph lanes by a team of blocks (below).
//
// What bounds the grid-wide frontier (frontier.cuh) on regional sets is the
// memory system: every relaxation reads a random 8-byte label, the labels of
// a set exceed the L2, and random 32-byte sectors beyond the L2 are served at
// about 37 G/s on a B200; and its rounds end in a barrier of the whole grid,
// so a round costs its slowest item.  A regional net is small, though: its
// distances (4 bytes a vertex) fit the shared memory of 1 to 16 blocks.  Here
// a relaxation is a shared-memory minimum (the own block's, or a cluster
// neighbour's over distributed shared memory), a round ends in a cluster
// barrier, nets do not wait for one another, and global memory is read only
// for edge records and written once for the result.
//
// Per block: distances L, two pending bitmaps (this round, next round) and a
// far bitmap, all indexed by the net's own compact index.  The net's selected
// tiles are numbered in order; each tile starts on a 32-vertex word, and runs
// of words are dealt to the cluster's blocks in turn.  The tile directory
// (bit and rank per 32 tiles) is the admission test of an edge and leads to
// the tile's bias, so destination vertex + bias = compact index.
//
// Rounds are those of the near/far frontier: improvements below the threshold
// are pending in the next round, the others are marked far; when no vertex is
// pending, the threshold rises to the smallest far distance + delta.  The
// predecessor is found once, after convergence: the smallest stable edge id
// among the admitted in-edges that give the vertex's distance -- what the
// packed 64-bit minimum of the other frontier kernels ends in.
//
// Host-polled runs (kPolled) launch a search for a chunk of rounds at a time.
// Between the launches its distances are in the label rows, without
// predecessors, its pending and far bitmaps in the lane's part of the second
// label slot (8 bytes a vertex of the union, so 8 a word fit), and its scalars
// in a SearchProgress.
//
// A round of a full block (49 K vertices) costs about 6 us -- two dependent
// global reads (row, records), the list of pending vertices, the barrier --
// plus 0.55 ns per relaxed edge (1 ns in a cluster of 8, where a fifth of the
// targets are in other blocks).  Neither DRAM (15 % of its rate) nor the L2
// (3 %) bounds it: a warp waits at the round's barriers, then for the records.
// Rows are read as one list of edges per 32 vertices: with 2 or 4 threads per row the
// loads' partial lines bounded the launch (B200, 256 regional nets, 2.1 M
// vertices, when measured: 12.4 and 10.6 ms against 10.5).  Relaxation launch of
// that set 22.6 -> 10.2 ms; 512 nets on 65 K vertices 7.8 -> 1.7 ms; 8 whole
// images of 65 K vertices 2.18 -> 0.47 ms; one net of 4,096 vertices 0.26 ->
// 0.11 ms.
#include "resident.cuh"

#include <cstddef>

namespace bfx {
namespace {

constexpr u32 kFull = 0xFFFFFFFFu;
constexpr u32 kPad = 0xFFFFFFFFu;   // L of a word's slots beyond its tile
constexpr u32 kMaxCluster = 16u;
constexpr u32 kListPer = 4u;        // pending vertices of a pass, per thread
constexpr size_t kBlockBytes = 225 * 1024;  // dynamic shared memory of one block, at most

// Block configurations, smallest share of an SM first: 256 and 512 threads
// (four and two blocks per SM, shared memory in proportion), one block per
// SM, clusters of 2 to 16 such blocks.
struct Shape {
  u32 ctas, threads;
  size_t bytes;   // dynamic shared memory limit per block
};
constexpr Shape kShapes[] = {{1, 256, 54 * 1024},  {1, 512, 111 * 1024}, {1, 1024, kBlockBytes}, {2, 1024, kBlockBytes},
                             {3, 1024, kBlockBytes}, {4, 1024, kBlockBytes}, {6, 1024, kBlockBytes},
                             {8, 1024, kBlockBytes}, {12, 1024, kBlockBytes}, {16, 1024, kBlockBytes}};
constexpr u32 kShapeCount = sizeof(kShapes) / sizeof(kShapes[0]);
// Nets that leave SMs idle are spread over larger shapes, up to 8 blocks and
// at least 64 words (2,048 vertices) a block: below that a round is its fixed
// latency (one 4,096-vertex net: 0.10 ms on 4 blocks, 0.23 ms on one).
constexpr size_t kLaunchStreams = 8;
constexpr u64 kTeamBytes = u64{270} << 20;
constexpr u32 kSpreadShape = 7u, kSpreadWords = 64u;

__host__ __device__ __forceinline__ u32 block_words(u32 words, u32 ctas, u32 run) {
  const u32 per = ctas << run;
  return ((words + per - 1u) / per) << run;
}

// --- distributed shared memory ---------------------------------------------

__device__ __forceinline__ u32 shared_address(const void* p) { return static_cast<u32>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ u32 map_rank(u32 address, u32 rank) {
  u32 r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(address), "r"(rank));
  return r;
}
// Loads and reductions by shared-memory address: here: in the own block, else
// in any block of the cluster (kCluster).  Neighbours lower the same words at
// the same time, so in a cluster both forms have cluster scope: two accesses
// whose scopes do not include each other's thread would not be atomic to one
// another.  Both are predicated, not branched to, so the loads of several
// edges are in flight together.
template <bool kCluster>
__device__ __forceinline__ u32 shared_load(u32 a, bool here) {
  u32 v;
  if (kCluster) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p ld.relaxed.cluster.shared::cta.u32 %0, [%1];\n\t@!p ld.relaxed.cluster.shared::cluster.u32 %0, [%1];\n\t}"
        : "=r"(v)
        : "r"(a), "r"(static_cast<u32>(here))
        : "memory");
  } else {
    asm volatile("ld.relaxed.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  }
  return v;
}
template <bool kCluster>
__device__ __forceinline__ void shared_min(u32 a, u32 v, bool here) {
  if (kCluster) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p red.relaxed.cluster.shared::cta.min.u32 [%0], %1;\n\t"
        "@!p red.relaxed.cluster.shared::cluster.min.u32 [%0], %1;\n\t}" ::"r"(a),
        "r"(v), "r"(static_cast<u32>(here))
        : "memory");
  } else {
    asm volatile("red.relaxed.cta.shared::cta.min.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
}
template <bool kCluster>
__device__ __forceinline__ void shared_or(u32 a, u32 v, bool here) {
  if (kCluster) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p red.relaxed.cluster.shared::cta.or.b32 [%0], %1;\n\t"
        "@!p red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;\n\t}" ::"r"(a),
        "r"(v), "r"(static_cast<u32>(here))
        : "memory");
  } else {
    asm volatile("red.relaxed.cta.shared::cta.or.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
}
__device__ __forceinline__ void remote_store(u32 a, u32 v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ u32 cluster_rank() {
  u32 r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// Barrier over the cluster (the block alone when it is its own cluster);
// executed by all threads.
__device__ __forceinline__ void cluster_sync(u32 ctas) {
  if (ctas == 1u) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// The step of a set without steps of its own (LaunchParams::auto_step) after
// its n-th split: doubled every eighth time, so that weights which spread over
// many orders of magnitude cost a logarithm of splits and not one per band.
__device__ __forceinline__ u32 grown_step(u32 step, u32 n) {
  return (n & 7u) == 0u ? __float_as_uint(__fadd_rn(__uint_as_float(step), __uint_as_float(step))) : step;
}

struct NetShared {
  u32 scan[33];
  u32 any[3];                  // a vertex is pending: by round % 3
  u32 stop;                    // the launch budget is spent
  u32 listed[2], cut[2];       // list of pending vertices, by pass parity: slots asked for, and where it was full
  u32 fmin[2][kMaxCluster];    // smallest far distance of each block, by split parity
};

// Block-wide exclusive scan of get(i), i < n, into put(i, sum); returns the
// total.  Executed by all threads.
template <typename Get, typename Put>
__device__ u32 block_scan(NetShared& s, u32 n, Get get, Put put) {
  const u32 per = (n + blockDim.x - 1u) / blockDim.x;
  const u32 begin = threadIdx.x * per, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  u32 local = 0u;
  for (u32 i = begin; i < min(begin + per, n); ++i) local += get(i);
  u32 x = local;
  for (u32 o = 1; o < 32u; o <<= 1) {
    const u32 y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31u) s.scan[warp] = x;
  __syncthreads();
  if (warp == 0u) {
    const u32 nw = blockDim.x >> 5;
    const u32 t = lane < nw ? s.scan[lane] : 0u;
    u32 z = t;
    for (u32 o = 1; o < 32u; o <<= 1) {
      const u32 y = __shfl_up_sync(kFull, z, o);
      if (lane >= o) z += y;
    }
    s.scan[lane] = z - t;
    if (lane == 31u) s.scan[32] = z;
  }
  __syncthreads();
  u32 run = s.scan[warp] + x - local;
  for (u32 i = begin; i < min(begin + per, n); ++i) {
    const u32 y = get(i);
    put(i, run);
    run += y;
  }
  const u32 total = s.scan[32];
  __syncthreads();
  return total;
}

// The edges of up to 32 rows (row: {first, count}, one per thread, threads
// beyond `take` none) as one list, so that a warp reads consecutive records
// and every thread has an edge whatever the rows' lengths.
constexpr u32 kSteps = 4u;  // list steps of 32 edges whose records are in flight together
struct EdgeList {
  u32 excl, shift, total;
  bool dense;  // every row of the first `take` has an edge: rows start at different places
  __device__ __forceinline__ EdgeList(uint2 row, u32 take) {
    const u32 lane = threadIdx.x & 31u;
    u32 incl = row.y;
    for (u32 o = 1; o < 32u; o <<= 1) {
      const u32 y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    excl = incl - row.y;
    shift = row.x - excl;
    total = __shfl_sync(kFull, incl, 31);
    dense = __all_sync(kFull, row.y != 0u || lane >= take);
    if (lane >= take) excl = kFull;
  }
  // Record of the thread's edge in the step at `base`, and its row's thread.
  __device__ __forceinline__ u32 edge(u32 base, u32& from, bool& live) const {
    const u32 lane = threadIdx.x & 31u;
    if (dense) {
      // rows that start in the step, one bit each; the row of a place is the
      // last that starts at or before it
      const u32 rel = excl - base;
      const u32 starts = __reduce_or_sync(kFull, rel < 32u ? 1u << rel : 0u);
      const u32 earlier = static_cast<u32>(__popc(__ballot_sync(kFull, excl < base)));
      from = earlier + static_cast<u32>(__popc(starts & ((2u << lane) - 1u))) - 1u;
    } else {
      u32 lo = 0u;
      for (u32 s = 16u; s > 0u; s >>= 1) {
        const u32 y = __shfl_sync(kFull, excl, static_cast<int>(lo + s));
        if (y <= base + lane) lo += s;
      }
      from = lo;
    }
    live = base + lane < total;
    from = live ? from : 0u;
    return base + lane + __shfl_sync(kFull, shift, static_cast<int>(from));
  }
};

// Where a compact index lives: block and slot.
struct Place {
  u32 owner, slot;
};

// kCluster: the net's words are dealt to several blocks (ctas > 1).  kWhole:
// every tile is one run of words, so it lies in one block and its distances
// are contiguous there.  kPolled: at most `chunk` rounds.
template <bool kCount, bool kCluster, bool kWhole, bool kPolled>
__global__ void __launch_bounds__(1024, 1)
    resident_kernel(LaunchParams p, const ResidentNet* nets, u32 cluster_ctas, u32 run, SearchProgress* progress,
                    u32 chunk) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ NetShared s;
  const u32 ctas = kCluster ? cluster_ctas : 1u;
  const ResidentNet net = nets[blockIdx.x / ctas];
  const u32 b = net.batch, ql = net.lane;
  const u32 rank = kCluster ? cluster_rank() : 0u;
  // uniform over the cluster
  if (engine_of(p, b) != BFX_ENGINE_FRONTIER_PUSH) return;
  SearchProgress was{};  // written at the end of an earlier launch
  if (kPolled) {
    was = progress[blockIdx.x / ctas];
    if (was.done != 0u) return;
  }
  const bool resumed = kPolled && was.rounds != 0u;
  const DBatch& B = p.batches[b];
  u32* const saved_near = reinterpret_cast<u32*>(B.dist[1] + static_cast<u64>(B.U) * ql);  // by the net's words
  u32* const saved_far = saved_near + net.words;
  DCtl& C = p.ctl[b];
  const u32 T = p.g.T, dw = (T + 31u) >> 5;
  const u32 M = block_words(net.words, ctas, run);  // words of this block
  uint2* const dir = reinterpret_cast<uint2*>(smem);
  u32* const L = reinterpret_cast<u32*>(dir + dw);
  u32* const near0 = L + M * 32u;
  u32* const near1 = near0 + M;
  u32* const far = near1 + M;
  u32* const gbase = far + M;          // first vertex of each word
  u32* const gtile = gbase + M;        // tile of each word
  // by tile rank, kWhole: {address of the tile's distances - 4 * its first
  // vertex, slot of its first vertex - that vertex}; else {compact index of
  // its first vertex - that vertex, 0}
  uint2* const where = reinterpret_cast<uint2*>(gtile + M + (M & 1u));
  unsigned short* const list = reinterpret_cast<unsigned short*>(where + net.tiles);  // pending slots of a pass
  const u32 list_cap = blockDim.x * kListPer;
  const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
  const u32 run_mask = (1u << run) - 1u;
  const u32 per_cta = kCluster ? 0xFFFFFFFFu / ctas + 1u : 0u;  // exact quotients below 2^28
  const auto place = [&](u32 idx) {
    if (!kCluster) return Place{0u, idx};
    const u32 w = idx >> 5, q = w >> run, deal = __umulhi(q, per_cta);  // q / ctas
    return Place{q - deal * ctas, (((deal << run) | (w & run_mask)) << 5) | (idx & 31u)};
  };
  const u32 L_at = shared_address(L);
  const u64 t0 = p.run->started;  // the budget is the relaxation's, however long the search was queued

  // --- the net's tiles and words -------------------------------------------
  for (u32 i = tid; i < dw; i += blockDim.x) dir[i] = make_uint2(0u, 0u);
  for (u32 i = tid; i < M * 32u; i += blockDim.x) L[i] = kPad;
  for (u32 i = tid; i < M; i += blockDim.x) near0[i] = near1[i] = far[i] = gbase[i] = gtile[i] = 0u;
  if (tid < 3u) s.any[tid] = 0u;
  if (tid == 3u) s.stop = s.listed[0] = s.listed[1] = 0u;
  if (tid == 4u) s.cut[0] = s.cut[1] = kFull;
  __syncthreads();
  const u32 R = B.range_count;
  for (u32 i = tid; i < R; i += blockDim.x) {
    const uint4 r = __ldg(B.ranges + i);
    if ((r.w >> ql) & 1u) atomicOr(&dir[r.x >> 5].x, 1u << (r.x & 31u));
  }
  __syncthreads();
  const u32 tiles = block_scan(s, dw, [&](u32 i) { return static_cast<u32>(__popc(dir[i].x)); },
                               [&](u32 i, u32 x) { dir[i].y = x; });
  const auto rank_of = [&](u32 tile) {
    const uint2 d = dir[tile >> 5];
    return d.y + static_cast<u32>(__popc(d.x & ((1u << (tile & 31u)) - 1u)));
  };
  bool sound = tiles == net.tiles;  // uniform: every block builds the same directory
  if (sound) {
    for (u32 i = tid; i < R; i += blockDim.x) {
      const uint4 r = __ldg(B.ranges + i);
      if ((r.w >> ql) & 1u) where[rank_of(r.x)].x = (r.z - r.y + 31u) >> 5;
    }
    __syncthreads();
    sound = block_scan(s, tiles, [&](u32 i) { return where[i].x; }, [&](u32 i, u32 x) { where[i].x = x; }) == net.words;
  }
  if (!sound) {  // the host's sizes are not the description's: nothing was written beyond them
    if (tid == 0u && rank == 0u) atomicOr(&C.error_bits, static_cast<u32>(BFX_DEVICE_ERROR_INVALID_CONTROLLER_STATE));
    return;
  }
  for (u32 base = warp * 32u; base < R; base += warps * 32u) {
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (base + lane < R) r = __ldg(B.ranges + base + lane);
    const u32 mine = ((r.w >> ql) & 1u) != 0u && r.z > r.y ? 1u : 0u;
    u32 first = 0u;
    if (mine) {
      const u32 ord = rank_of(r.x);
      first = where[ord].x;
      if (kWhole) {
        const Place at = place(first * 32u);
        const u32 base = kCluster ? map_rank(L_at, at.owner) : L_at;
        where[ord] = make_uint2(base + (at.slot - r.y) * 4u, at.slot - r.y);
      } else {
        where[ord] = make_uint2(first * 32u - r.y, 0u);
      }
    }
    for (u32 todo = __ballot_sync(kFull, mine); todo != 0u; todo &= todo - 1u) {
      const int from = __ffs(todo) - 1;
      const u32 begin = __shfl_sync(kFull, r.y, from), end = __shfl_sync(kFull, r.z, from);
      const u32 word = __shfl_sync(kFull, first, from), tile = __shfl_sync(kFull, r.x, from);
      for (u32 k = 0; k * 32u < end - begin; ++k) {
        const Place at = place((word + k) * 32u);
        if (at.owner != rank) continue;
        if (k * 32u + lane < end - begin) {
          u32 d = dev::kInfBits;
          if (resumed) {
            const u32 cv = begin + k * 32u + lane - B.tiles[tile].y;
            d = dev::hi(B.dist[0][(static_cast<u64>(cv) << B.shift) + ql]);
          }
          L[at.slot + lane] = d;
        }
        if (lane == 0u) {
          gbase[at.slot >> 5] = begin + k * 32u;
          gtile[at.slot >> 5] = tile;
          if (resumed) {
            ((was.rounds & 1u) ? near1 : near0)[at.slot >> 5] = saved_near[word + k];
            far[at.slot >> 5] = saved_far[word + k];
          }
        }
      }
    }
  }
  cluster_sync(ctas);  // every block's distances are set up
  // Address of an endpoint's distance and its slot (at - 4 * slot: the
  // address of its block's distances); at == 0: its tile is not selected.
  struct Endpoint {
    u32 at, slot;
  };
  const auto endpoint = [&](const uint4& rec) {
    const uint2 d = dir[rec.w >> 5];
    const u32 bit = 1u << (rec.w & 31u);
    if ((d.x & bit) == 0u) return Endpoint{0u, 0u};
    const uint2 t = where[d.y + static_cast<u32>(__popc(d.x & (bit - 1u)))];
    if (kWhole) return Endpoint{t.x + rec.x * 4u, t.y + rec.x};
    const Place pl = place(t.x + rec.x);
    return Endpoint{map_rank(L_at, pl.owner) + pl.slot * 4u, pl.slot};
  };
  const u32 near0_off = M * 128u;  // offsets from L
  // --- sources ---------------------------------------------------------------
  const u32 src0 = B.src_off[ql], src1 = B.src_off[ql + 1u];
  for (u32 i = resumed ? src1 : src0 + tid; i < src1; i += blockDim.x) {
    const u32 v = B.src[i], t = p.g.owner[v];
    if (((dir[t >> 5].x >> (t & 31u)) & 1u) == 0u) continue;  // reported by the seed kernel
    const Endpoint e = endpoint(make_uint4(v, 0u, 0u, t));
    shared_min<kCluster>(e.at, 0u, false);
    shared_or<kCluster>(e.at - e.slot * 4u + near0_off + (e.slot >> 5) * 4u, 1u << (e.slot & 31u), false);
  }
  cluster_sync(ctas);

  // --- rounds ------------------------------------------------------------------
  u32 delta = p.deltas ? p.deltas[b] : p.auto_step;
  u32 tau = delta, splits = 0u, rounds = 0u, pass = 0u;
  if (resumed) {
    delta = was.delta;
    tau = was.tau;
    splits = was.splits;
    rounds = was.rounds;
  }
  bool paused = false;
  u32 cnt[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  u64 total_cnt[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  for (;; ++rounds) {
    u32* const cur = (rounds & 1u) ? near1 : near0;
    u32* const nxt = (rounds & 1u) ? near0 : near1;
    if (kPolled && rounds - was.rounds == chunk) {
      // after a barrier, so no neighbour changes this block's words any more
      for (u32 w = warp; w < M; w += warps) {
        const u32 of = kCluster ? ((((w >> run) * ctas + rank) << run) | (w & run_mask)) : w;  // the net's word
        const u32 d = L[w * 32u + lane];
        if (d != kPad) {
          const u32 cv = gbase[w] + lane - B.tiles[gtile[w]].y;
          B.dist[0][(static_cast<u64>(cv) << B.shift) + ql] = (static_cast<u64>(d) << 32) | kFull;
        }
        if (lane == 0u && of < net.words) {
          saved_near[of] = cur[w];
          saved_far[of] = far[w];
        }
      }
      paused = true;
      break;
    }
    const u32 nxt_off = near0_off + ((rounds & 1u) ? 0u : M * 4u), far_off = near0_off + M * 8u;
    bool any = false;

    // Relaxes `take` <= 32 pending vertices, one per thread.
    const auto relax = [&](u32 slot, u32 v, uint2 row, u32 take) {
      u32 d = dev::kInfBits, so = 0u, tile = kFull;
      if (lane < take) {
        d = shared_load<kCluster>(L_at + slot * 4u, true);  // neighbours may be lowering it
        so = slot - v;
        tile = gtile[slot >> 5];
        if (kCount) {
          cnt[0] += 1u;
          cnt[1] += row.y;
          cnt[2] += 1u;
        }
      }
      const EdgeList list_of(row, take);
      for (u32 base = 0; base < list_of.total; base += 32u * kSteps) {
        uint4 rec[kSteps];
        u32 from[kSteps];
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) {
          bool live;
          const u32 at = list_of.edge(base + k * 32u, from[k], live);
          rec[k] = make_uint4(0u, 0u, 0u, kFull);
          if (live) rec[k] = __ldg(p.g.csr + at);
        }
        // candidates and their vertices' places, then the distances there,
        // then the improvements
        u32 cand[kSteps], at[kSteps], to[kSteps], cur[kSteps];
        bool here[kSteps];
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) {
          const int i = static_cast<int>(from[k]);
          const u32 sd = __shfl_sync(kFull, d, i), ss = __shfl_sync(kFull, so, i), st = __shfl_sync(kFull, tile, i);
          cand[k] = __float_as_uint(__fadd_rn(__uint_as_float(sd), __uint_as_float(rec[k].y)));
          // own tile: in this block, at the vertex's own offset
          to[k] = rec[k].x + ss;
          at[k] = L_at + to[k] * 4u;
          here[k] = true;
          if (!(kWhole && rec[k].w == st)) {
            Endpoint e{0u, 0u};
            if (rec[k].w != kFull) e = endpoint(rec[k]);
            here[k] = e.at == 0u;
            at[k] = e.at == 0u ? L_at : e.at;
            to[k] = e.slot;
            cand[k] = e.at == 0u ? kFull : cand[k];
          }
          if (kCount) cnt[3] += cand[k] != kFull;
        }
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) cur[k] = shared_load<kCluster>(at[k], here[k]);
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) {
          // The minimum needs no answer: whoever lowers a distance below what
          // it read marks the vertex, pending in the next round or far, and
          // marking twice is harmless.
          if (cand[k] < cur[k]) {
            shared_min<kCluster>(at[k], cand[k], here[k]);
            const bool near = cand[k] < tau;
            any |= near;
            shared_or<kCluster>(at[k] - to[k] * 4u + (near ? nxt_off : far_off) + (to[k] >> 5) * 4u,
                                __funnelshift_l(0u, 1u, to[k]), here[k]);
            if (kCount) {
              cnt[5] += 1u;
              cnt[6] += 1u;
            }
          }
        }
      }
    };

    // This block's pending vertices, listed and relaxed in passes of at most
    // list_cap: each warp lists one word of every group of `warps` words, a
    // different one for neighbouring lanes (bank of each word its own), and
    // the list is cut into equal shares for the warps.
    for (;; ++pass) {
      for (u32 base = 0; base < M; base += warps * 32u) {
        const u32 w = base + lane * warps + (warp + lane) % warps;
        u32 bits = w < M ? cur[w] : 0u;
        u32 n = static_cast<u32>(__popc(bits)), at = n;
        for (u32 o = 1; o < 32u; o <<= 1) {
          const u32 y = __shfl_up_sync(kFull, at, o);
          if (lane >= o) at += y;
        }
        const u32 total = __shfl_sync(kFull, at, 31);
        if (total == 0u) continue;
        u32 first = 0u;
        if (lane == 31u) {
          first = atomicAdd(&s.listed[pass & 1u], total);
          if (first + total > list_cap) atomicMin(&s.cut[pass & 1u], first);
        }
        first = __shfl_sync(kFull, first, 31);
        if (first + total > list_cap) continue;  // the words keep their bits for the next pass
        at += first - n;
        if (bits != 0u) cur[w] = 0u;
        for (; bits != 0u; bits &= bits - 1u) {
          list[at++] = static_cast<unsigned short>((w << 5) + static_cast<u32>(__ffs(bits)) - 1u);
        }
      }
      __syncthreads();
      const u32 cut = s.cut[pass & 1u], n = min(s.listed[pass & 1u], cut);
      if (tid == 0u) {  // the next pass's; its readers of the pass before passed the barrier above
        s.listed[(pass + 1u) & 1u] = 0u;
        s.cut[(pass + 1u) & 1u] = kFull;
      }
      // shares of 8, 16 or 32 vertices
      const u32 share = n > 16u * warps ? 32u : (n > 8u * warps ? 16u : 8u);
      // (the next share's rows are read while one share is relaxed)
      u32 i = warp * share, slot = 0u, v = 0u;
      uint2 row = make_uint2(0u, 0u);
      const auto fetch = [&](u32 at) {
        row = make_uint2(0u, 0u);
        if (lane < share && at + lane < n) {
          slot = list[at + lane];
          v = gbase[slot >> 5] + (slot & 31u);
          row = __ldg(p.g.csr_row + v);
        }
      };
      if (i < n) fetch(i);
      for (; i < n; i += warps * share) {
        const u32 this_slot = slot, this_v = v;
        const uint2 this_row = row;
        if (i + warps * share < n) fetch(i + warps * share);
        relax(this_slot, this_v, this_row, min(share, n - i));
      }
      if (cut == kFull) break;
      __syncthreads();
    }
    ++pass;
    if (kCount) {
      for (int i = 0; i < 7; ++i) {
        total_cnt[i] += cnt[i];
        cnt[i] = 0u;
      }
    }
    if (__any_sync(kFull, any) && lane < ctas) remote_store(map_rank(shared_address(&s.any[rounds % 3u]), lane), 1u);
    if ((rounds & 255u) == 0u && rank == 0u && warp == 0u) {
      // one thread's clock decides for the whole cluster: blocks that left at
      // different rounds would wait for, or read, blocks that are gone
      const bool over = lane == 0u && dev::global_ns() - t0 > p.budget_ns;
      if (__shfl_sync(kFull, over, 0) && lane < ctas) remote_store(map_rank(shared_address(&s.stop), lane), 1u);
    }
    cluster_sync(ctas);
    const bool more = s.any[rounds % 3u] != 0u;
    if (s.stop != 0u) {
      if (tid == 0u && rank == 0u) atomicExch(&p.run->abort, 1u);
      break;
    }
    // the slot of the round after next; its last readers passed the barrier above
    if (tid == 0u) s.any[(rounds + 2u) % 3u] = 0u;
    if (more) continue;

    // --- split: no vertex is pending, the threshold rises ---------------------
    // A far vertex below the threshold was pending when it got there: dropped.
    u32 least = dev::kInfBits;
    for (u32 w = tid; w < M; w += blockDim.x) {
      u32 f = far[w], keep = f;
      for (; f != 0u; f &= f - 1u) {
        const u32 k = static_cast<u32>(__ffs(f)) - 1u;
        const u32 x = L[w * 32u + k];
        if (x < tau) {
          keep &= ~(1u << k);
        } else {
          least = min(least, x);
        }
      }
      far[w] = keep;
    }
    least = __reduce_min_sync(kFull, least);
    if (lane == 0u) s.scan[warp] = least;
    __syncthreads();
    if (warp == 0u) {
      least = __reduce_min_sync(kFull, lane < warps ? s.scan[lane] : dev::kInfBits);
      if (lane < ctas) remote_store(map_rank(shared_address(&s.fmin[splits & 1u][rank]), lane), least);
    }
    cluster_sync(ctas);
    least = dev::kInfBits;
    for (u32 i = 0; i < ctas; ++i) least = min(least, s.fmin[splits & 1u][i]);
    if (least >= dev::kInfBits) break;  // nothing far: converged
    ++splits;
    if (p.deltas == nullptr) delta = grown_step(delta, splits);
    const u32 stepped = __float_as_uint(__fadd_rn(__uint_as_float(least), __uint_as_float(delta)));
    tau = max(stepped, least + 1u);  // at least the next float above the smallest far distance
    for (u32 w = tid; w < M; w += blockDim.x) {
      u32 f = far[w], move = 0u;
      const u32 all = f;
      for (; f != 0u; f &= f - 1u) {
        const u32 k = static_cast<u32>(__ffs(f)) - 1u;
        if (L[w * 32u + k] < tau) move |= 1u << k;
      }
      if (move != 0u) {
        nxt[w] |= move;  // empty but for this split's moves
        far[w] = all & ~move;
      }
    }
    cluster_sync(ctas);
  }
  if (!paused) ++rounds;  // rounds run

  // --- result: distances and predecessors -------------------------------------
  // After the last barrier no block changes its distances.  A warp takes a
  // word's in-edges as one list; the tight ones (about one per vertex) lower
  // the vertex's predecessor in shared memory, where the list was.
  __syncthreads();
  volatile u32* const best = reinterpret_cast<u32*>(list) + warp * 32u;
  for (u32 w = paused ? M : warp; w < M; w += warps) {
    const u32 d = L[w * 32u + lane];
    const bool act = d < dev::kInfBits;
    if (!__any_sync(kFull, act)) continue;
    const u32 v = gbase[w] + lane, tile = gtile[w], so = w * 32u - gbase[w];
    uint2 col = make_uint2(0u, 0u);
    if (act) {
      col.x = __ldg(p.g.csc_off + v);
      col.y = __ldg(p.g.csc_off + v + 1u) - col.x;
    }
    best[lane] = kFull;
    __syncwarp();
    const EdgeList list_of(col, 32u);
    for (u32 base = 0; base < list_of.total; base += 32u * kSteps) {
      uint4 rec[kSteps];
      u32 from[kSteps];
#pragma unroll
      for (u32 k = 0; k < kSteps; ++k) {
        bool live;
        const u32 at = list_of.edge(base + k * 32u, from[k], live);
        rec[k] = make_uint4(0u, 0u, 0u, kFull);
        if (live) rec[k] = __ldg(p.g.csc + at);
      }
      u32 at[kSteps], x[kSteps];
      bool here[kSteps];
#pragma unroll
      for (u32 k = 0; k < kSteps; ++k) {
        at[k] = L_at + (rec[k].x + so) * 4u;
        here[k] = true;
        if (!(kWhole && rec[k].w == tile)) {
          Endpoint e{0u, 0u};
          if (rec[k].w != kFull) e = endpoint(rec[k]);
          here[k] = e.at == 0u;
          at[k] = e.at == 0u ? L_at : e.at;
          if (e.at == 0u) rec[k].y = kFull;  // NaN: not an admitted edge
        }
      }
#pragma unroll
      for (u32 k = 0; k < kSteps; ++k) x[k] = shared_load<kCluster>(at[k], here[k]);
#pragma unroll
      for (u32 k = 0; k < kSteps; ++k) {
        const u32 sd = __shfl_sync(kFull, d, static_cast<int>(from[k]));
        // an unreached endpoint sums to infinity, never to the distance
        if (__float_as_uint(__fadd_rn(__uint_as_float(x[k]), __uint_as_float(rec[k].y))) == sd) {
          shared_min<false>(shared_address(const_cast<u32*>(best + from[k])), rec[k].z, true);
        }
      }
    }
    __syncwarp();
    u32 eid = best[lane];
    __syncwarp();
    if (act) {
      if (d == 0u) {  // a source of the lane holds (0, 0)
        u32 lo = src0, hi = src1;
        while (lo < hi) {
          const u32 mid = (lo + hi) >> 1;
          if (B.src[mid] < v) lo = mid + 1u; else hi = mid;
        }
        if (lo < src1 && B.src[lo] == v) eid = 0u;
      }
      const u32 cv = v - B.tiles[tile].y;
      B.dist[0][(static_cast<u64>(cv) << B.shift) + ql] = (static_cast<u64>(d) << 32) | eid;
    }
  }
  if (tid == 0u && rank == 0u) {
    atomicMax(&C.rounds, rounds);
    atomicMax(reinterpret_cast<unsigned long long*>(&p.run->work[7]), static_cast<unsigned long long>(rounds));
    if (kPolled) {
      progress[blockIdx.x / ctas] = SearchProgress{rounds, tau, delta, splits, 0u, 0u, paused ? 0u : 1u, 0u};
      if (paused) atomicExch(&p.run->open, 1u);
    }
  }
  if (kCount) {
    for (int i = 0; i < 7; ++i) {
      u64 x = total_cnt[i];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
      if (lane == 0u && x) atomicAdd(reinterpret_cast<unsigned long long*>(&p.run->work[i]), x);
    }
  }
  cluster_sync(ctas);  // neighbours may still read this block's distances
}

// ---------------------------------------------------------------------------
// Whole-graph lanes: a team of blocks per lane, distances in global memory.
//
// A lane over the whole graph needs no tile table (compact index = vertex) but
// no cluster holds it.  Its 32-bit distances and bitmaps are 4.4 bytes a
// vertex, so with a few lanes in progress most random reads of a relaxation
// stay in the L2 (the grid-wide frontier relaxes all lanes of a batch at once,
// and its label rows of 8 bytes a lane come from DRAM).  The rounds are the
// cluster searches', with a barrier over the team's blocks.  The label rows
// are written and the predecessors found for all lanes of a batch together.
// B200, relaxation launches before and after: 32 lanes of 4.2M vertices 63.0
// -> 22.8 ms (20.1 of it the searches, 110 G edges/s, 2.6 TB/s of DRAM; 2.5
// the predecessors), 64 lanes of 16.8M vertices 567 -> 205 ms, one lane of
// 2.1M vertices 4.1 -> 2.9 ms.
// ---------------------------------------------------------------------------

// Scratch of a lane, in the batch's second label slot (8 bytes a vertex and
// lane): distances, two pending bitmaps, the far bitmap.
struct LaneScratch {
  u32 *L, *near0, *near1, *far;
};
__device__ __forceinline__ LaneScratch lane_scratch(const DBatch& B, u32 V, u32 ql) {
  LaneScratch s;
  s.L = reinterpret_cast<u32*>(B.dist[1] + static_cast<u64>(V) * ql);
  s.near0 = s.L + V;
  s.near1 = s.near0 + ((V + 31u) >> 5);
  s.far = s.near1 + ((V + 31u) >> 5);
  return s;
}

constexpr u32 kTeamList = 4096u;  // pending vertices of a block's pass

template <bool kCount, bool kPolled>
__global__ void __launch_bounds__(1024, 1)
    team_kernel(LaunchParams p, const ResidentNet* nets, u32 net_count, u32 teams, TeamState* states,
                SearchProgress* progress, u32 chunk) {
  __shared__ u32 s_list[kTeamList];
  __shared__ u32 s_listed[2], s_cut[2], s_min[32];
  const u32 per = gridDim.x / teams, team = blockIdx.x / per, rank = blockIdx.x - team * per;
  if (team >= teams) return;
  TeamState& S = states[team];
  const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
  const u32 V = p.g.V, words = (V + 31u) >> 5;
  const u64 t0 = p.run->started;  // the budget is the relaxation's, however long the search was queued
  if (tid < 2u) {
    s_listed[tid] = 0u;
    s_cut[tid] = kFull;
  }
  u32 r = 0u, splits = 0u, pass = 0u;  // rounds and splits of the team so far: its flags rotate over them
  u64 cnt[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  const auto barrier = [&]() {
    if (dev::grid_barrier(&S.sync, per, kBarrierTimeoutNs)) return true;
    if (tid == 0u) atomicExch(&p.run->abort, 1u);
    return false;
  };
  SearchProgress was{};  // written at the end of an earlier launch
  if (kPolled) was = progress[team];
  u32 turn = was.turns, ran = 0u;
  bool paused = false;
  for (u32 n = team + turn * teams; n < net_count && !paused; n += teams, ++turn) {
    const u32 b = nets[n].batch, ql = nets[n].lane;
    if (engine_of(p, b) != BFX_ENGINE_FRONTIER_PUSH) continue;
    const DBatch& B = p.batches[b];
    DCtl& C = p.ctl[b];
    const LaneScratch m = lane_scratch(B, V, ql);
    const u64 at = static_cast<u64>(rank) * blockDim.x + tid, stride = static_cast<u64>(per) * blockDim.x;
    const bool resumed = kPolled && was.begun != 0u && turn == was.turns;
    if (!resumed) {
      for (u64 i = at; i < V; i += stride) m.L[i] = dev::kInfBits;
      for (u64 i = at; i < 3ull * words; i += stride) m.near0[i] = 0u;
      if (!barrier()) return;
      if (rank == 0u) {
        for (u32 i = B.src_off[ql] + tid; i < B.src_off[ql + 1u]; i += blockDim.x) {
          const u32 v = B.src[i];
          m.L[v] = 0u;
          dev::red_or(m.near0 + (v >> 5), 1u << (v & 31u));
        }
      }
      if (!barrier()) return;
    }
    u32 delta = p.deltas ? p.deltas[b] : p.auto_step;
    u32 tau = delta, rounds = 0u, splits0 = splits;
    if (resumed) {
      delta = was.delta;
      tau = was.tau;
      rounds = was.rounds;
      splits0 -= was.splits;
    }
    for (;; ++rounds, ++ran) {
      if (kPolled && ran == chunk) {  // after a barrier: the lane's scratch is whole
        if (rank == 0u && tid == 0u) {
          progress[team] = SearchProgress{rounds, tau, delta, splits - splits0, 1u, turn, 0u, 0u};
          atomicExch(&p.run->open, 1u);
        }
        paused = true;
        break;
      }
      u32* const cur = (rounds & 1u) ? m.near1 : m.near0;
      u32* const nxt = (rounds & 1u) ? m.near0 : m.near1;
      bool any = false;
      const auto relax = [&](u32 v, uint2 row, u32 take) {
        u32 d = dev::kInfBits;
        if (lane < take) {
          d = dev::ld_cg(m.L + v);
          if (kCount) {
            cnt[0] += 1u;
            cnt[1] += row.y;
            cnt[2] += 1u;
            cnt[3] += row.y;
          }
        }
        const EdgeList edges(row, take);
        for (u32 base = 0; base < edges.total; base += 32u * kSteps) {
          uint2 rec[kSteps];
          u32 cand[kSteps], x[kSteps];
#pragma unroll
          for (u32 k = 0; k < kSteps; ++k) {
            u32 from;
            bool live;
            const u32 e = edges.edge(base + k * 32u, from, live);
            rec[k] = make_uint2(0u, kFull);  // NaN weight: improves nothing
            if (live) rec[k] = __ldg(reinterpret_cast<const uint2*>(p.g.csr + e));
            cand[k] = __shfl_sync(kFull, d, static_cast<int>(from));
          }
#pragma unroll
          for (u32 k = 0; k < kSteps; ++k) {
            cand[k] = __float_as_uint(__fadd_rn(__uint_as_float(cand[k]), __uint_as_float(rec[k].y)));
            x[k] = rec[k].y != kFull ? dev::ld_cg(m.L + rec[k].x) : 0u;
          }
#pragma unroll
          for (u32 k = 0; k < kSteps; ++k) {
            if (cand[k] < x[k]) {
              dev::red_min_u32(m.L + rec[k].x, cand[k]);
              const bool near = cand[k] < tau;
              any |= near;
              dev::red_or((near ? nxt : m.far) + (rec[k].x >> 5), 1u << (rec[k].x & 31u));
              if (kCount) {
                cnt[5] += 1u;
                cnt[6] += 1u;
              }
            }
          }
        }
      };
      // The block's words: groups of 32 dealt over the team's blocks.
      for (;; ++pass) {
        for (u32 g = rank + warp * per; g * 32u < words; g += warps * per) {
          const u32 w = g * 32u + lane;
          u32 bits = w < words ? dev::ld_cg(cur + w) : 0u;
          const u32 c = static_cast<u32>(__popc(bits));
          u32 to = c;
          for (u32 o = 1; o < 32u; o <<= 1) {
            const u32 y = __shfl_up_sync(kFull, to, o);
            if (lane >= o) to += y;
          }
          const u32 total = __shfl_sync(kFull, to, 31);
          if (total == 0u) continue;
          u32 first = 0u;
          if (lane == 31u) {
            first = atomicAdd(&s_listed[pass & 1u], total);
            if (first + total > kTeamList) atomicMin(&s_cut[pass & 1u], first);
          }
          first = __shfl_sync(kFull, first, 31);
          if (first + total > kTeamList) continue;  // the words keep their bits for the next pass
          to += first - c;
          if (bits != 0u) cur[w] = 0u;
          for (; bits != 0u; bits &= bits - 1u) s_list[to++] = w * 32u + static_cast<u32>(__ffs(bits)) - 1u;
        }
        __syncthreads();
        const u32 cut = s_cut[pass & 1u], listed = min(s_listed[pass & 1u], cut);
        if (tid == 0u) {  // the next pass's; its readers of the pass before passed the barrier above
          s_listed[(pass + 1u) & 1u] = 0u;
          s_cut[(pass + 1u) & 1u] = kFull;
        }
        const u32 share = listed > 16u * warps ? 32u : (listed > 8u * warps ? 16u : 8u);
        u32 i = warp * share, v = 0u;
        uint2 row = make_uint2(0u, 0u);
        const auto fetch = [&](u32 from) {
          row = make_uint2(0u, 0u);
          if (lane < share && from + lane < listed) {
            v = s_list[from + lane];
            row = __ldg(p.g.csr_row + v);
          }
        };
        if (i < listed) fetch(i);
        for (; i < listed; i += warps * share) {
          const u32 this_v = v;
          const uint2 this_row = row;
          if (i + warps * share < listed) fetch(i + warps * share);
          relax(this_v, this_row, min(share, listed - i));
        }
        if (cut == kFull) break;
        __syncthreads();
      }
      ++pass;
      if (__syncthreads_or(any) && tid == 0u) atomicExch(&S.any[r % 3u], 1u);
      if ((r & 63u) == 0u && rank == 0u && tid == 0u && dev::global_ns() - t0 > p.budget_ns) {
        atomicExch(&S.sync.abort, 1u);
      }
      if (!barrier()) return;
      const bool more = dev::ld_cg(&S.any[r % 3u]) != 0u;
      // the slot of the round after next; its last readers passed the barrier above
      if (rank == 0u && tid == 0u) S.any[(r + 2u) % 3u] = 0u;
      ++r;
      if (more) continue;

      // --- split: far vertices below the next threshold become pending ---------
      // The first scan takes tau + delta; where that moves none, the second
      // takes the smallest far distance + delta.
      bool converged = false;
      const u32 old = tau;
      for (u32 scan = 0;; ++scan) {
        if (scan == 0u) tau = __float_as_uint(__fadd_rn(__uint_as_float(tau), __uint_as_float(delta)));
        u32 least = dev::kInfBits;
        bool moved = false;
        for (u32 g = rank + warp * per; g * 32u < words; g += warps * per) {
          const u32 w = g * 32u + lane;
          const u32 f = w < words ? dev::ld_cg(m.far + w) : 0u;
          u32 keep = f, move = 0u;
          // eight words at a time, a word's 32 distances one read
          for (u32 todo = __ballot_sync(kFull, f != 0u); todo != 0u;) {
            u32 from[8], x[8];
#pragma unroll
            for (u32 k = 0; k < 8u; ++k) {
              from[k] = todo != 0u ? static_cast<u32>(__ffs(todo)) - 1u : 32u;
              todo &= todo - 1u;
            }
#pragma unroll
            for (u32 k = 0; k < 8u; ++k) {
              const u32 y = from[k] < 32u ? (g * 32u + from[k]) * 32u + lane : V;
              x[k] = y < V ? dev::ld_cg(m.L + y) : dev::kInfBits;
            }
#pragma unroll
            for (u32 k = 0; k < 8u; ++k) {
              if (from[k] == 32u) continue;  // warp-uniform
              const bool mine = ((__shfl_sync(kFull, f, static_cast<int>(from[k])) >> lane) & 1u) != 0u;
              // below the old threshold: was pending when it got there
              const u32 stay = __ballot_sync(kFull, mine && x[k] >= tau);
              const u32 go = __ballot_sync(kFull, mine && x[k] < tau && x[k] >= old);
              if (mine && x[k] >= tau) least = min(least, x[k]);
              if (lane == from[k]) {
                keep = stay;
                move = go;
              }
            }
          }
          if (keep != f) m.far[w] = keep;
          if (move != 0u) {
            nxt[w] = move;  // empty before the split
            moved = true;
          }
        }
        least = __reduce_min_sync(kFull, least);
        if (lane == 0u) s_min[warp] = least;
        const bool block_moved = __syncthreads_or(moved) != 0;
        if (warp == 0u) {
          least = __reduce_min_sync(kFull, lane < warps ? s_min[lane] : dev::kInfBits);
          if (lane == 0u) {
            atomicMax(&S.least[splits % 3u], ~least);
            if (block_moved) atomicExch(&S.moved[splits % 3u], 1u);
          }
        }
        if (!barrier()) return;
        least = ~dev::ld_cg(&S.least[splits % 3u]);
        const bool go = dev::ld_cg(&S.moved[splits % 3u]) != 0u;
        if (rank == 0u && tid == 0u) S.least[(splits + 2u) % 3u] = S.moved[(splits + 2u) % 3u] = 0u;
        ++splits;
        if (p.deltas == nullptr) delta = grown_step(delta, splits - splits0);
        if (go) break;
        if (least >= dev::kInfBits) {
          converged = true;
          break;
        }
        const u32 stepped = __float_as_uint(__fadd_rn(__uint_as_float(least), __uint_as_float(delta)));
        tau = max(stepped, least + 1u);
      }
      if (converged) break;
    }
    const u32 run_rounds = paused ? rounds : rounds + 1u;
    if (!paused) ++ran;
    if (tid == 0u && rank == 0u) {
      atomicMax(&C.rounds, run_rounds);
      atomicMax(reinterpret_cast<unsigned long long*>(&p.run->work[7]), static_cast<unsigned long long>(run_rounds));
    }
  }
  if (kPolled && !paused && turn != was.turns && rank == 0u && tid == 0u) {
    progress[team] = SearchProgress{0u, 0u, 0u, 0u, 0u, turn, 1u, 0u};
  }
  if (kCount) {
    for (int i = 0; i < 7; ++i) {
      u64 x = cnt[i];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
      if (lane == 0u && x) atomicAdd(reinterpret_cast<unsigned long long*>(&p.run->work[i]), x);
    }
  }
}

// Label rows of a whole-graph batch from its lanes' distances, the predecessor
// word unreached: a warp turns 32 vertices x W lanes through shared memory.
__global__ void __launch_bounds__(256) team_rows_kernel(LaunchParams p, u32 b) {
  __shared__ u32 s_rows[8][32 * 33];
  if (engine_of(p, b) != BFX_ENGINE_FRONTIER_PUSH) return;
  const DBatch& B = p.batches[b];
  const u32 V = p.g.V, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  u32* const rows = s_rows[warp];
  for (u32 v0 = (blockIdx.x * 8u + warp) * 32u; v0 < V; v0 += gridDim.x * 256u) {
    for (u32 l = 0; l < B.W; ++l) {
      u32 x = dev::kInfBits;
      if (((B.valid >> l) & 1u) && v0 + lane < V) x = lane_scratch(B, V, l).L[v0 + lane];
      rows[lane * 33u + l] = x;
    }
    __syncwarp();
    const u32 n = min(V - v0, 32u) << B.shift;
    u64* const out = B.dist[0] + (static_cast<u64>(v0) << B.shift);
    for (u32 k = lane; k < n; k += 32u) {
      out[k] = (static_cast<u64>(rows[(k >> B.shift) * 33u + (k & (B.W - 1u))]) << 32) | kFull;
    }
    __syncwarp();
  }
}

// Predecessors of a whole-graph batch, in place (distances are the high words,
// which no thread writes): per (vertex, lane) the smallest stable edge id
// among the in-edges that give its distance.
__global__ void __launch_bounds__(256) team_predecessor_kernel(LaunchParams p, u32 b) {
  __shared__ u32 s_best[8][32];
  if (engine_of(p, b) != BFX_ENGINE_FRONTIER_PUSH) return;
  const DBatch& B = p.batches[b];
  const u32 V = p.g.V, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const auto source = [&](u32 v, u32 ql) {
    u32 lo = B.src_off[ql], hi = B.src_off[ql + 1u];
    const u32 end = hi;
    while (lo < hi) {
      const u32 mid = (lo + hi) >> 1;
      if (B.src[mid] < v) lo = mid + 1u; else hi = mid;
    }
    return lo < end && B.src[lo] == v;
  };
  u32* const words = reinterpret_cast<u32*>(B.dist[0]);  // {predecessor, distance} pairs
  if (B.W == 1u) {
    // 32 vertices' in-edges as one list
    volatile u32* const best = s_best[warp];
    for (u32 v0 = (blockIdx.x * 8u + warp) * 32u; v0 < V; v0 += gridDim.x * 256u) {
      const u32 v = v0 + lane;
      const u32 d = v < V ? words[2ull * v + 1u] : dev::kInfBits;
      uint2 col = make_uint2(0u, 0u);
      if (d < dev::kInfBits) {
        col.x = __ldg(p.g.csc_off + v);
        col.y = __ldg(p.g.csc_off + v + 1u) - col.x;
      }
      best[lane] = kFull;
      __syncwarp();
      const EdgeList edges(col, 32u);
      for (u32 base = 0; base < edges.total; base += 32u * kSteps) {
        uint4 rec[kSteps];
        u32 from[kSteps], x[kSteps];
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) {
          bool live;
          const u32 e = edges.edge(base + k * 32u, from[k], live);
          rec[k] = make_uint4(0u, kFull, kFull, 0u);
          if (live) rec[k] = __ldg(p.g.csc + e);
        }
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) x[k] = rec[k].y != kFull ? words[2ull * rec[k].x + 1u] : dev::kInfBits;
#pragma unroll
        for (u32 k = 0; k < kSteps; ++k) {
          const u32 dv = __shfl_sync(kFull, d, static_cast<int>(from[k]));
          if (__float_as_uint(__fadd_rn(__uint_as_float(x[k]), __uint_as_float(rec[k].y))) == dv) {
            shared_min<false>(shared_address(const_cast<u32*>(best + from[k])), rec[k].z, true);
          }
        }
      }
      __syncwarp();
      if (d < dev::kInfBits) words[2ull * v] = d == 0u && source(v, 0u) ? 0u : best[lane];
      __syncwarp();
    }
    return;
  }
  // W threads per vertex, one per lane; they read its in-edge records together
  // and then each its own distances, four in-edges in flight.
  const u32 W = B.W, ql = lane & (W - 1u), vpw = 32u >> B.shift;
  for (u32 v0 = (blockIdx.x * 8u + warp) * vpw; v0 < V; v0 += gridDim.x * 8u * vpw) {
    const u32 v = v0 + (lane >> B.shift);
    const u64 at = (static_cast<u64>(v) << B.shift) + ql;
    u32 d = dev::kInfBits, cb = 0u, count = 0u;
    if (v < V) {
      d = words[2u * at + 1u];
      cb = __ldg(p.g.csc_off + v);
      count = __ldg(p.g.csc_off + v + 1u) - cb;
    }
    u32 eid = kFull;
    const u32 most = __reduce_max_sync(kFull, count);
    for (u32 e = 0; e < most; e += W) {
      uint4 mine = make_uint4(0u, kFull, kFull, 0u);  // NaN weight: gives no distance
      if (e + ql < count) mine = __ldg(p.g.csc + cb + e + ql);
      const u32 here = min(W, most - e);
      for (u32 k = 0; k < here; k += 4u) {
        u32 u[4], w[4], id[4], x[4];
#pragma unroll
        for (u32 j = 0; j < 4u; ++j) {
          const int from = static_cast<int>(min(k + j, W - 1u));
          u[j] = __shfl_sync(kFull, mine.x, from, static_cast<int>(W));
          w[j] = __shfl_sync(kFull, mine.y, from, static_cast<int>(W));
          id[j] = __shfl_sync(kFull, mine.z, from, static_cast<int>(W));
        }
#pragma unroll
        for (u32 j = 0; j < 4u; ++j) {
          x[j] = w[j] != kFull ? words[2u * ((static_cast<u64>(u[j]) << B.shift) + ql) + 1u] : dev::kInfBits;
        }
#pragma unroll
        for (u32 j = 0; j < 4u; ++j) {
          if (__float_as_uint(__fadd_rn(__uint_as_float(x[j]), __uint_as_float(w[j]))) == d) eid = min(eid, id[j]);
        }
      }
    }
    if (d < dev::kInfBits) words[2u * at] = d == 0u && source(v, ql) ? 0u : eid;
  }
}

template <bool kCount>
const void* team_entry(bool polled) {
  return polled ? reinterpret_cast<const void*>(team_kernel<kCount, true>)
                : reinterpret_cast<const void*>(team_kernel<kCount, false>);
}

// (one block: a tile is contiguous in any case)
template <bool kCount, bool kPolled>
const void* resident_entry(bool cluster, bool whole) {
  if (!cluster) return reinterpret_cast<const void*>(resident_kernel<kCount, false, true, kPolled>);
  return whole ? reinterpret_cast<const void*>(resident_kernel<kCount, true, true, kPolled>)
               : reinterpret_cast<const void*>(resident_kernel<kCount, true, false, kPolled>);
}

const void* resident_entry(bool count, bool polled, bool cluster, bool whole) {
  if (count) return polled ? resident_entry<true, true>(cluster, whole) : resident_entry<true, false>(cluster, whole);
  return polled ? resident_entry<false, true>(cluster, whole) : resident_entry<false, false>(cluster, whole);
}

}  // namespace

namespace {

// Dynamic shared memory of one block.
size_t block_bytes(u32 words, u32 tiles, u32 ctas, u32 threads, u32 tile_count, u32 run) {
  const size_t m = block_words(words, ctas, run);
  return (size_t{tile_count} + 31) / 32 * 8 + m * 32 * 4 + (m * 5 + (m & 1)) * 4 + size_t{tiles} * 8 +
         size_t{threads} * kListPer * 2;
}

// Smallest shape that holds the net (kShapeCount: none).
u32 smallest_shape(const bfx_resident_graph* graph, const ResidentNet& n, u32 run, u32 shapes) {
  for (u32 k = 0; k < shapes; ++k) {
    // a list entry is a 16-bit slot
    if (block_words(n.words, kShapes[k].ctas, run) <= 2048u &&
        block_bytes(n.words, n.tiles, kShapes[k].ctas, kShapes[k].threads, graph->g.T, run) <=
            kShapes[k].bytes) {
      return k;
    }
  }
  return kShapeCount;
}

void set_attributes(const void* kernel) {
  BFX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBlockBytes)));
  BFX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

}  // namespace

// The block configurations of the current device: all, or those up to the
// largest cluster that it can hold at once.  Sets the kernels' attributes,
// which hold for the device, so that launches need not.
u32 resident_shapes() {
  for (int k = 0; k < 4; ++k) {
    for (int kind = 0; kind < 3; ++kind) {
      set_attributes(resident_entry((k & 1) != 0, (k & 2) != 0, kind != 0, kind == 2));
    }
  }
  const void* kernel = resident_entry(false, false, true, true);
  u32 shapes = 1u;
  for (; shapes < kShapeCount; ++shapes) {
    if (kShapes[shapes].ctas == 1u) continue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kShapes[shapes].ctas);
    cfg.blockDim = dim3(kShapes[shapes].threads);
    cfg.dynamicSmemBytes = kShapes[shapes].bytes;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kShapes[shapes].ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    const cudaError_t err = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (err != cudaSuccess) cudaGetLastError();
    if (err != cudaSuccess || clusters < 1) break;
  }
  return shapes;
}

void resident_select(bfx_workspace* ws, const std::vector<u32>& full, std::vector<ResidentNet>& nets,
                     std::vector<ResidentNet>& whole, std::vector<u32>& fit) {
  const bfx_resident_graph* graph = ws->graph;
  const u32 run = graph->word_run, shapes = graph->resident_shapes;
  std::sort(nets.begin(), nets.end(), [](const ResidentNet& a, const ResidentNet& b) {
    return a.words != b.words ? a.words > b.words : (a.batch != b.batch ? a.batch < b.batch : a.lane < b.lane);
  });
  std::vector<ResidentNet> kept;
  kept.reserve(nets.size());
  whole.clear();
  for (const ResidentNet& n : nets) {
    if (smallest_shape(graph, n, run, shapes) != kShapeCount) {
      kept.push_back(n);
    } else if (full[n.batch] != 0u) {
      whole.push_back(n);
    } else {
      continue;
    }
    fit[n.batch] |= 1u << n.lane;
  }
  nets.swap(kept);
  // lanes of a batch in turn, batch by batch
  std::sort(whole.begin(), whole.end(), [](const ResidentNet& a, const ResidentNet& b) {
    return a.batch != b.batch ? a.batch < b.batch : a.lane < b.lane;
  });
}

namespace {

// Launches the whole-graph lanes' searches.
u32 launch_teams(bfx_workspace* ws, const LaunchParams& p, bool count, SearchProgress* progress, u32 chunk) {
  if (ws->whole.empty()) return 0;
  // Lanes at a time: as many as kTeamBytes of distances allow, in equal turns.
  // More teams hide one another's barriers and read latency, until their wave
  // fronts outgrow the L2.  Measured (ms): 32 lanes of 4.2M vertices (17 MB)
  // on 1 / 2 / 4 / 8 / 16 teams 51.5 / 33.8 / 25.9 / 22.8 / 22.4; 64 lanes of
  // 16.8M vertices (67 MB) on 1 / 2 / 4 / 6 / 8 / 16 teams 297 / 227 / 205 /
  // 231 / 223 / 259.
  u32 lanes = static_cast<u32>(ws->whole.size());
  const u64 lane_bytes = static_cast<u64>(p.g.V) * 4u;
  const u32 most = std::max(1u, std::min(kMaxTeams, static_cast<u32>(kTeamBytes / lane_bytes)));
  u32 teams = (lanes + most - 1u) / most;  // turns
  teams = (lanes + teams - 1u) / teams;
  const ResidentNet* d_whole = ws->d_whole;
  TeamState* states = ws->d_teams;
  BFX_CUDA(cudaMemsetAsync(states, 0, sizeof(TeamState) * kMaxTeams, ws->stream));
  LaunchParams params = p;
  void* args[] = {&params, &d_whole, &lanes, &teams, &states, &progress, &chunk};
  const void* kernel = count ? team_entry<true>(progress != nullptr) : team_entry<false>(progress != nullptr);
  BFX_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(static_cast<u32>(ws->sm_count) / teams * teams), dim3(1024), args,
                                       0, ws->stream));
  ws->last_kernels[1] = kernel;
  return 1;
}

// Label rows and predecessors of the whole-graph lanes.
u32 launch_team_labels(bfx_workspace* ws, const LaunchParams& p) {
  u32 launches = 0;
  u32 last = 0xFFFFFFFFu;
  for (const ResidentNet& n : ws->whole) {
    if (n.batch == last) continue;
    last = n.batch;
    team_rows_kernel<<<ws->sm_count * 6, 256, 0, ws->stream>>>(p, n.batch);
    BFX_CUDA(cudaGetLastError());
    team_predecessor_kernel<<<ws->sm_count * 8, 256, 0, ws->stream>>>(p, n.batch);
    BFX_CUDA(cudaGetLastError());
    launches += 2;
  }
  return launches;
}

// Launches the searches of the nets that have clusters of their own.
u32 launch_resident(bfx_workspace* ws, const LaunchParams& p, bool count, SearchProgress* progress, u32 chunk) {
  const std::vector<ResidentNet>& nets = ws->nets;
  if (nets.empty()) return 0;
  const u32 run = ws->graph->word_run;
  const u32 shapes = ws->graph->resident_shapes;
  // A net takes the smallest shape that holds it; where the nets together
  // leave SMs idle, every net takes a larger one, as far as it has words.
  std::vector<u32> smallest(nets.size()), shape(nets.size());
  for (size_t i = 0; i < nets.size(); ++i) smallest[i] = smallest_shape(ws->graph, nets[i], run, shapes);
  for (u32 up = 0; up < shapes; ++up) {
    std::vector<u32> next(nets.size());
    u64 threads = 0;
    for (size_t i = 0; i < nets.size(); ++i) {
      u32 k = smallest[i];
      while (k < std::min({smallest[i] + up, kSpreadShape, shapes - 1u}) &&
             nets[i].words >= kSpreadWords * kShapes[k].ctas) {
        ++k;
      }
      next[i] = k;
      threads += kShapes[k].ctas * kShapes[k].threads;
    }
    if (up > 0 && threads > 1024ull * static_cast<u64>(ws->sm_count)) break;
    shape.swap(next);
  }
  // one contiguous group of nets per shape: a larger shape holds what a smaller one does
  for (size_t i = nets.size(); i-- > 1;) shape[i - 1] = std::max(shape[i - 1], shape[i]);
  std::vector<std::pair<u32, std::pair<u32, u32>>> groups;  // shape, [first, last)
  for (size_t i = 0; i < nets.size(); ++i) {  // nets are sorted by size, so a shape's nets are contiguous
    if (groups.empty() || groups.back().first != shape[i]) {
      groups.push_back({shape[i], {static_cast<u32>(i), static_cast<u32>(i)}});
    }
    groups.back().second.second = static_cast<u32>(i) + 1u;
  }
  // The shapes run side by side on up to kLaunchStreams streams in turn,
  // largest first; ws->stream is the first of them.
  const size_t used = std::min<size_t>(groups.size(), kLaunchStreams);
  ws->resident_sides.reserve(kLaunchStreams);
  while (ws->resident_sides.size() + 1 < used) {
    SideStreams<CudaStreams>::Side side{};
    BFX_CUDA(cudaStreamCreateWithFlags(&side.stream, cudaStreamNonBlocking));
    const cudaError_t err = cudaEventCreateWithFlags(&side.done, cudaEventDisableTiming);
    if (err != cudaSuccess) cudaStreamDestroy(side.stream);
    BFX_CUDA(err);
    ws->resident_sides.push_back(side);
  }
  if (used > 1 && !ws->resident_fork) BFX_CUDA(cudaEventCreateWithFlags(&ws->resident_fork, cudaEventDisableTiming));
  SideStreams<CudaStreams> sides(ws->stream, ws->resident_fork, ws->resident_sides.data(), used - 1);
  u32 launches = 0;
  for (size_t i = 0; i < groups.size(); ++i) {
    const Shape& sh = kShapes[groups[i].first];
    const u32 first = groups[i].second.first, last = groups[i].second.second;
    const size_t on = i % kLaunchStreams;
    const cudaStream_t stream = on == 0 ? ws->stream : ws->resident_sides[on - 1].stream;
    size_t bytes = 0;
    for (u32 n = first; n < last; ++n) {
      bytes = std::max(bytes, block_bytes(nets[n].words, nets[n].tiles, sh.ctas, sh.threads, p.g.T, run));
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((last - first) * sh.ctas);
    cfg.blockDim = dim3(sh.threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = sh.ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = sh.ctas > 1u ? 1u : 0u;
    LaunchParams params = p;
    const ResidentNet* d_nets = ws->d_nets + first;
    u32 ctas = sh.ctas, run_shift = run;
    SearchProgress* net_progress = progress ? progress + first : nullptr;
    void* args[] = {&params, &d_nets, &ctas, &run_shift, &net_progress, &chunk};
    const void* kernel = resident_entry(count, progress != nullptr, sh.ctas > 1u, ws->graph->word_whole);
    BFX_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
    if (i == 0) ws->last_kernels[0] = kernel;
    ++launches;
  }
  sides.join();
  return launches;
}

}  // namespace

u32 launch_searches(bfx_workspace* ws, const LaunchParams& p, bool count) {
  u32 launches = launch_teams(ws, p, count, nullptr, 0u) + launch_team_labels(ws, p);
  launches += launch_resident(ws, p, count, nullptr, 0u);
  return launches;
}

// A chunk costs about 0.1 ms beside its rounds (host calls of up to eight
// streams, the net's tables and distances set up again): 40 nets of 67 rounds,
// 8 at a time, 1.76 ms a request on a B200, 0.93 in one launch, and 4.7 in the
// grid-wide rounds.  One graph launch per chunk costs more than it saves
// (2.2 ms: it is made anew for every prepared set).
u32 poll_searches(bfx_workspace* ws, const LaunchParams& p, bool count, bool clusters, u32 chunk,
                  std::chrono::steady_clock::time_point deadline) {
  const size_t bytes = (kMaxTeams + ws->nets.size()) * sizeof(SearchProgress);
  ws->progress.reserve(bytes, ws->graph->device);
  auto* const progress = static_cast<SearchProgress*>(ws->progress.ptr);
  BFX_CUDA(cudaMemsetAsync(progress, 0, bytes, ws->stream));
  ws->status_host.reserve(256);
  auto* const seen = static_cast<u32*>(ws->status_host.ptr);  // {open, abort}
  static_assert(offsetof(DRun, abort) == offsetof(DRun, open) + 4);
  u32 launches = 0;
  for (;;) {
    BFX_CUDA(cudaMemsetAsync(&p.run->open, 0, 4, ws->stream));
    launches += launch_teams(ws, p, count, progress, chunk);
    if (clusters) launches += launch_resident(ws, p, count, progress + kMaxTeams, chunk);
    BFX_CUDA(cudaMemcpyAsync(seen, &p.run->open, 8, cudaMemcpyDeviceToHost, ws->stream));
    BFX_CUDA(cudaStreamSynchronize(ws->stream));
    ++ws->last_host_checks;
    if (seen[0] == 0u || seen[1] != 0u) break;
    if (std::chrono::steady_clock::now() > deadline) {
      BFX_CUDA(cudaMemsetAsync(&p.run->abort, 1, 1, ws->stream));
      break;
    }
  }
  return launches + launch_team_labels(ws, p);
}

void resident_release(bfx_workspace* ws) {
  for (const auto& side : ws->resident_sides) {
    cudaStreamDestroy(side.stream);
    cudaEventDestroy(side.done);
  }
  if (ws->resident_fork) cudaEventDestroy(ws->resident_fork);
}

}  // namespace bfx
