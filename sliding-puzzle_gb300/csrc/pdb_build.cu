// GPU breadth-first construction of the additive pattern databases, layout
// conversions, and the batched heuristic kernel.
//
// The reference loads two 6-tile tables from files it does not ship
// (src/24puzzle_block_parallel_with_pdb.cu:164-230).  Their contents are
// defined here by the abstraction that reproduces the reference's golden
// node counts (benchmarks/pdb_expand_nodes.csv, all 50 rows):
//   * an abstract state is the pattern tiles' cells plus the connected region
//     of non-pattern cells that holds the blank (other tiles move for free
//     inside a region);
//   * one abstract move slides a pattern tile into a neighbouring cell of the
//     blank's region, cost 1;
//   * the goal is the pattern tiles on their goal cells with the blank in the
//     region of its home cell 0;
//   * a table entry is the distance to the goal, minimised over the blank's
//     regions (the reference's index holds no blank position).
// The search runs level by level over the abstract states themselves: a queue
// of (placement, region) entries, each appended once, whose slice [bounds[d],
// bounds[d + 1]) is level d.  The regions of a placement depend only on which
// cells are occupied, so a table over the C(n, k) subsets gives every cell's
// region number (at most 5), and one visited bit per region makes 64 MB of a
// 6-tile table's 181 M states: it stays in L2.  A placement's first visit
// writes its entry straight into the lookup layout.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sp_defs.h"
#include "sp_device.cuh"
#include "sp_kernels.h"

namespace sp {

namespace {

// n choose k for the subset numbers.
constexpr uint32_t choose(int n, int k) {
  uint64_t r = 1;
  for (int i = 0; i < k; ++i) r = r * (uint64_t)(n - i) / (uint64_t)(i + 1);
  return n < k ? 0u : (uint32_t)r;
}

template <int W>
struct Geo {
  static constexpr int N = W * W, K = W == 5 ? 6 : 5;
  static constexpr uint32_t kFull = (1u << N) - 1u;
  static constexpr int kLoBits = (N + 1) / 2;  // a cell mask in two halves, for its subset number
  static constexpr uint32_t kSubsets = choose(N, K);
  static constexpr uint32_t kSubsetWords = (kSubsets + 31) / 32;
  // cells of one column
  static constexpr uint32_t column(int c) {
    uint32_t m = 0;
    for (int r = 0; r < W; ++r) m |= 1u << (r * W + c);
    return m;
  }
  // weight of digit i of a placement's rank / of its lookup index
  static constexpr uint32_t rank_weight(int i) {
    uint32_t w = 1;
    for (int m = i + 1; m < K; ++m) w *= (uint32_t)(N - m);
    return w;
  }
  static constexpr uint32_t index_weight(int i) {
    uint32_t w = 1;
    for (int m = i + 1; m < K; ++m) w *= (uint32_t)N;
    return w;
  }
};

template <int W>
__host__ __device__ __forceinline__ uint32_t flood(uint32_t free_cells, uint32_t from) {
  using G = Geo<W>;
  uint32_t r = from, prev;
  do {
    prev = r;
    r = (r | ((r << 1) & ~G::column(0)) | ((r >> 1) & ~G::column(W - 1)) | (r << W) | (r >> W)) & free_cells;
  } while (r != prev);
  return r;
}

// Cells of placement `rank` (lexicographic rank of the k-permutation of
// cells, the byte order of the reference's table files): the digits by
// constant divisions, each then moved past the cells used before it, which
// are kept sorted.
template <int W>
__device__ __forceinline__ void unrank(uint32_t rank, int (&pos)[Geo<W>::K]) {
  using G = Geo<W>;
  int sorted[G::K];
#pragma unroll
  for (int i = G::K - 1; i >= 0; --i) {
    const uint32_t q = rank / (uint32_t)(G::N - i);
    pos[i] = (int)(rank - q * (uint32_t)(G::N - i));
    rank = q;
  }
#pragma unroll
  for (int i = 0; i < G::K; ++i) {
    int p = pos[i];
#pragma unroll
    for (int m = 0; m < i; ++m) p += p >= sorted[m];
    pos[i] = p;
    sorted[i] = p;
#pragma unroll
    for (int m = i; m > 0; --m) {
      const int lo = min(sorted[m - 1], sorted[m]), hi = max(sorted[m - 1], sorted[m]);
      sorted[m - 1] = lo;
      sorted[m] = hi;
    }
  }
}

template <int W>
__device__ __forceinline__ uint32_t lookup_index(const int (&pos)[Geo<W>::K]) {
  uint32_t x = 0;
#pragma unroll
  for (int j = 0; j < Geo<W>::K; ++j) x = x * (uint32_t)Geo<W>::N + (uint32_t)pos[j];
  return x;
}

// Per-build tables: the subset number of a k-cell mask is the sum of its low
// half's entry and its high half's (their colexicographic numbers; the high
// half's cells come after the k - popc(high) low ones), and per subset the
// region number of every free cell as three bit planes (regions in the order
// of their lowest cells), the number of regions in w.  `split`: a bit per
// subset with more than one region.
struct SubsetTables {
  uint16_t *lo;
  uint32_t *hi, *split;
  uint4 *regions;
};

template <int W>
__global__ void subset_kernel(SubsetTables S, unsigned long long *n_regions) {
  using G = Geo<W>;
  auto colex = [](uint32_t mask, int base, int first) -> uint32_t {  // i-th set bit p -> C(base + p, first + i)
    uint32_t r = 0;
    for (int i = first; mask; mask &= mask - 1u) {
      ++i;
      const int n = base + __ffs(mask) - 1;
      uint64_t c = 1;
      for (int q = 0; q < i; ++q) c = c * (uint64_t)(n - q) / (uint64_t)(q + 1);
      r += n < i ? 0u : (uint32_t)c;
    }
    return r;
  };
  const uint32_t mask = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t hi = mask >> G::kLoBits, lo = mask & ((1u << G::kLoBits) - 1u);
  if (hi == 0 && __popc(lo) <= G::K) S.lo[lo] = (uint16_t)colex(lo, 0, 0);
  if (lo == 0 && __popc(hi) <= G::K) S.hi[hi] = colex(hi, G::kLoBits, G::K - __popc(hi));
  if (mask > G::kFull || __popc(mask) != G::K) return;
  const uint32_t sub = colex(mask, 0, 0);
  uint32_t free_cells = G::kFull & ~mask, n = 0;
  uint4 v = make_uint4(0, 0, 0, 0);
  while (free_cells) {
    const uint32_t r = flood<W>(G::kFull & ~mask, free_cells & (0u - free_cells));
    free_cells &= ~r;
    if (n & 1u) v.x |= r;
    if (n & 2u) v.y |= r;
    if (n & 4u) v.z |= r;
    ++n;
  }
  v.w = n;
  S.regions[sub] = v;
  if (n > 1) atomicOr(S.split + sub / 32, 1u << (sub % 32));
  atomicAdd(n_regions, (unsigned long long)n);
}

// One table's search.
struct BfsArgs {
  SubsetTables subsets;
  uint32_t *queue;    // rank << 3 | region of every state, in the order found
  uint32_t cap;       // its entries: the number of states
  uint32_t *visited;  // regions 0-3 of a placement: a nibble
  uint32_t *extra;    // region 4: a bit
  uint8_t *lookup;
  uint32_t *bounds;   // level d: queue[bounds[d] .. bounds[d + 1])
  uint32_t *tail;     // entries in the queue
  uint32_t *done;     // blocks of this level that have finished
  uint32_t goal;      // lookup index of the goal
};

struct Goal {
  uint32_t rank, region, index;
};

__global__ void bfs_start_kernel(BfsArgs A, Goal g) {
  A.queue[0] = g.rank << 3 | g.region;
  A.visited[g.rank >> 3] = 1u << (4 * (g.rank & 7u) + g.region);  // the blank's home region is number 0..3
  A.lookup[g.index] = 0;
  A.bounds[0] = 0;
  A.bounds[1] = 1;
  *A.tail = 1;
  *A.done = 0;
}

// Expand level d: a lane takes a state, its warp tries the K * 4 moves in
// turn, four at a time with their reads and then their atomics in flight
// together (2.9 ms; one at a time 3.1), tests a child's visited bit by a
// plain read first -- 9 in 10 were seen before -- and appends what is new to
// the queue through a buffer of the warp, one reservation per 128-256
// entries.  A child's rank and lookup index
// differ from its parent's by constants, except that a vertical move also
// passes up to W - 1 occupied cells.
// Bound by its reads of the visited bits (64 MB) and, where the occupied
// cells divide the board (37 % of the subsets), of the region table (2.8 MB),
// all in L2, at half of the issue slots: the largest level of a 6-tile table
// (21 M states, 225 M children) takes 2.9 ms, 181 G L2 sectors/s.  Both
// 24-puzzle tables 546 -> 52 ms, the three 15-puzzle ones 6.1 -> 1.7 ms.
// The version before it scanned a [placement][region]
// byte array of 4.1 GB per level, expanded the 1-3 hits of a warp in turn and
// waited for the host after each level.
constexpr int kBfsBlock = 512;
constexpr uint32_t kBfsBuf = 256;
template <int W>
__global__ void __launch_bounds__(kBfsBlock) bfs_level_kernel(BfsArgs A, int d) {
  using G = Geo<W>;
  constexpr int N = G::N, K = G::K;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ uint32_t s_hi[1u << (N - G::kLoBits)], s_split[G::kSubsetWords];
  __shared__ uint16_t s_lo[1u << G::kLoBits];
  __shared__ uint32_t s_buf[kBfsBlock / 32][kBfsBuf];
  const uint32_t s0 = A.bounds[d], s1 = A.bounds[d + 1];
  if (s0 == s1) {  // an empty level: the search is over
    if (blockIdx.x == 0 && threadIdx.x == 0) A.bounds[d + 2] = s1;
    return;
  }
  for (uint32_t i = threadIdx.x; i < (1u << G::kLoBits); i += kBfsBlock) s_lo[i] = __ldg(A.subsets.lo + i);
  for (uint32_t i = threadIdx.x; i < (1u << (N - G::kLoBits)); i += kBfsBlock) s_hi[i] = __ldg(A.subsets.hi + i);
  for (uint32_t i = threadIdx.x; i < G::kSubsetWords; i += kBfsBlock) s_split[i] = __ldg(A.subsets.split + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t *buf = s_buf[threadIdx.x >> 5];
  uint32_t n_buf = 0;  // the same in all lanes
  auto flush = [&]() {
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(A.tail, n_buf);
    at = __shfl_sync(FULL, at, 0);
    for (uint32_t i = lane; i < n_buf; i += 32)
      if (at + i < A.cap) A.queue[at + i] = buf[i];
    __syncwarp();
    n_buf = 0;
  };
  auto subset = [&](uint32_t mask) -> uint32_t {
    return s_lo[mask & ((1u << G::kLoBits) - 1u)] + s_hi[mask >> G::kLoBits];
  };
  const uint32_t warps = gridDim.x * (kBfsBlock / 32), warp = (blockIdx.x * kBfsBlock + threadIdx.x) >> 5;
  // a small level is spread over K times as many warps, a tile each
  const uint32_t packs = (s1 - s0 + 31) / 32;
  const bool spread = packs * K <= warps;
  const int only = spread ? (int)(warp % K) : -1;
  for (uint32_t pack = spread ? warp / K : warp; pack < packs; pack += warps) {
    const uint32_t base = s0 + 32 * pack;
    const bool valid = base + lane < s1;
    const uint32_t ent = valid ? A.queue[base + lane] : 0u;
    const uint32_t rank = ent >> 3;
    int pos[K];
    unrank<W>(rank, pos);
    const uint32_t index = lookup_index<W>(pos);
    uint32_t mask = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) mask |= 1u << pos[j];
    const uint4 e = __ldg(A.subsets.regions + subset(mask));
    uint32_t reg = valid ? G::kFull & ~mask : 0u;  // cells of the blank's region
    reg &= ent & 1u ? e.x : ~e.x;
    reg &= ent & 2u ? e.y : ~e.y;
    reg &= ent & 4u ? e.z : ~e.z;
    // bit p set: the tile on cell p can move that way into the region
    const uint32_t can[4] = {reg << W, (reg & ~G::column(0)) >> 1, (reg & ~G::column(W - 1)) << 1, reg >> W};
    uint32_t earlier = 0;  // cells of the tiles before j
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int p = pos[j];
      if (only >= 0 && only != j) {
        earlier |= 1u << p;
        continue;
      }
      constexpr int step[4] = {-W, 1, -1, W};
      // the tile's four moves: their reads first, all in flight together
      uint4 ce[4];
      uint32_t r2[4], word[4];
#pragma unroll
      for (int dir = 0; dir < 4; ++dir) {
        ce[dir] = make_uint4(0, 0, 0, 0);
        r2[dir] = word[dir] = 0;
        if ((can[dir] >> p) & 1u) {
          const int c = p + step[dir];
          const uint32_t sub = subset(mask ^ (1u << p) ^ (1u << c));
          if ((s_split[sub / 32] >> (sub % 32)) & 1u) ce[dir] = __ldg(A.subsets.regions + sub);  // else region 0
          int change = step[dir];  // of digit j: the cells passed, less those of earlier tiles
          int32_t later = 0;       // of the later digits: one more tile before them, or one less
          if (dir == 0 || dir == 3) {
            const uint32_t passed = mask & (((1u << (W - 1)) - 1u) << (min(p, c) + 1));
            const int nb = __popc(passed & earlier);
            change += dir == 3 ? -nb : nb;
#pragma unroll
            for (int i = j + 1; i < K; ++i)
              if ((passed >> pos[i]) & 1u) later += (int32_t)G::rank_weight(i);
            if (dir == 0) later = -later;
          }
          r2[dir] = rank + (uint32_t)(change * (int32_t)G::rank_weight(j) + later);
          word[dir] = __ldcg(A.visited + (r2[dir] >> 3));
        }
      }
      // then the bits of the unseen children, again in flight together
      uint32_t region[4], old[4];
#pragma unroll
      for (int dir = 0; dir < 4; ++dir) {
        region[dir] = ((ce[dir].x >> p) & 1u) | ((ce[dir].y >> p) & 1u) << 1 | ((ce[dir].z >> p) & 1u) << 2;
        const uint32_t bit = 4 * (r2[dir] & 7u) + region[dir];
        old[dir] = 0xFFFFFFFFu;
        if ((can[dir] >> p) & 1u) {
          if (region[dir] > 3) old[dir] = atomicOr(A.extra + (r2[dir] >> 5), 1u << (r2[dir] & 31u));
          else if (!((word[dir] >> bit) & 1u)) old[dir] = atomicOr(A.visited + (r2[dir] >> 3), 1u << bit);
        }
      }
#pragma unroll
      for (int dir = 0; dir < 4; ++dir) {
        const uint32_t sh = 4 * (r2[dir] & 7u);
        const bool fresh = !((old[dir] >> (region[dir] > 3 ? r2[dir] & 31u : sh + region[dir])) & 1u);
        if (fresh) {
          const uint32_t x = index + (uint32_t)(step[dir] * (int32_t)G::index_weight(j));
          // the placement's entry is written by its first visit, of any
          // region; the bits of five regions are in two words, so for these
          // the entry itself tells (writers of one level write the same value)
          const bool first = ce[dir].w > 4 ? x != A.goal && __ldcg(A.lookup + x) == 0 : ((old[dir] >> sh) & 15u) == 0;
          if (first) A.lookup[x] = (uint8_t)(d + 1);
        }
        const unsigned got = __ballot_sync(FULL, fresh);
        if (fresh) buf[n_buf + __popc(got & ((1u << lane) - 1u))] = r2[dir] << 3 | region[dir];
        n_buf += __popc(got);
      }
      __syncwarp();
      if (n_buf > kBfsBuf - 128) flush();
      earlier |= 1u << p;
    }
  }
  if (n_buf) flush();
  // the last block to finish closes the next level
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(A.done, 1u) == gridDim.x - 1) {
      *A.done = 0;
      A.bounds[d + 2] = atomicAdd(A.tail, 0u);
    }
  }
}

template <int W>
__global__ void compact_lookup_kernel(const uint8_t *src, uint8_t *dst, uint32_t T, int to_lookup) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < T; r += gridDim.x * blockDim.x) {
    int pos[Geo<W>::K];
    unrank<W>(r, pos);
    const uint32_t x = lookup_index<W>(pos);
    if (to_lookup) dst[x] = src[r];
    else dst[r] = src[x];
  }
}

template <int W, bool PDB>
__global__ void heuristic_kernel(const uint8_t *boards, int n, int32_t *hout, const HeurTables *ht,
                                 const uint8_t *tables) {
  constexpr int N = W * W;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  hout[i] = board_h<W, PDB>(boards + (size_t)i * N, ht, tables);
}

int grid_for(uint64_t T, int block) {
  uint64_t g = (T + block - 1) / block;
  if (g > 152ull * 64ull) g = 152ull * 64ull;
  return (int)(g ? g : 1);
}

}  // namespace

uint64_t compact_table_size(int w) {
  PatternSet ps = pattern_set(w);
  uint64_t s = 1;
  for (int i = 0; i < ps.k; ++i) s *= (uint64_t)(w * w - i);
  return s;
}

uint64_t lookup_table_stride(int w) { return w == 4 ? (1ull << 20) : (1ull << 28); }

static cudaError_t launch_compact_lookup(int w, const uint8_t *src, uint8_t *dst, int to_lookup, cudaStream_t st) {
  const uint64_t T = compact_table_size(w);
  if (w == 4) compact_lookup_kernel<4><<<grid_for(T, 256), 256, 0, st>>>(src, dst, (uint32_t)T, to_lookup);
  else compact_lookup_kernel<5><<<grid_for(T, 256), 256, 0, st>>>(src, dst, (uint32_t)T, to_lookup);
  note_launch();
  return cudaGetLastError();
}

cudaError_t pdb_compact_to_lookup(int w, const uint8_t *compact, uint8_t *lookup, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(lookup, 0, lookup_table_stride(w), st);
  if (e != cudaSuccess) return e;
  return launch_compact_lookup(w, compact, lookup, 1, st);
}

cudaError_t pdb_lookup_to_compact(int w, const uint8_t *lookup, uint8_t *compact, cudaStream_t st) {
  return launch_compact_lookup(w, lookup, compact, 0, st);
}

namespace {

// Levels launched between two looks at the queue from the host: the launches
// after the last level cost about 3 us each, a look about 15.
constexpr int kLevelsPerLook = 8;
constexpr int kMaxLevels = 254;  // distances are bytes

// The goal: pattern tiles home, blank in the region of cell 0.
template <int W>
Goal goal_state(const PatternSet &ps, int table) {
  using G = Geo<W>;
  Goal g{0, 0, 0};
  uint32_t occ = 0;
  for (int j = 0; j < G::K; ++j) {
    const int cell = ps.table_tiles[table][j];
    g.rank += G::rank_weight(j) * (uint32_t)(cell - __builtin_popcount(occ & ((1u << cell) - 1u)));
    g.index += G::index_weight(j) * (uint32_t)cell;
    occ |= 1u << cell;
  }
  // regions are numbered by their lowest cells, so cell 0's, when it is free
  // (it is the blank's home), is number 0
  return g;
}

template <int W>
cudaError_t build_tables(uint8_t *lookup, cudaStream_t st) {
  using G = Geo<W>;
  const PatternSet ps = pattern_set(W);
  const uint64_t T = compact_table_size(W);
  constexpr size_t lo_n = (size_t)1 << G::kLoBits, hi_n = (size_t)1 << (G::N - G::kLoBits);
  const size_t vis_n = (T + 7) / 8, extra_n = (T + 31) / 32;
  // one allocation: 16-byte records first, then words; the state counter is 8-byte aligned
  const size_t words = 4 * (size_t)G::kSubsets + 2 + G::kSubsetWords + lo_n / 2 + hi_n + vis_n + extra_n + kMaxLevels +
                       kLevelsPerLook + 8;
  uint32_t *mem = nullptr, *queue = nullptr, *h_bounds = nullptr;
  cudaError_t e = cudaMalloc(&mem, words * sizeof(uint32_t));
  if (e == cudaSuccess)
    e = cudaMallocHost(&h_bounds, (kMaxLevels + kLevelsPerLook + 4) * sizeof(uint32_t));
  int blocks = 0, dev = 0, sms = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, bfs_level_kernel<W>, kBfsBlock, 0);
  if (e == cudaSuccess) {
    BfsArgs A{};
    A.subsets.regions = reinterpret_cast<uint4 *>(mem);
    unsigned long long *n_regions = reinterpret_cast<unsigned long long *>(mem + 4 * (size_t)G::kSubsets);
    A.subsets.split = mem + 4 * (size_t)G::kSubsets + 2;
    A.subsets.lo = reinterpret_cast<uint16_t *>(A.subsets.split + G::kSubsetWords);
    A.subsets.hi = A.subsets.split + G::kSubsetWords + lo_n / 2;
    A.visited = A.subsets.hi + hi_n;
    A.extra = A.visited + vis_n;
    A.bounds = A.extra + extra_n;
    A.tail = A.bounds + kMaxLevels + kLevelsPerLook + 4;
    A.done = A.tail + 1;
    // subset tables; the number of states is k! placements for every region of a subset
    e = cudaMemsetAsync(n_regions, 0, sizeof(unsigned long long) + G::kSubsetWords * sizeof(uint32_t), st);
    if (e == cudaSuccess) {
      subset_kernel<W><<<(G::kFull >> 8) + 1, 256, 0, st>>>(A.subsets, n_regions);
      note_launch();
      e = cudaGetLastError();
    }
    unsigned long long *h_regions = reinterpret_cast<unsigned long long *>(h_bounds);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(h_regions, n_regions, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) {
      uint64_t states = *h_regions;
      for (int i = 2; i <= G::K; ++i) states *= (uint64_t)i;
      A.cap = (uint32_t)states;
      e = cudaMalloc(&queue, states * sizeof(uint32_t));
      A.queue = queue;
    }
    for (int t = 0; e == cudaSuccess && t < ps.n_tables; ++t) {
      A.lookup = lookup + (size_t)t * lookup_table_stride(W);
      e = cudaMemsetAsync(A.lookup, 0, lookup_table_stride(W), st);
      if (e == cudaSuccess) e = cudaMemsetAsync(A.visited, 0, (vis_n + extra_n) * sizeof(uint32_t), st);
      if (e != cudaSuccess) break;
      const Goal g = goal_state<W>(ps, t);
      A.goal = g.index;
      bfs_start_kernel<<<1, 1, 0, st>>>(A, g);
      note_launch();
      e = cudaGetLastError();
      bool over = false;
      for (int d = 0; e == cudaSuccess && !over && d < kMaxLevels; d += kLevelsPerLook) {
        const int n = kMaxLevels - d < kLevelsPerLook ? kMaxLevels - d : kLevelsPerLook;
        for (int l = 0; l < n && e == cudaSuccess; ++l) {
          bfs_level_kernel<W><<<sms * blocks, kBfsBlock, 0, st>>>(A, d + l);
          note_launch();
          e = cudaGetLastError();
        }
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(h_bounds, A.bounds + d + n, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        over = e == cudaSuccess && h_bounds[0] == h_bounds[1];
      }
    }
  }
  cudaFree(queue);
  cudaFree(mem);
  cudaFreeHost(h_bounds);
  return e;
}

}  // namespace

cudaError_t build_pdb_tables(int w, uint8_t *lookup, cudaStream_t st) {
  return w == 4 ? build_tables<4>(lookup, st) : build_tables<5>(lookup, st);
}

cudaError_t launch_heuristic(int w, bool pdb, const uint8_t *boards, int n, int32_t *h,
                             const HeurTables *ht, const uint8_t *tables, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (n + 127) / 128;
  if (w == 4) {
    if (pdb) heuristic_kernel<4, true><<<blocks, 128, 0, st>>>(boards, n, h, ht, tables);
    else heuristic_kernel<4, false><<<blocks, 128, 0, st>>>(boards, n, h, ht, tables);
  } else {
    if (pdb) heuristic_kernel<5, true><<<blocks, 128, 0, st>>>(boards, n, h, ht, tables);
    else heuristic_kernel<5, false><<<blocks, 128, 0, st>>>(boards, n, h, ht, tables);
  }
  note_launch();
  return cudaGetLastError();
}

}  // namespace sp
