// Root set ("frontier") of a batch on the device.
//
// The root set of an instance is its search tree expanded to a uniform depth
// D with no pruning and no duplicate detection (the reference builds a root
// set of BLOCK_NUM nodes per instance, create_root_set in
// src/24puzzle_block_parallel_with_pdb.cu:454-490).  Without pruning the
// tree's shape -- which move sequences it holds, in breadth-first order --
// depends only on the cell of the blank, so the host builds one template per
// blank cell (moves from the root, parent, depth, children) and this kernel
// applies it to every instance at once: blocks replay each node's moves on the
// instance's board and compute h, and an instance's last one finds the prefix
// maximum of g + h along each node's path and writes
//   * the leaves (depth D) as SubRoot records sorted by that maximum, ties in
//     tree order (the active roots of a threshold round are then a prefix);
//   * per maximum value: the number of leaves, the children generated by
//     interior nodes, and the shallowest goal node (h == 0), which is what
//     the threshold loop needs to count the nodes above the roots.
// Bound by latency for one instance, on the path of every call: one 15-puzzle's
// root set, with a block per instance for all of it and boards in local
// memory, 84 us by Manhattan and 142 by tables (24-puzzles 205), now 55 and 58
// (82), of which finding h takes 6 (26 for 50 24-puzzles).
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/slide.h"
#include "sp_defs.h"
#include "sp_device.cuh"
#include "sp_kernels.h"

namespace sp {
namespace {

constexpr int kFrontThreads = 1024;
constexpr int kFrontWarps = kFrontThreads / 32;

// A thread's board: words of four cells, one column per thread ([word][thread]:
// no bank conflict whatever cell a thread indexes; as byte arrays in local
// memory, where the lanes of a warp hit up to 32 lines an access, the replays
// took most of the kernel's time).
template <int W, int T>
struct BoardColumn {
  static constexpr int kWords = (W * W + 3) / 4;
  uint32_t *col;
  __device__ __forceinline__ uint8_t &cell(int c) const {
    return reinterpret_cast<uint8_t *>(col + (c >> 2) * T)[c & 3];
  }
  // the board after `depth` moves of `path` from the root; returns the blank's cell
  __device__ __forceinline__ int replay(const uint32_t *root, int blank, uint64_t path, int depth) const {
#pragma unroll
    for (int q = 0; q < kWords; ++q) col[q * T] = root[q];
    for (int j = 0; j < depth; ++j) {
      const int src = blank + move_delta(W, (int)((path >> (2 * j)) & 3u));
      cell(blank) = cell(src);
      blank = src;
    }
    cell(blank) = 0;
    return blank;
  }
};

// The root's board as words, and its blank; the block synchronises afterwards.
template <int W>
__device__ __forceinline__ void load_root(const uint8_t *tiles, uint32_t (&s_root)[8], int &s_blank) {
  if (threadIdx.x < 32) {
    const uint8_t v = threadIdx.x < W * W ? tiles[threadIdx.x] : (uint8_t)0;
    reinterpret_cast<uint8_t *>(s_root)[threadIdx.x] = v;
    if (threadIdx.x < W * W && v == 0) s_blank = threadIdx.x;
  }
}

// `chunks` blocks per instance, so that a single instance's 11400 nodes are
// spread over SMs too; the one that finishes last does the rest.
template <int W, bool PDB>
__global__ void __launch_bounds__(kFrontThreads) frontier_kernel(FrontArgs A, uint32_t chunks) {
  constexpr int N = W * W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t li = blockIdx.x / chunks, first = blockIdx.x % chunks * kFrontThreads;
  const uint32_t inst = A.live[li];
  const uint32_t ti = A.live_tmpl[li];
  const FrontTmpl T = A.tmpl[ti];
  if (first >= T.n_nodes) return;
  const uint32_t *lev = A.lev + (size_t)ti * kFrontLevStride;
  const uint64_t *path = A.path + T.node_off;
  const int32_t *parent = A.parent + T.node_off;
  const uint8_t *nchild = A.nchild + T.node_off;
  const uint8_t *depth = A.depth + T.node_off;
  int16_t *F = A.f + A.live_scratch[li];
  int16_t *M = A.maxf + A.live_scratch[li];

  using Col = BoardColumn<W, kFrontThreads>;
  __shared__ uint32_t s_root[8], s_board[Col::kWords][kFrontThreads], s_lev[kFrontLevStride];
  __shared__ int s_blank, s_bad, s_last;
  __shared__ uint32_t s_leaf[kFrontBuckets], s_child[kFrontBuckets], s_goal[kFrontBuckets];
  __shared__ uint32_t s_wcnt[kFrontWarps][kFrontBuckets];
  const Col bd{&s_board[0][tid]};

  load_root<W>(A.tiles + (size_t)inst * N, s_root, s_blank);
  __syncthreads();
  // 1. g + h of every node
  if (const uint32_t x = first + tid; x < T.n_nodes) {
    const int dep = depth[x];
    bd.replay(s_root, s_blank, path[x], dep);
    uint64_t ra = 0, rb = 0, fa = 0, fb = 0;
    int h = 0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const uint32_t t = (bd.col[(c / 4) * kFrontThreads] >> (8 * (c % 4))) & 0xFFu;
      if (PDB) {  // the packed index sums (HeurTables::sum)
        const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(A.ht->sum) + (t * N + c) * (W == 4 ? 1u : 2u);
        const ulonglong2 v = __ldg(rec);
        if (W == 4) {
          ra += v.x;
          fa += v.y;
        } else {
          const ulonglong2 u = __ldg(rec + 1);
          ra += v.x;
          rb += v.y;
          fa += u.x;
          fb += u.y;
        }
      } else if (t) {
        h += abs(c / W - (int)t / W) + abs(c % W - (int)t % W);
      }
    }
    if (PDB) {
      constexpr int kPat = W == 4 ? 3 : 4;
      int hr = 0, hf = 0;
#pragma unroll
      for (int p = 0; p < kPat; ++p) {
        const uint32_t base = W == 4 ? (uint32_t)p << 20 : (p ? 1u << 28 : 0u);
        hr += __ldg(A.pdb + (sum_field<W>(ra, rb, p) | base));
        hf += __ldg(A.pdb + (sum_field<W>(fa, fb, p) | base));
      }
      h = max(hr, hf);
    }
    F[x] = (int16_t)(dep + h);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(A.arrived + li, 1u) == (T.n_nodes - 1u) / kFrontThreads;
  for (int b = tid; b < kFrontBuckets; b += kFrontThreads) {
    s_leaf[b] = 0;
    s_child[b] = 0;
    s_goal[b] = 0xFFFFFFFFu;
    for (int q = 0; q < kFrontWarps; ++q) s_wcnt[q][b] = 0;
  }
  for (uint32_t d = tid; d <= T.D + 1; d += kFrontThreads) s_lev[d] = lev[d];
  if (tid == 0) s_bad = 0;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int h0 = __ldcg(F);  // other blocks' values: past L1
  // 2. prefix maximum of g + h along each path, one level at a time (the
  //    parent of a level-d node is on level d - 1)
  for (uint32_t d = 0; d <= T.D; ++d) {
    for (uint32_t x = s_lev[d] + tid; x < s_lev[d + 1]; x += kFrontThreads) {
      const int f = __ldcg(F + x);
      M[x] = (int16_t)(d ? max(f, (int)M[parent[x]]) : f);
    }
    __syncthreads();
  }
  // 3. per maximum (bucket = maxf - h0): leaves, interior children, goals
  for (uint32_t x = tid; x < T.n_nodes; x += kFrontThreads) {
    const int b = M[x] - h0;
    const int dep = depth[x];
    if (b < 0 || b >= kFrontBuckets) {
      s_bad = 1;
      continue;
    }
    if ((uint32_t)dep == T.D) atomicAdd(&s_leaf[b], 1u);
    else atomicAdd(&s_child[b], (uint32_t)nchild[x]);
    if (__ldcg(F + x) == dep) atomicMin(&s_goal[b], ((uint32_t)dep << 24) | x);
  }
  __syncthreads();
  if (s_bad) {  // h changed by more than the bucket range allows along a path
    if (tid == 0) atomicCAS(A.error, 0, (int32_t)SP_ERR_ARG);
    return;
  }
  if (warp == 0) {  // exclusive prefix of the leaf counts, kept in s_leaf
    constexpr int kEach = kFrontBuckets / 32;
    uint32_t v[kEach], sum = 0;
#pragma unroll
    for (int q = 0; q < kEach; ++q) sum += v[q] = s_leaf[lane * kEach + q];
    uint32_t c = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, c, o);
      if (lane >= o) c += u;
    }
    c -= sum;
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
      s_leaf[lane * kEach + q] = c;
      c += v[q];
    }
  }
  __syncthreads();
  // 4. the leaves in tree order, each to its bucket's next position (a
  //    stable counting sort: ranks within a warp from the match mask, then
  //    the counts of the lower warps of the same chunk)
  const uint32_t l0 = s_lev[T.D], l1 = s_lev[T.D + 1];
  const uint32_t base = A.live_base[li];
  for (uint32_t c0 = l0; c0 < l1; c0 += kFrontThreads) {
    const uint32_t x = c0 + tid;
    const bool valid = x < l1;
    const int b = valid ? M[x] - h0 : kFrontBuckets;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, b);
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    if (valid && rank == 0) s_wcnt[warp][b] = __popc(peers);
    __syncthreads();
    if (valid) {
      uint32_t pos = s_leaf[b] + rank;
      for (int q = 0; q < warp; ++q) pos += s_wcnt[q][b];
      const uint32_t j = base + pos;
      const int blank = bd.replay(s_root, s_blank, path[x], (int)T.D);
      const uint32_t pre = T.D ? (uint32_t)(path[x] >> (2 * (T.D - 1))) & 3u : kNoPre;
      const uint32_t tail = (uint32_t)blank << 8 | T.D << 16 | pre << 24;
      auto word = [&](int q) -> uint32_t { return q < Col::kWords ? bd.col[q * kFrontThreads] : 0u; };
      uint4 *dst = reinterpret_cast<uint4 *>(A.subs + j);
      dst[0] = make_uint4(word(0), word(1), word(2), word(3));
      dst[1] = make_uint4(word(4), word(5), (word(6) & 0xFFu) | tail, inst);
      A.leaf_maxf[j] = M[x];
      A.leaf_h[j] = (uint8_t)(__ldcg(F + x) - (int)T.D);
      A.leaf_node[j] = (int32_t)x;
    }
    __syncthreads();
    for (int bb = tid; bb < kFrontBuckets; bb += kFrontThreads) {
      uint32_t t = 0;
      for (int q = 0; q < kFrontWarps; ++q) {
        t += s_wcnt[q][bb];
        s_wcnt[q][bb] = 0;
      }
      s_leaf[bb] += t;
    }
    __syncthreads();
  }
  // 5. per-instance summary (s_leaf now holds inclusive counts)
  FrontInst *O = A.out + li;
  if (tid == 0) {
    O->h0 = h0;
    O->n_leaves = l1 - l0;
  }
  for (int b = tid; b < kFrontBuckets; b += kFrontThreads) {
    O->leaf_cum[b] = s_leaf[b];
    O->child[b] = s_child[b];
    O->goal[b] = s_goal[b];
  }
}

}  // namespace

cudaError_t launch_frontier(int w, bool pdb, int n_live, uint32_t max_nodes, const FrontArgs &A, cudaStream_t st) {
  if (n_live <= 0) return cudaSuccess;
  const uint32_t chunks = (max_nodes + kFrontThreads - 1) / kFrontThreads;
  const uint64_t grid64 = (uint64_t)n_live * chunks;
  if (!chunks || grid64 > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
  const uint32_t grid = (uint32_t)grid64;
  if (w == 4) {
    if (pdb) frontier_kernel<4, true><<<grid, kFrontThreads, 0, st>>>(A, chunks);
    else frontier_kernel<4, false><<<grid, kFrontThreads, 0, st>>>(A, chunks);
  } else {
    if (pdb) frontier_kernel<5, true><<<grid, kFrontThreads, 0, st>>>(A, chunks);
    else frontier_kernel<5, false><<<grid, kFrontThreads, 0, st>>>(A, chunks);
  }
  note_launch();
  return cudaGetLastError();
}

}  // namespace sp
