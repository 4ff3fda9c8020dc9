// sp_idas_parallel: Horie's host-callable search (src_horie/idas_parallel_host.h:33-34,
// src_horie/idas_parallel.cu:239-244), the one C function of the reference
// that a host program can call.
//
// Semantics kept from the reference (src_horie/idas_parallel.cu:172-236):
// every root of the 15-puzzle is searched on its own, depth-first, moves
// tried in the order up, right, left, down, the reverse of the last move
// skipped (none at the root), a child entered only if its depth below the
// root + 1 + h <= f_limit, h updated by the caller's h-difference table
// (h_diff[tile][its cell][blank's move]; the reverse move on backtracking),
// moves allowed by the caller's movable table [cell][move]; the search of a
// root stops at its first goal, and the root's plan row is [len, moves...]
// or [-1].  The root's own depth is not counted: roots are searched as if at
// depth 0.  No node counts: the reference reports none on this path.  Two
// guards the reference lacks: a path never grows past the plan row (251
// moves), and a root that 30 s of its block's search have not settled gives up
// with [-2] (a block's roots start together and share its threads; a root never
// has fewer than one while it is open).
//
// GPU shape: a block for one root, or for several when there are many.  A
// depth-first search visits its tree's nodes in the order of their move
// sequences, so a root's tree is cut into intervals of that order, one per
// thread: a thread without work takes the untried moves of the shallowest
// open level of one that has some, which is the end of that thread's
// interval.  A thread's first goal is the first of its interval; the root's
// answer is the one of the earliest interval, and threads that are past it
// stop.  The version before walked each root by one thread and took as long
// as the slowest: 4096 roots of 26 moves 22-34 ms, now 0.95; 600 of them 16-27
// and 0.38; 400000 of 8 moves 0.10 and 0.08.
// Every thread holds its board packed 4 bits per cell in a 64-bit register
// and its moves, 2 bits per level, in shared memory ([word][thread]: every
// thread owns a bank); both tables are copied into shared memory by each
// block (or, with null table pointers, built there from the Manhattan
// distance as the reference's init_mdist / init_movable_table do,
// src_horie/idas_parallel_host.c:88-129).  With a table whose reverse moves
// do not take back what the moves added, h depends on the whole walk so far
// and one thread walks the root alone; so do the board and h of a root without
// a blank, which leaves its block's roots to one thread each too.  Allocates nothing; launches on the
// caller's stream and returns, like the reference.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/slide.h"
#include "sp_defs.h"
#include "sp_kernels.h"

namespace sp {
namespace {

constexpr int kW = 4, kN = 16;
constexpr int kFpWords = (SP_PLAN_STRIDE + 15) / 16;  // 2-bit moves per thread, 16 per word
constexpr unsigned long long kFpLimitNs = 30000000000ull;  // 30 s per root
// Steps between two looks for idle threads: short while many are idle.
constexpr int kFpStepsFew = 16, kFpStepsMany = 64;

__device__ __forceinline__ unsigned long long fp_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

struct FpTables {
  union {
    int8_t hdiff[kN * kN * 4];  // [tile][cell][move], the reference's layout
    uint32_t word[kN * kN];     // the four moves of a (tile, cell)
  };
  uint8_t moves[kN];          // [cell]: bit d = move d allowed
};

// Board, blank and h of a walk.
struct FpNode {
  uint64_t b;
  int blank, h;
  __device__ __forceinline__ int tile_at(int c) const { return (int)((b >> (4 * c)) & 15u); }
  // h after the blank's move d
  __device__ __forceinline__ int h_after(const FpTables &T, int d) const {
    const int to = blank + move_delta(kW, d);
    return h + T.hdiff[(tile_at(to) * kN + to) * 4 + d];
  }
  // the blank moves by d: the tile at the blank's new cell slides into its old one
  __device__ __forceinline__ void apply(const FpTables &T, int d) {
    const int to = blank + move_delta(kW, d);
    const uint64_t t = (uint64_t)tile_at(to);
    h += T.hdiff[((int)t * kN + to) * 4 + d];
    b ^= (t << (4 * to)) ^ (t << (4 * blank));
    blank = to;
  }
};

// The reference's walk by one thread, h changed by the table on the way back
// too.  Returns the path's length, -1 without a goal, -2 past the time limit;
// the moves are left in stk[word * stride].
__device__ int walk_alone(FpNode x, const FpTables &T, int f_limit, uint32_t *stk, int stride) {
  auto at = [&](int i) -> int { return (int)((stk[(i >> 4) * stride] >> (2 * (i & 15))) & 3u); };
  int depth = 0, dir = 0;
  unsigned long long t0 = 0;
  uint32_t spin = 0;
  for (;;) {
    if ((++spin & 4095u) == 0) {
      const unsigned long long now = fp_now();
      if (!t0) t0 = now;
      else if (now - t0 > kFpLimitNs) return -2;
    }
    if (x.h == 0) return depth;
    if ((depth == 0 || at(depth - 1) != 3 - dir) && ((T.moves[x.blank] >> dir) & 1u)) {
      if (depth + 1 + x.h_after(T, dir) <= f_limit && depth + 1 < SP_PLAN_STRIDE) {
        x.apply(T, dir);
        uint32_t &w = stk[(depth >> 4) * stride];
        w = (w & ~(3u << (2 * (depth & 15)))) | ((uint32_t)dir << (2 * (depth & 15)));
        ++depth;
        dir = 0;
        continue;
      }
    }
    while (++dir == 4) {
      if (depth == 0) return -1;
      dir = at(--depth);
      x.apply(T, 3 - dir);
    }
  }
}

// Block b's T threads search roots b * per .. (per <= MAX).
template <int T, int MAX>
__global__ void __launch_bounds__(T) first_path_kernel(const uint8_t *input, int n, int per, int8_t *plan, int f_limit,
                                                       const int8_t *hdiff_in, const uint8_t *movable_in) {
  __shared__ FpTables s_tab;
  __shared__ uint32_t s_stack[kFpWords][T];
  // per root: its board, blank and h; its earliest goal's moves; the thread
  // that may replace these; whether any thread still searches it
  __shared__ uint64_t s_board[MAX];
  __shared__ uint32_t s_best[kFpWords][MAX];
  __shared__ int s_best_len[MAX];
  __shared__ uint16_t s_claim[MAX];
  __shared__ uint8_t s_blank[MAX], s_h[MAX], s_open[MAX];
  __shared__ int s_alone, s_stop, s_idle, s_offers, s_min;
  __shared__ uint16_t s_from[T], s_level[T];  // offers: the thread and the level of its open moves
  __shared__ uint16_t s_rid[T];               // the thread's root
  const int tid = threadIdx.x;
  const int first = blockIdx.x * per, nr = min(per, n - first);
  if (tid == 0) s_alone = 0;
  for (int i = tid; i < kN * kN; i += T) {
    uint32_t w = 0;
    if (!hdiff_in) {
      // the tile at `cell` moves against the blank's move (blank up, right,
      // left, down: tile down, left, right, up): one step closer to or
      // farther from its goal cell (the tile's number)
      const int t = i / kN, c = i % kN;
      const int gr = t / kW, gc = t % kW, r = c / kW, cc = c % kW;
      w = (gr > r ? 0xFFu : 1u) | (gc < cc ? 0xFF00u : 0x100u) | (gc > cc ? 0xFF0000u : 0x10000u) |
          (gr < r ? 0xFF000000u : 0x1000000u);
    } else if (((uintptr_t)hdiff_in & 3u) == 0) {
      w = reinterpret_cast<const uint32_t *>(hdiff_in)[i];
    } else {
      for (int d = 0; d < 4; ++d) w |= (uint32_t)(uint8_t)hdiff_in[4 * i + d] << (8 * d);
    }
    s_tab.word[i] = w;
  }
  // a caller's movable table is also held to the board's edges, so that no
  // table can move the blank off the board
  for (int c = tid; c < kN; c += T) {
    uint32_t m = legal_moves(kW, c);
    if (movable_in)
      for (int d = 0; d < 4; ++d)
        if (!movable_in[c * 4 + d]) m &= ~(1u << d);
    s_tab.moves[c] = (uint8_t)m;
  }
  __syncthreads();
  if (hdiff_in) {
    for (int i = tid; i < kN * kN * 4; i += T) {
      const int t = i / (kN * 4), c = (i / 4) % kN, d = i % 4;
      const int to = c - move_delta(kW, d);  // the blank came to c by d, from `to`
      if (to >= 0 && to < kN && ((legal_moves(kW, to) >> d) & 1u) &&
          s_tab.hdiff[i] + s_tab.hdiff[(t * kN + to) * 4 + 3 - d] != 0)
        s_alone = 1;
    }
  }

  int rid = tid < nr ? tid : 0;
  if (tid < nr) {
    const uint8_t *tiles = input + (size_t)(first + tid) * kN;
    uint32_t word[4];
    if (((uintptr_t)input & 15u) == 0) {
      const uint4 v = *reinterpret_cast<const uint4 *>(tiles);
      word[0] = v.x, word[1] = v.y, word[2] = v.z, word[3] = v.w;
    } else {
      for (int q = 0; q < 4; ++q)
        word[q] = tiles[4 * q] | (uint32_t)tiles[4 * q + 1] << 8 | (uint32_t)tiles[4 * q + 2] << 16 |
                  (uint32_t)tiles[4 * q + 3] << 24;
    }
    FpNode r{0, 0, 0};
#pragma unroll
    for (int c = 0; c < kN; ++c) {
      const uint32_t t = (word[c / 4] >> (8 * (c % 4))) & 15u;
      r.b |= (uint64_t)t << (4 * c);
      if (!t) r.blank = c;
      else r.h += abs(c / kW - (int)t / kW) + abs(c % kW - (int)t % kW);
    }
    if (r.tile_at(r.blank)) s_alone = 1;
    s_board[tid] = r.b;
    s_blank[tid] = (uint8_t)r.blank;
    s_h[tid] = (uint8_t)r.h;
    s_best_len[tid] = r.h == 0 ? 0 : -1;
    s_open[tid] = 0;
  }
  if (tid == 0) {
    s_stop = 0;
    s_idle = T - nr;
  }
  __syncthreads();
  auto root = [&](int r) { return FpNode{s_board[r], s_blank[r], s_h[r]}; };
  if (s_alone) {
    if (tid < nr) {
      int8_t *row = plan + (size_t)(first + tid) * SP_PLAN_STRIDE;
      const int len = walk_alone(root(tid), s_tab, f_limit, &s_stack[0][tid], T);
      row[0] = (int8_t)len;
      for (int i = 0; i < len; ++i) row[1 + i] = (int8_t)((s_stack[i >> 4][tid] >> (2 * (i & 15))) & 3u);
    }
    return;
  }

  // ---- the thread's walk ----
  FpNode x = root(rid);
  bool active = tid < nr && x.h != 0, found = false;
  int depth = 0;
  int base = 0, bblank = x.blank;  // levels below base have no untried moves of this thread; the blank's cell there
  uint32_t rem = s_tab.moves[x.blank];  // untried moves of the current node
  uint32_t top = 0;                   // the stack word holding level depth - 1 (completed words are in shared memory)
  auto move_at = [&](int i) -> int { return (int)((s_stack[i >> 4][tid] >> (2 * (i & 15))) & 3u); };
  // first difference in the order of walks between this thread's path and its
  // root's best: < 0 before, > 0 after, 0 one is the other's beginning
  auto order = [&]() -> int {
    const int len = min(depth, s_best_len[rid]);
    for (int w = 0; 16 * w < len; ++w) {
      uint32_t diff = s_stack[w][tid] ^ s_best[w][rid];
      if (16 * (w + 1) > len) diff &= (1u << (2 * (len & 15))) - 1u;
      if (diff) {
        const int sh = (__ffs(diff) - 1) & ~1;
        return (int)((s_stack[w][tid] >> sh) & 3u) - (int)((s_best[w][rid] >> sh) & 3u);
      }
    }
    return 0;
  };
  const unsigned long long t0 = fp_now();
  __syncthreads();
  for (;;) {
    // 1. walk
    const int steps = 4 * s_idle > T ? kFpStepsFew : kFpStepsMany;
    for (int s = 0; s < steps && active; ++s) {
      if (rem) {
        const int d = __ffs(rem) - 1;
        rem &= rem - 1u;
        const int nh = x.h_after(s_tab, d);
        if (depth + 1 + nh <= f_limit && depth + 1 < SP_PLAN_STRIDE) {
          x.apply(s_tab, d);
          const int sh = 2 * (depth & 15);
          top = sh ? (top & ~(3u << sh)) | ((uint32_t)d << sh) : (uint32_t)d;  // sh 0: a new word
          if (sh == 30) s_stack[depth >> 4][tid] = top;
          ++depth;
          rem = s_tab.moves[x.blank] & ~(1u << (3 - d));
          if (x.h == 0) {
            found = true;
            active = false;
          }
        }
      } else if (depth == base) {
        active = false;
      } else {
        --depth;  // undo the move of level depth, held in top
        const int d = (int)((top >> (2 * (depth & 15))) & 3u);
        if ((depth & 15) == 0 && depth > 0) top = s_stack[(depth >> 4) - 1][tid];
        x.apply(s_tab, 3 - d);
        rem = s_tab.moves[x.blank] & (0xFu << (d + 1));
        if (depth > 0) rem &= ~(1u << (3 - (int)((top >> (2 * ((depth - 1) & 15))) & 3u)));
      }
    }
    if (depth > 0) s_stack[(depth - 1) >> 4][tid] = top;
    // 2. goals of this round, one thread of a root after the other: the
    // earliest stays
    while (__syncthreads_or(found)) {
      if (found) s_claim[rid] = (uint16_t)tid;
      __syncthreads();
      if (found && s_claim[rid] == tid) {
        const int o = s_best_len[rid] < 0 ? -1 : order();
        if (o < 0 || (o == 0 && depth < s_best_len[rid])) {
          for (int w = 0; 16 * w < depth; ++w) s_best[w][rid] = s_stack[w][tid];
          s_best_len[rid] = depth;
        }
        found = false;
      }
    }
    if (active && s_best_len[rid] >= 0 && order() > 0) active = false;  // the answer is before all that is left here
    if (tid == 0) {
      s_idle = 0;
      s_offers = 0;
      s_min = SP_PLAN_STRIDE;
      if (fp_now() - t0 > kFpLimitNs) s_stop = 1;
    }
    __syncthreads();
    // 3. who is idle, and what could be given away: each thread's shallowest
    // level with an untried move
    int level = SP_PLAN_STRIDE, place = 0;
    if (!active) {
      place = atomicAdd(&s_idle, 1);
    } else {
      while (base < depth) {
        const int d = move_at(base);
        uint32_t un = s_tab.moves[bblank] & (0xFu << (d + 1));
        if (base > 0) un &= ~(1u << (3 - move_at(base - 1)));
        if (un) break;
        bblank += move_delta(kW, d);
        ++base;
      }
      if (base < depth) {
        level = base;
        atomicMin(&s_min, level);
      }
    }
    __syncthreads();
    const int idle = s_idle;
    if (idle == T || s_stop) break;
    if (idle) {
      // shallow levels only: the others' subtrees are small
      int offer = -1;
      if (level <= s_min + 2 && level < SP_PLAN_STRIDE) {
        offer = atomicAdd(&s_offers, 1);
        if (offer < idle) {
          s_from[offer] = (uint16_t)tid;
          s_level[offer] = (uint16_t)level;
          s_rid[tid] = (uint16_t)rid;
        }
      }
      __syncthreads();
      if (!active && place < s_offers) {
        // the moves after the one taken at `level` of the giver's path
        const int from = s_from[place], lev = s_level[place];
        rid = s_rid[from];
        x = root(rid);
        top = 0;
        for (int i = 0; i < lev; ++i) {
          if ((i & 15) == 0) {
            top = s_stack[i >> 4][from];
            s_stack[i >> 4][tid] = top;
          }
          x.apply(s_tab, (int)((top >> (2 * (i & 15))) & 3u));
        }
        const int d = (int)((s_stack[lev >> 4][from] >> (2 * (lev & 15))) & 3u);
        rem = s_tab.moves[x.blank] & (0xFu << (d + 1));
        if (lev > 0) rem &= ~(1u << (3 - (int)((top >> (2 * ((lev - 1) & 15))) & 3u)));
        depth = base = lev;
        bblank = x.blank;
        active = true;
      } else if (offer >= 0 && offer < idle) {
        bblank += move_delta(kW, move_at(base));
        ++base;
      }
      __syncthreads();  // the givers' paths have been read
    }
  }
  if (active) s_open[rid] = 1;  // stopped by the time limit
  __syncthreads();
  if (tid < nr) {
    int8_t *row = plan + (size_t)(first + tid) * SP_PLAN_STRIDE;
    const int len = s_open[tid] ? -2 : s_best_len[tid];
    row[0] = (int8_t)len;
    for (int i = 0; i < len; ++i) row[1 + i] = (int8_t)((s_best[i >> 4][tid] >> (2 * (i & 15))) & 3u);
  }
}

}  // namespace
}  // namespace sp

extern "C" int sp_idas_parallel(const uint8_t *d_input, int n, int8_t *d_plan, int f_limit,
                                const int8_t *d_h_diff_table, const uint8_t *d_movable_table, void *stream) {
  if (n < 0 || (n > 0 && (!d_input || !d_plan)) || f_limit < 0 || f_limit > SP_PLAN_STRIDE - 1) return SP_ERR_ARG;
  if (n == 0) return SP_OK;
  // an error the caller left pending is the caller's: report it without clearing it
  if (cudaPeekAtLastError() != cudaSuccess) return SP_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  // few roots: the hardest one decides, and more threads shorten it (64 roots
  // of 26 moves: 0.26 ms with 512, 0.39 with 128); many: a wave of blocks
  // holds all, several roots each, so that a block's threads start busy
  // (60000 roots of 20 moves: 0.50 ms with about 1024 blocks, 0.73 with 4096,
  // 2.3 with a block per root; 4096 of 26 moves: 0.95, 1.02, 1.02)
  if (n <= 304) {
    sp::first_path_kernel<512, 1><<<n, 512, 0, st>>>(d_input, n, 1, d_plan, f_limit, d_h_diff_table, d_movable_table);
  } else if (n <= 1024) {
    sp::first_path_kernel<256, 1><<<n, 256, 0, st>>>(d_input, n, 1, d_plan, f_limit, d_h_diff_table, d_movable_table);
  } else {
    const int per = n / 1024 < 128 ? n / 1024 : 128;
    sp::first_path_kernel<128, 128><<<(n + per - 1) / per, 128, 0, st>>>(d_input, n, per, d_plan, f_limit, d_h_diff_table,
                                                                        d_movable_table);
  }
  sp::note_launch();
  return cudaGetLastError() == cudaSuccess ? SP_OK : SP_ERR_CUDA;
}
