// Threshold-round search kernel of libslide.
//
// One launch searches one IDA* threshold for every unsolved instance of a
// batch.  It replaces the reference's per-round dfs_kernel
// (src/24puzzle_block_parallel_with_pdb.cu:520-648: one 32-thread block per
// root, 8 nodes x 4 moves per round, three __syncthreads per round, a
// 326-entry shared Node stack) with:
//
//  * one lane = one depth-first search over a task (a root-set node, possibly
//    narrowed to some of its first moves); no block barriers in the loop;
//  * the lane's whole state that is indexed by cell, pattern or level in
//    shared memory, one column of words per lane (LaneRows below), so that no
//    index costs a bank conflict, a 64-bit shift or a select;
//  * what a move changes from one table entry per (tile, cell, move): the
//    pattern-index changes or the Manhattan change
//    (src/15puzzle_block_parallel.cu:271-272 takes two constant-memory
//    lookups), and the child's move mask;
//  * PDB indices kept per pattern as mixed-radix integers and updated by one
//    add per move, so a generated child costs one regular and one reflected
//    table lookup instead of the reference's eight
//    (src/24puzzle_block_parallel_with_pdb.cu:426-429); the idea of updating
//    only the moved tile's pattern is Horie's (src_horie/idas_pdb.cu:221-254);
//    undoing a move restores the two overwritten values from the level's
//    bytes instead of looking them up again;
//  * generating a child and undoing a move share one code path (both slide
//    one tile into the blank), without a branch between the two.
//    Bound by issue and by table reads in flight.  Against the version with
//    register boards and indices, whose lanes drifted apart (9-15 of 32
//    active per instruction, 18-21 warp instructions per node), this step
//    alone, then with the choices of donors, block and L1 described below (21-24
//    and 5-9): 100 random 15-puzzles 28.8 -> 19.7 -> 15.9 ms, 4096 mixed ones
//    348 -> 211 -> 156 ms (the large rounds 70 -> 116 -> 140 G nodes/s), 100
//    Manhattan walks 29.2 -> 18.9 -> 8.9 ms, 16384 24-puzzle roots 166 -> 101
//    -> 59 ms (each chain on inputs of its own: other instances of a kind take up
//    to a fifth more or less);
//  * load balance by a device task pool: lanes claim slots warp-aggregated
//    (ballot + one atomicAdd per warp); claims may run ahead of the pool's
//    tail, and while any lane waits, busy lanes donate the untried moves of
//    their shallowest open level as a new task (the reference's closest
//    counterpart is Horie's intra-warp sharing, src_horie/idas_dynamic.cu
//    :200-247; the reference's own balance is the host re-split of
//    :839-897, done by the host round loop here).
//
// The multi-iteration variant (MULTI) runs every instance's whole threshold
// loop in one launch: the warp whose lane finishes an instance's last task of
// an iteration publishes that instance's next iteration (warp_advance), so
// instances never wait for each other and the host is not involved between
// iterations.  Its heavy roots go out as split tasks that expand one level
// per claim (breadth-first across lanes); an instance whose next iteration
// is predicted to be large is handed back to the host round loop.
//
// Every wait is bounded: a warp whose lanes all wait and see no change of the
// pool for timeout_ns sets SP_ERR_TIMEOUT and every warp returns.  Nothing
// traps.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/slide.h"
#include "sp_defs.h"
#include "sp_device.cuh"
#include "sp_kernels.h"

namespace sp {

namespace {

// Pool words are read with GPU-scope relaxed loads (coherent across SMs, never
// served from a stale L1 line); readiness of a slot with an acquire load, so
// the record written before its release store is visible.
__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int32_t ld_volatile(const int32_t *p) {
  int32_t v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Blank displacement of move d without compares: the four displacements as
// signed bytes of one immediate, byte d sign-extended by one permute.
template <int W>
__device__ __forceinline__ int step_delta(uint32_t d) {
  constexpr uint32_t pack = W == 4 ? 0x04FF01FCu : 0x05FF01FBu;  // -W, +1, -1, +W
  int r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(pack), "r"(d * 0x1111u + 0x8880u));
  return r;
}
// legal_moves from 4-bit masks of every cell packed into 64-bit immediates.
constexpr uint64_t legal_pack(int w, int first, int count) {
  uint64_t v = 0;
  for (int c = 0; c < count; ++c) {
    const int cell = first + c, r = cell / w, cc = cell % w;
    const uint64_t m = (r > 0 ? 1u : 0u) | (cc < w - 1 ? 2u : 0u) | (cc > 0 ? 4u : 0u) | (r < w - 1 ? 8u : 0u);
    v |= m << (4 * c);
  }
  return v;
}
template <int W>
__device__ __forceinline__ uint32_t step_legal(int blank) {
  const uint64_t w = W == 4 ? legal_pack(4, 0, 16) : blank < 16 ? legal_pack(5, 0, 16) : legal_pack(5, 16, 9);
  return (uint32_t)(w >> (4 * (blank & 15))) & 15u;
}
// Lowest move of a non-empty 4-bit move mask: sixteen 2-bit answers in one
// immediate.
__device__ __forceinline__ uint32_t first_move(uint32_t mask) { return (0x12131210u >> (2 * mask)) & 3u; }

}  // namespace

// Multi-iteration mode: split-piece load in units of the instance's average
// root load (1, 2 and 4 measure alike).
#ifndef SP_MULTI_PIECE
#define SP_MULTI_PIECE 1.0
#endif

// Multi-iteration mode: an iteration's roots go out as bulk tasks, each for
// up to kBulk of them: Task::sub is the first one's place (in P.order when
// `mask` is not 0, else the SubRoot itself), `plen` their number, bit 7 of
// `flags` set.  The warp whose lane claims a bulk publishes its roots, one per
// lane, so that the advancing warp's own publication takes a few rounds
// instead of one per 32 roots, each with a slot's acquire and release behind
// it.  Bulks are not counted as outstanding: their roots are, from the start.
constexpr uint32_t kBulk = 32;
constexpr uint32_t kBulkFlag = 0x80u;

// Publish task `D` at reserved pool index t (multi-iteration mode, where every
// index must be filled): waits a bounded time for the slot.
__device__ __forceinline__ void publish_root(const RoundParams &P, uint32_t t, uint32_t sub, uint32_t plen,
                                             uint32_t mask, uint32_t flags) {
  const uint32_t s = t & (P.cap - 1u);
  bool free_slot = false;
  for (int spin = 0; spin < (1 << 14) && !free_slot; ++spin) {
    free_slot = ld_acquire(&P.seq[s]) == t;
    if (!free_slot) __nanosleep(64);
  }
  if (!free_slot) {
    if (atomicCAS(&P.ctl->error, 0, SP_ERR_CAPACITY) == 0) P.ctl->err_info[0] = t;
    return;
  }
  Task *D = &P.tasks[s];
  D->mask = (uint8_t)mask;
  D->sub = sub;
  D->plen = (uint8_t)plen;
  D->flags = (uint8_t)flags;
  st_release(&P.seq[s], t + 1u);
}

// Multi-iteration mode: the warp of the lane that finished an instance's last
// task of an iteration completes that iteration (adds the root-set interior
// count, checks for a goal) and publishes the next iteration's roots -- the
// threshold loop of src/24puzzle_block_parallel_with_pdb.cu:772-921 run on the
// device, per instance, with no barrier across instances.  Called by all 32
// lanes of a warp with the same instance i; `hist` is the warp's 32 words of
// shared memory.  Kept out of line: it is cold, and inlined its registers
// would crowd the search loop.  When the instance's next iteration is
// predicted small (below P.pair_nodes) it is published together with this
// one, and the call that completes such a pair settles both in order.
// Bound by latency: nothing of the instance runs meanwhile.  So the reads of
// its state are in flight together, the searches for the active roots take 32
// probes at a time, the two passes over the roots' loads (sum and histogram;
// order and split) have eight loads in flight, all arithmetic is 32-bit float
// (it only orders and splits work), and the publication goes out in bulks.
// The device loop's launch on 100 random 15-puzzles 3.2 -> 2.6 ms, on one
// 15-puzzle walk of 40 moves 0.61 -> 0.52 ms.
__device__ __noinline__ void warp_advance(const RoundParams &P, uint32_t i, uint32_t *hist) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  PoolCtl *ctl = P.ctl;
  // per instance, two limits and two solution records, by iteration parity
  int r = ld_volatile(&P.inst_iter[i]);
  const uint32_t pair = ld_volatile(&P.inst_pair[i]);
  const int lim0 = ld_volatile(&P.inst_limit[2 * i]), lim1 = ld_volatile(&P.inst_limit[2 * i + 1]);
  const uint32_t flag0 = ld_volatile(&P.sol[2 * i].flag), flag1 = ld_volatile(&P.sol[2 * i + 1].flag);
  const int goal = P.goal_maxf[i];
  const uint32_t base = P.inst_sub_base[i], ns = P.inst_nsub[i];
  const uint32_t ioff = P.inter_off[i], ilen = P.inter_len[i];
  // children of root-set interior nodes within L (entries ascending in f)
  auto interior = [&](int L) -> unsigned long long {
    uint32_t n = 0;
    for (uint32_t q = 0; q < ilen; q += 32) {
      const unsigned in = __ballot_sync(FULL, q + lane < ilen && P.inter_f[ioff + q + lane] <= L);
      n += (uint32_t)__popc(in);
      if (in != FULL) break;
    }
    return n ? P.inter_cum[ioff + n - 1] : 0ull;
  };
  // number of active roots: the prefix of [lo, ns) with maxf <= L, 32 probes a step
  auto active = [&](uint32_t lo, int L) -> uint32_t {
    uint32_t hi = ns;  // roots below lo are active, roots from hi on are not
    while (lo < hi) {
      const uint32_t step = (hi - lo + 31) / 32, at = lo + (uint32_t)lane * step;
      const unsigned in = __ballot_sync(FULL, at < hi && P.sub_maxf[base + at] <= L);
      if (!in) break;  // root lo is not active
      const uint32_t last = lo + (31u - (uint32_t)__clz(in)) * step;  // active
      hi = min(hi, last + step);
      lo = last + 1;
    }
    return lo;
  };
  int L = r & 1 ? lim1 : lim0;
  {
    const unsigned long long in = interior(L);
    if (lane == 0) atomicAdd(&P.iter_nodes[(size_t)i * kMaxIters + r], in);
  }
  if (pair) {
    // iterations r and r + 1 ran together and have both finished: r's goal
    // decides first (r + 1's counts are then never read)
    const bool stop = (r & 1 ? flag1 : flag0) != 0u || goal <= L;
    if (stop || r + 1 >= kMaxIters) {
      if (lane == 0) {
        P.inst_final[i] = r;
        P.inst_fin_ns[i] = globaltimer();
        if (!stop) P.inst_status[i] = SP_ERR_LIMIT;
      }
      return;
    }
    ++r;
    L += 2;
    const unsigned long long in = interior(L);
    if (lane == 0) {
      P.inst_iter[i] = r;
      P.inst_pair[i] = 0u;
      atomicAdd(&P.iter_nodes[(size_t)i * kMaxIters + r], in);
    }
  }
  for (;;) {
    // every task of iteration r has finished: the goal flag is final
    const bool stop = (r & 1 ? flag1 : flag0) != 0u || goal <= L;
    if (stop || r + 1 >= kMaxIters) {
      if (lane == 0) {
        P.inst_final[i] = r;
        P.inst_fin_ns[i] = globaltimer();
        if (!stop) P.inst_status[i] = SP_ERR_LIMIT;
      }
      return;
    }
    ++r;
    L += 2;
    const uint32_t na = active(0, L);
    if (lane == 0) {
      P.inst_iter[i] = r;
      const_cast<int32_t *>(P.inst_limit)[2 * i + (r & 1)] = L;
    }
    if (!na) {
      const unsigned long long in = interior(L);
      if (lane == 0) atomicAdd(&P.iter_nodes[(size_t)i * kMaxIters + r], in);
      continue;
    }
    // loads of iteration r - 1 (summed by atomics in L2: read past L1); the
    // prediction of root q's next load is that times the root's own predicted
    // growth (learned balancer; otherwise the instance's, common to all)
    const unsigned long long *ld = P.sub_loads + (size_t)((r - 1) & 1) * P.n_subs + base;
    unsigned long long *nx = P.sub_loads + (size_t)(r & 1) * P.n_subs + base;
    auto pred_load = [&](uint32_t q, unsigned long long load) -> float {
      float lq = (float)load;
      if (P.sub_growth && load) {
        const int j = min(kGrowthSlacks - 1, max(0, (L - 2 - P.sub_maxf[base + q]) >> 1));
        lq *= exp2f((float)P.sub_growth[(size_t)(base + q) * kGrowthSlacks + j] * (1.0f / 16.0f));
      }
      return lq;
    };
    // longest first: bucket = binary exponent of the prediction (0: no load)
    auto bucket = [](float lq) -> int {
      return lq >= 1.0f ? min(31, (int)((__float_as_uint(lq) >> 23) & 0xFFu) - 126) : 0;
    };
    hist[lane] = 0;
    __syncwarp();
    unsigned long long tot = 0;
    float ptot = 0.f;
    for (uint32_t q0 = 0; q0 < na; q0 += 256) {
      unsigned long long v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t q = q0 + 32 * u + lane;
        v[u] = q < na ? __ldcg(ld + q) : 0ull;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t q = q0 + 32 * u + lane;
        if (q >= na) continue;
        tot += v[u];
        const float lq = pred_load(q, v[u]);
        ptot += lq;
        atomicAdd(&hist[bucket(lq)], 1u);
      }
    }
    for (int o = 16; o; o >>= 1) {
      tot += __shfl_xor_sync(FULL, tot, o);
      ptot += __shfl_xor_sync(FULL, ptot, o);
    }
    // the next iteration's size: this one's times the instance's growth
    float grow = 6.0f;
    if (r >= 2) {
      const unsigned long long prev = __ldcg(&P.iter_nodes[(size_t)i * kMaxIters + (r - 2)]);
      if (prev) grow = fminf(30.0f, fmaxf(2.0f, (float)tot / (float)prev));
    }
    if (P.handback_nodes && (float)tot * grow >= (float)P.handback_nodes) {
      // a large iteration is next: the host round loop finishes this
      // instance (its loads of iteration r - 1 stay in `ld`)
      if (lane == 0) {
        P.inst_final[i] = r - 1;
        P.inst_fin_ns[i] = globaltimer();
        P.inst_status[i] = kStatusHandback;
      }
      return;
    }
    const float avg = ptot / (float)na;
    for (uint32_t q = lane; q < ns; q += 32) nx[q] = 0;
    __syncwarp();
    const uint32_t c = hist[lane];
    uint32_t suf = c;  // roots in buckets >= lane
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_down_sync(FULL, suf, o);
      if (lane + o < 32) suf += v;
    }
    hist[lane] = suf - c;  // first position of bucket `lane`
    __syncwarp();
    // iteration r + 1 goes out with r when it is predicted small: the two
    // run together and the instance advances once both have finished, so a
    // chain of small iterations is not paced by one iteration at a time
    uint32_t na2 = 0;
    if (P.pair_nodes && r + 2 < kMaxIters && (float)tot * grow * grow < (float)P.pair_nodes) na2 = active(na, L + 2);
    // the roots in order, each with its split: root q | levels << 26
    const float piece = avg * (float)SP_MULTI_PIECE;
    for (uint32_t q0 = 0; q0 < na; q0 += 256) {
      unsigned long long v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t q = q0 + 32 * u + lane;
        v[u] = q < na ? __ldcg(ld + q) : 0ull;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t q = q0 + 32 * u + lane;
        if (q >= na) continue;
        const float lq = pred_load(q, v[u]);
        const uint32_t at = atomicAdd(&hist[bucket(lq)], 1u);
        int kk = 0;
        if (P.static_split && piece > 0.f && lq > 2.0f * piece) {
          // static split from the loads just measured: a root with x pieces'
          // load goes out as a split task of about log(x)/log(2.4) levels (the
          // reference cuts it into ceil(load/avg) pieces,
          // src/24puzzle_block_parallel_with_pdb.cu:839-897)
          kk = (int)ceilf(__log2f(lq / piece) * (1.0f / 1.2630344f));
          kk = max(0, min(kk, min(10, L - (int)P.subs[base + q].g - 1)));
        }
        P.order[base + at] = q | (uint32_t)kk << 26;
      }
    }
    if (na2) {
      unsigned long long *lz = P.sub_loads + (size_t)((r + 1) & 1) * P.n_subs + base;
      for (uint32_t q = lane; q < ns; q += 32) lz[q] = 0;
      if (lane == 0) {
        const_cast<int32_t *>(P.inst_limit)[2 * i + ((r + 1) & 1)] = L + 2;
        P.inst_pair[i] = 1u;
      }
    }
    __threadfence();
    __syncwarp();
    // the whole iteration (pair) is outstanding before its first task is visible
    const uint32_t nb = (na + kBulk - 1) / kBulk, nb2 = (na2 + kBulk - 1) / kBulk;
    uint32_t t0 = 0;
    if (lane == 0) {
      atomicAdd(&P.inst_out[i], na + na2);
      atomicAdd(&ctl->outstanding, na + na2);
      __threadfence();
      t0 = atomicAdd(&ctl->tail, nb + nb2);
    }
    t0 = __shfl_sync(FULL, t0, 0);
    __syncwarp();  // orders lane 0's counts before the other lanes' publications, which the shuffle does not
    for (uint32_t b = lane; b < nb + nb2; b += 32) {
      const bool second = b >= nb;
      const uint32_t q0 = (second ? b - nb : b) * kBulk, left = (second ? na2 : na) - q0;
      publish_root(P, t0 + b, base + q0, min(kBulk, left), second ? 0u : 1u,
                   kBulkFlag | (uint32_t)((second ? r + 1 : r) & 1) << 6);
    }
    __syncwarp();
    return;
  }
}

// Most lanes of a warp that donate in one pass of its loop (8 / 16 / 32: one
// random 15-puzzle 1.87 / 1.81 / 1.81 ms, 100 of them 17.84 / 17.71 / 17.76, a
// walk of 40 moves 0.78 / 0.75 / 0.75).
#ifndef SP_MAX_DONORS
#define SP_MAX_DONORS 16
#endif

// Longest sleep of a warp with no lane searching between pool polls (ns): a
// new iteration waits for it, other warps lose issue slots to the polls (2048 /
// 4096 / 16384: one random 15-puzzle 1.93 / 1.81 / 2.12 ms, 100 of them 17.90 /
// 17.72 / 18.75, 50 24-puzzles 45.2 / 45.1 / 45.9, a walk of 40 moves 0.75 / 0.75
// / 0.97).
#ifndef SP_MAX_BACKOFF_NS
#define SP_MAX_BACKOFF_NS 4096
#endif

// Resident threads per SM that the search kernels are compiled for, and the
// shared memory that these may take together.  The PDB search is bound by its
// table reads in flight: a read that misses L1 holds an L1 line until L2
// answers, so the part of the SM's 256 KB that is left to L1 limits them, and
// more warps pay only with a larger L1.  A round's kernel therefore is one
// block per SM: the move tables are there once instead of three or four times,
// and 164 KB of shared memory, 92 KB of L1, hold as many threads and about as
// many shared levels as 192 KB did in blocks of 256 (4096 15-puzzles: 100 /
// 132 / 164 / 196 KB 207 / 183 / 156 / 161 ms, blocks of 256 166 ms and at 228
// KB 260; 16384 24-puzzle roots 78.6 / 74.6 / 63.7 / 67.9, blocks of 256
// 68.2).  Threads, 15-puzzle: 768 / 896 / 1024 166 / 157 / 156 ms;
// 24-puzzle, whose rows are longer, so that more threads leave it fewer shared
// levels: 640 / 768 / 896 / 1024 65.3 / 63.8 / 70.3 / 72.7.
// Blocks of 128 threads, and of 256 in a named number per SM, stay for a caller
// that asks for them.  Manhattan reads no tables and is bound by issue and
// shared memory's latency: 1024 threads (blocks of 256, 768 an SM / one of 768
// / 896 / 1024: 2048 24-puzzle roots 11.25 / 11.08 / 10.31 / 10.00 ms, 100
// 15-puzzle walks 9.47 / 9.35 / 9.03 / 9.10).
// The device loop is bound by its chains of small iterations, not by reads in
// flight, and would spill 188 bytes at 64 registers: 768 threads (100 random
// 15-puzzles 17.2 -> 17.0 ms).
constexpr int big_block(int w, bool pdb) { return pdb && w == 5 ? 768 : 1024; }
constexpr int shared_per_sm(int block) { return (block > 256 ? 164 : 192) * 1024; }
constexpr int blocks_on_sm(int w, bool pdb, bool multi, int block) {
  return block > 256 ? 1 : (pdb && w == 4 && !multi ? 1024 : 768) / block;
}

// What a lane keeps in shared memory: 32-bit words, one column per lane
// ([row][thread]), so that a lane only ever touches its own bank whatever
// cell, pattern or level it indexes (a byte of a word included).
//   board   4 cells to a word, a byte each; the blank's own byte is stale
//   index   PDB: per pattern its table index with the table's base in it
//           (width 4: base in bits 20-21 and the table value in bits 24-31;
//           width 5: base in bit 28, the values as bytes of two more words)
//   cold    data of rare events
//   level   per level of the walk a byte with the moves still untried there
//           (bits 0-3), the reverse of the move taken (bits 4-5) and whether
//           it made h larger (bit 6, rounds alone) and, for
//           the PDB, a byte in each of two more planes: the regular and the
//           reflected table value that move overwrote; PDB levels beyond the
//           shared ones are in local memory
// The level bytes hold what an undo needs, so it neither recomputes the
// move mask nor reads a table, and donating a level is clearing its mask.
constexpr uint32_t kHarder = 64u;
template <int W, bool PDB, int BLOCK, int WORDS, bool MULTI>
struct LaneRows {
  static constexpr int N = W * W;
  static constexpr int kMaxLev = WORDS * 16;
  static constexpr int kPat = W == 4 ? 3 : 4;
  static constexpr int kBoard = 0;
  static constexpr int kIdx = kBoard + (N + 3) / 4;
  static constexpr int kVal = kIdx + (PDB ? 2 * kPat : 0);
  static constexpr int kCold = kVal + (PDB && W == 5 ? 2 : 0);
  static constexpr int kSub = kCold, kSplit = kCold + 1, kDebtAt = kCold + 2, kDebtSub = kCold + 3;
  static constexpr int kInst = MULTI ? kCold + 4 : kSub, kDone = MULTI ? kCold + 5 : kSub;  // device loop alone
  static constexpr int kLevel = kCold + (MULTI ? 6 : 4);
  // move tables of the block (bytes), pool cache and publication buckets
  static constexpr int kMoveTable = PDB ? (W == 4 ? 8 * 4 * N * N : 8 * N * N + 4 * N) : 4 * N * N;
  static constexpr int kFixed = kMoveTable + 64 + (MULTI ? BLOCK * 4 : 4) + BLOCK / 32 * 64;
  // shared levels: what fits beside the rest (1 KB is reserved per block)
  static constexpr int kBudget = shared_per_sm(BLOCK) / blocks_on_sm(W, PDB, MULTI, BLOCK) - 1024;
  static constexpr int kFit = (kBudget - kFixed) / (4 * BLOCK) - kLevel;
  static constexpr int kShared = PDB && kFit / 3 * 4 < kMaxLev ? kFit / 3 * 4 : kMaxLev;
  static constexpr int kDeep = kMaxLev - kShared;
  static constexpr int kPlane = kShared / 4;  // rows of one plane of level bytes
  static constexpr int kRows = kLevel + (PDB ? 3 : 1) * kPlane;
};

// What a warp keeps in shared memory: its statistics and, for its idle spells,
// the pool state it last saw.
struct WarpState {
  unsigned long long steps, slots, idle, begin, last_change;
  uint32_t last_out, last_tail, last_hb, beat, backoff, pad;
};
static_assert(sizeof(WarpState) == 64, "WarpState layout");

template <int W, bool PDB, int BLOCK, int WORDS, bool MULTI>
__device__ __forceinline__ void search_round(const RoundParams &P) {
  using R = LaneRows<W, PDB, BLOCK, WORDS, MULTI>;
  constexpr int N = W * W;
  constexpr unsigned FULL = 0xffffffffu;
  // One entry per (tile, cell it slides from, blank's move): what the step
  // needs of a move in one shared read.
  //   PDB, width 4: per partition the pattern-index change << 8 | pattern; the
  //     regular one also holds the child's move mask (legal, not the reverse)
  //     in bits 4-7
  //   PDB, width 5: the change is the difference of two (tile, cell) codes
  //     (a full table would take 20 KB), the pattern in their top 4 bits
  //   Manhattan: the child's move mask, bit 4 set when the tile gets farther
  __shared__ uint2 s_mv[PDB ? (W == 4 ? 4 * N * N : N * N) : 1];
  __shared__ uint8_t s_rem[PDB && W == 5 ? 4 * N : 4];
  __shared__ uint8_t s_md[PDB ? 4 : 4 * N * N];
  __shared__ uint32_t s_lane[R::kRows][BLOCK];
  // multi-iteration mode: per-warp bucket counts of the longest-first publication
  __shared__ uint32_t s_hist[MULTI ? BLOCK / 32 : 1][32];
  // block-wide cache of the pool state: at most one global poll per block per poll_ns
  __shared__ uint32_t s_pool[5];  // head, tail, error, outstanding, heartbeat
  __shared__ unsigned long long s_pool_t;
  __shared__ WarpState s_warp[BLOCK / 32];
  __shared__ uint32_t s_stat[5];  // donation counters: tries, slot not free, hungry polls, tasks done, donor found
  if (threadIdx.x < 5) s_stat[threadIdx.x] = 0;
  if ((threadIdx.x & 31) == 0) {
    s_warp[threadIdx.x >> 5] = WarpState{};
    s_warp[threadIdx.x >> 5].begin = (unsigned long long)clock64();
    s_warp[threadIdx.x >> 5].backoff = 256;
  }
  if (threadIdx.x == 0) {
    s_pool[0] = s_pool[1] = s_pool[2] = s_pool[4] = 0;
    s_pool[3] = 1;
    s_pool_t = 0;
    if (MULTI) atomicMin(P.t_begin_ns, globaltimer());
  }

  const HeurTables *ht = P.ht;
  auto child_moves = [](int cell, int d) -> uint32_t { return legal_moves(W, cell) & ~(1u << (3 - d)); };
  if (PDB && W == 5) {
    for (int i = threadIdx.x; i < N * N; i += BLOCK) {
      const int t = i / N;
      s_mv[i] = make_uint2(ht->code[0][i] | (uint32_t)ht->pat[0][t] << 28,
                           ht->code[1][i] | (uint32_t)ht->pat[1][t] << 28);
    }
    for (int i = threadIdx.x; i < 4 * N; i += BLOCK) s_rem[i] = (uint8_t)child_moves(i / 4, i % 4);
  } else {
    for (int i = threadIdx.x; i < 4 * N * N; i += BLOCK) {
      const int d = i % 4, c = (i / 4) % N, t = i / (4 * N);
      const int to = c - move_delta(W, d);
      const bool legal = to >= 0 && to < N && ((legal_moves(W, to) >> d) & 1u);
      if (PDB) {
        uint2 v = make_uint2(0, 0);
        if (legal && t) {
          v.x = (ht->code[0][t * N + to] - ht->code[0][t * N + c]) << 8 | child_moves(c, d) << 4 | ht->pat[0][t];
          v.y = (ht->code[1][t * N + to] - ht->code[1][t * N + c]) << 8 | ht->pat[1][t];
        }
        s_mv[i] = v;
      } else {
        s_md[i] = (uint8_t)(child_moves(c, d) | (legal && ht->mdd[(d * N + c) * N + t] > 0 ? 16u : 0u));
      }
    }
  }
  __syncthreads();

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  uint32_t *const me = &s_lane[0][tid];                      // row r of the lane: me[r * BLOCK]
  uint8_t *const mb = reinterpret_cast<uint8_t *>(me);
  // local memory: the task's moves above its start (its pool slot is freed),
  // the board it started from (in a task's layout: cells, blank), and the
  // levels beyond the shared ones, their three bytes in a word
  uint32_t prefix[kPathWords], start_board[7], deep[R::kDeep > 0 ? R::kDeep : 1] = {0};
  WarpState &ws = s_warp[tid >> 5];
  uint32_t *const s_cold0 = s_lane[R::kDone], *const s_cold1 = s_lane[R::kDebtAt],
           *const s_cold2 = s_lane[R::kDebtSub];
  // the task's SubRoot; its instance (multi-iteration mode: bit 31 = the
  // parity of the task's iteration); its split levels (a split task hands
  // every node at relative depth 1 to the pool)
  uint32_t &sub = s_lane[R::kSub][tid], &cur_inst = s_lane[R::kInst][tid], &splitk = s_lane[R::kSplit][tid];
  PoolCtl *ctl = P.ctl;

  // ---- lane state -------------------------------------------------------
  int state = 0;  // 0 idle, 1 holds a claimed slot, 2 searching
  uint32_t slot = 0;
  int blank = 0, k = 0;
  uint32_t boff = 0;             // board_off(blank)
  uint32_t rem = 0;              // moves still untried at the current node
  int hr = 0, hf = 0;            // h of the two partitions (Manhattan: hr alone)
  int budget = 0;                // a child of level k is entered when its h <= budget - k
  int krare = 0;                 // entering a child of a level from here on needs a second look: the
                                 // first level of a split task, levels beyond the shared ones or the
                                 // last that the lane's stack and path can hold
  int plen = 0;
  int lo = 0;                    // donation: no level below lo has untried moves
  int lo_slack = 0;              // the limit less f at level lo (kHarder)
  uint32_t cnt = 0;              // generated nodes not yet added to the task's counters
  // Rare per-lane events, flags in a register and their data in shared memory:
  //  * kAdvance: the lane finished an instance's iteration; the warp advances
  //    that instance (s_cold0) at the top of its next loop;
  //  * kDebt: a reserved pool index (s_cold1) whose ring slot did not free
  //    in time is owed: the lane kept the work and publishes a null task (no
  //    moves, SubRoot s_cold2) there later, so no index stays unpublished.
  //  * kBulkHeld: the lane claimed a bulk (its first place and its header in
  //    the lane's words for a task's SubRoot and split).
  constexpr uint32_t kAdvance = 1u, kDebt = 2u, kBulkHeld = 4u;
  uint32_t events = 0;

  auto board_off = [&](int c) -> uint32_t {
    return (uint32_t)c + (uint32_t)(c >> 2) * (4u * BLOCK - 4u) + 4u * BLOCK * R::kBoard;
  };
  auto level_off = [&](int j) -> uint32_t {
    return (uint32_t)j + (uint32_t)(j >> 2) * (4u * BLOCK - 4u) + 4u * BLOCK * R::kLevel;
  };
  auto level_get = [&](int j) -> uint32_t {
    return R::kDeep > 0 && j >= R::kShared ? deep[j - R::kShared] & 0xFFu : mb[level_off(j)];
  };
  auto level_cut = [&](int j) {  // no move of level j is left to try
    if (R::kDeep > 0 && j >= R::kShared) deep[j - R::kShared] &= ~15u;
    else mb[level_off(j)] &= (uint8_t)~15u;
  };
  // The lane's first `len` moves below its SubRoot -- the task's prefix, then
  // its walk's first len - plen levels -- as words handed to put(index, word).
  // The levels come four to a shared word: the complement of bits 4-5 of
  // each byte, squeezed to 8 bits.
  auto write_path = [&](int len, auto put) {
    int wi = 0;
    for (; 16 * (wi + 1) <= plen; ++wi) put(wi, prefix[wi]);
    const int lev = len - plen;
    uint32_t acc = 0;
    int at = plen & 15;  // moves in acc
    if (at) acc = prefix[wi] & ((1u << (2 * at)) - 1u);
    for (int j = 0; j < lev; j += 4) {
      uint32_t x = 0;
      if (R::kDeep > 0 && j >= R::kShared) {
        for (int q = j; q < min(j + 4, R::kMaxLev); ++q) x |= (deep[q - R::kShared] & 0xFFu) << (8 * (q - j));
      } else {
        x = me[(R::kLevel + (j >> 2)) * BLOCK];
      }
      x = ~(x >> 4) & 0x03030303u;
      x = (x | x >> 6 | x >> 12 | x >> 18) & 0xFFu;
      const int n = min(4, lev - j);
      if (n < 4) x &= (1u << (2 * n)) - 1u;
      acc |= x << (2 * at);
      at += n;
      if (at >= 16) {
        put(wi++, acc);
        at -= 16;
        acc = at ? x >> (2 * (n - at)) : 0u;
      }
    }
    if (at) put(wi, acc);
  };
  // Publish, at reserved and free pool index t, the lane's node at `level` of
  // its walk, restricted to the moves in `mask`.
  auto publish_node = [&](uint32_t t, int level, uint32_t mask, uint32_t flags) {
    uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint8_t *const wb = reinterpret_cast<uint8_t *>(w);
    constexpr int kWords = (N + 3) / 4;
    int at;
    if (level == k) {  // the current board
      for (int q = 0; q < kWords; ++q) w[q] = me[(R::kBoard + q) * BLOCK];
      at = blank;
    } else {  // from the task's start (a shallow level)
      for (int q = 0; q < kWords; ++q) w[q] = start_board[q];
      at = (int)(start_board[6] >> 8 & 0xFFu);
      for (int j = 0; j < level; ++j) {
        const int from = at + step_delta<W>(3u - (level_get(j) >> 4 & 3u));
        wb[at] = wb[from];
        at = from;
      }
    }
    const int len = plen + level;
    wb[25] = (uint8_t)at;
    wb[26] = 0;
    wb[27] = (uint8_t)mask;
    w[7] = sub;
    Task *D = &P.tasks[t & (P.cap - 1u)];
    uint4 *out = reinterpret_cast<uint4 *>(D);
    out[0] = make_uint4(w[0], w[1], w[2], w[3]);
    out[1] = make_uint4(w[4], w[5], w[6], w[7]);
    *reinterpret_cast<uint32_t *>(out + 2) =
        (uint32_t)len | flags << 8 | (uint32_t)min(budget - level, kMaxBudget) << 16;
    write_path(len, [&](int wi, uint32_t v) { D->path[wi] = v; });
    st_release(&P.seq[t & (P.cap - 1u)], t + 1u);
  };
  auto lookup = [&](uint32_t off) -> uint32_t { return __ldg(P.pdb + off); };
  // h of the lane's board (its blank byte 0) from nothing: pattern indices
  // and table values too
  auto full_h = [&]() -> int {
    if (PDB) {
      uint64_t ra = 0, rb = 0, fa = 0, fb = 0;
#pragma unroll 4
      for (int c = 0; c < N; ++c) {
        const uint32_t t = mb[4 * BLOCK * (R::kBoard + c / 4) + c % 4];
        const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(ht->sum) + (t * N + c) * (W == 4 ? 1u : 2u);
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
      }
      hr = hf = 0;
#pragma unroll
      for (int p = 0; p < R::kPat; ++p) {
        const uint32_t base = W == 4 ? (uint32_t)p << 20 : (p ? 1u << 28 : 0u);
        const uint32_t a = sum_field<W>(ra, rb, p) | base, b = sum_field<W>(fa, fb, p) | base;
        const uint32_t va = lookup(a), vb = lookup(b);
        me[(R::kIdx + p) * BLOCK] = W == 4 ? a | va << 24 : a;
        me[(R::kIdx + R::kPat + p) * BLOCK] = W == 4 ? b | vb << 24 : b;
        if (W == 5) {
          mb[R::kVal * 4 * BLOCK + p] = (uint8_t)va;
          mb[(R::kVal + 1) * 4 * BLOCK + p] = (uint8_t)vb;
        }
        hr += (int)va;
        hf += (int)vb;
      }
      return max(hr, hf);
    } else {
      hr = 0;
#pragma unroll
      for (int c = 0; c < N; ++c) {
        const int t = mb[4 * BLOCK * (R::kBoard + c / 4) + c % 4];
        if (t) hr += abs(c / W - t / W) + abs(c % W - t % W);
      }
      return hr;
    }
  };
  auto set_error = [&](int code, uint32_t info) {
    if (atomicCAS(&ctl->error, 0, code) == 0) ctl->err_info[0] = info;
  };
  // Wait a bounded time for the ring slot of reserved pool index t (normally
  // free at once: its previous occupant, index t - cap, was claimed long
  // before).
  auto slot_free = [&](uint32_t t, int spins) -> bool {
    for (int spin = 0; spin < spins; ++spin) {
      if (ld_acquire(&P.seq[t & (P.cap - 1u)]) == t) return true;
      __nanosleep(64);
    }
    return false;
  };
  // Add the lane's count to the task's counters.
  auto flush_count = [&]() {
    if (!cnt) return;
    if (MULTI) {
      // the instance stays in its current iteration while the task is
      // outstanding; the task's own is that one or, in a pair, the next
      const uint32_t ci = cur_inst & 0x7FFFFFFFu, tp = cur_inst >> 31;
      const int cur_iter = ld_volatile(&P.inst_iter[ci]);
      const int task_iter = cur_iter + (((uint32_t)cur_iter & 1u) != tp ? 1 : 0);
      atomicAdd(&P.iter_nodes[(size_t)ci * kMaxIters + task_iter], (unsigned long long)cnt);
      atomicAdd(&P.sub_loads[(size_t)tp * P.n_subs + sub], (unsigned long long)cnt);
    } else {
      atomicAdd(&P.sub_nodes[sub], (unsigned long long)cnt);
    }
    cnt = 0;
  };
  auto finish_task = [&]() {
    atomicAdd(&s_stat[3], 1u);
    state = 0;
    flush_count();
    if (MULTI) {
      __threadfence();
      // the last task of the iteration: the warp advances the instance at the
      // top of its next loop, and only then does this task leave
      // `outstanding`, so that never reads 0 while work is still to come
      if (atomicSub(&P.inst_out[cur_inst & 0x7FFFFFFFu], 1u) == 1u) {
        events |= kAdvance;
        s_cold0[tid] = cur_inst & 0x7FFFFFFFu;
        return;
      }
      __threadfence();
    }
    // one launch, one threshold: the counts are read after the kernel, so no
    // fence; the tasks this one gave away were counted before, by this lane or
    // ahead of the warp barrier in the donation below
    atomicSub(&ctl->outstanding, 1u);
  };
  // Copy the claimed record out of its ring slot, free the slot for the
  // producer of index slot + cap, and start the task.  A task below its root
  // brings its board: its claimant waits for one read of the record instead
  // of the record, the root and a replay of the path (the hungry phases hand
  // out tasks of a few hundred nodes).  Returns whether the lane searches.
  auto take_task = [&]() -> bool {
    const uint32_t s = slot & (P.cap - 1u);
    const uint4 *T = reinterpret_cast<const uint4 *>(&P.tasks[s]);
    uint4 b0 = __ldcg(T), b1 = __ldcg(T + 1);
    const uint32_t meta = __ldcg(reinterpret_cast<const uint32_t *>(T + 2));  // plen, flags, budget
    sub = b1.w;
    plen = (int)(meta & 0xFFu);
    const uint32_t flags = (meta >> 8) & 0xFFu, mask = b1.z >> 24;
    if (MULTI && (flags & kBulkFlag)) {  // a bulk: the warp publishes its roots
      st_release(&P.seq[s], slot + P.cap);
      state = 0;
      events |= kBulkHeld;
      splitk = (uint32_t)plen | mask << 8 | flags << 16;
      return false;
    }
    const uint32_t *path = P.tasks[s].path;
    const int moves = min(plen, kMaxPath);  // a record with more is refused below
    for (int wi = 0; 16 * wi < moves; ++wi) prefix[wi] = __ldcg(path + wi);
    st_release(&P.seq[s], slot + P.cap);  // the copies above complete before the slot is reused
    splitk = flags & 0x3Fu;
    const uint32_t parity = flags >> 6 & 1u;
    cnt = 0;
    k = 0;
    lo = 0;
    int pre = -1;
    if (plen == 0) {  // a root as it is
      const uint4 *rec = reinterpret_cast<const uint4 *>(&P.subs[sub]);
      b0 = rec[0];
      b1 = rec[1];
      if (MULTI) cur_inst = b1.w | parity << 31;
      // below 0 no root is entered, whatever its g and h; a caller's limit of
      // INT_MIN less g would wrap
      const int limit = max(MULTI ? ld_volatile(&P.inst_limit[2 * b1.w + parity]) : P.inst_limit[b1.w], -1);
      budget = limit - (int)((b1.z >> 16) & 0xFFu) - 1;
      pre = (b1.z >> 24) == kNoPre ? -1 : (int)(b1.z >> 24);
    } else {
      if (MULTI) cur_inst = P.subs[sub].inst | parity << 31;
      budget = (int)meta >> 16;
    }
    blank = (int)((b1.z >> 8) & 0xFFu);
    if (!mask) return false;  // a null task
    const uint32_t word[7] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z};
    if (!record_ok(W, word, plen)) {  // corrupt: never index out of range
      set_error(SP_ERR_ARG, 0x100u);
      return false;
    }
    me[(R::kBoard + 0) * BLOCK] = start_board[0] = b0.x;
    me[(R::kBoard + 1) * BLOCK] = start_board[1] = b0.y;
    me[(R::kBoard + 2) * BLOCK] = start_board[2] = b0.z;
    me[(R::kBoard + 3) * BLOCK] = start_board[3] = b0.w;
    if (W == 5) {
      me[(R::kBoard + 4) * BLOCK] = start_board[4] = b1.x;
      me[(R::kBoard + 5) * BLOCK] = start_board[5] = b1.y;
      me[(R::kBoard + 6) * BLOCK] = b1.z;  // cell 24, then the record's blank
    }
    start_board[6] = b1.z;
    boff = board_off(blank);
    mb[boff] = 0;
    const int h = full_h();
    rem = step_legal<W>(blank) & mask;
    if (pre >= 0) rem &= ~(1u << (3 - pre));
    krare = splitk ? 0 : min(min(R::kShared, R::kMaxLev - 1), kMaxPath - plen);
    lo_slack = budget + 1 - h;
    return h <= budget + 1;
  };
  auto record_goal = [&]() {
    const SubRoot *root = &P.subs[sub];
    const uint32_t si = root->inst;
    Solution *S = &P.sol[MULTI ? 2 * si + (cur_inst >> 31) : si];
    const int len = plen + k;
    // shortest goal depth over all lanes; from the root's depth, which may be
    // up to 255, so that no record between holds a depth in a byte
    atomicMax(&S->best, 0xFFFFFFFFu - ((uint32_t)root->g + (uint32_t)len));
    if (atomicCAS(&S->flag, 0u, 1u) == 0u) {
      S->sub = sub;
      S->len = (uint32_t)len;
      write_path(len, [&](int wi, uint32_t w) { S->path[wi] = w; });
      __threadfence();
    }
  };

  // One edge of the depth-first search: generate the next child of the
  // current node, or undo the move into the current node.  Both slide one
  // tile into the blank's cell and update the pattern index the same way, so
  // they share one code path (lanes of a warp at different points of their
  // walks stay converged); only the child's table lookups, the f-test and
  // the level's word differ.
  // It is written with selects and reads that both kinds of lane make, one
  // branch for what is entered and one for the rare cases: branches on the kind
  // made the compiler give each kind a copy of the shared code (9 lanes per
  // instruction; 18 with warp syncs in between, 19 and a tenth fewer
  // instructions this way).
  // go on; task exhausted; child to hand to the pool; not searching
  enum { kStepOn, kStepDone, kStepEmit, kStepIdle };
  auto step = [&]() -> int {
    const bool gen = rem != 0;
    const int lev = gen ? k : k - 1;  // the level whose bytes this step writes or reads
    const uint32_t at = level_off(R::kDeep > 0 ? min(lev, R::kShared - 1) : lev);
    // an undo: the level's moves, and the table values it had before the
    // descent (a generating lane reads too, and drops it)
    uint32_t e = mb[at], vr = 0, vf = 0;
    if (PDB) {
      vr = mb[at + 4u * BLOCK * R::kPlane];
      vf = mb[at + 8u * BLOCK * R::kPlane];
    }
    if (R::kDeep > 0 && lev >= R::kShared) {
      const uint32_t w = deep[lev - R::kShared];
      e = w & 0xFFu;
      vr = (w >> 8) & 0xFFu;
      vf = w >> 16 & 0xFFu;
    }
    const uint32_t dm = gen ? first_move(rem) : e >> 4 & 3u;  // the blank's move this step
    rem &= rem - 1u;
    cnt += gen;
    const int from = blank + step_delta<W>(dm);
    const uint32_t foff = board_off(from);
    const uint32_t t = mb[foff];  // slides from `from` into the blank's cell
    uint32_t qr = 0, qf = 0, nr = 0, nf = 0, oldr = 0, oldf = 0, child;
    int nhr, nhf = 0;
    if (PDB) {
      if (W == 4) {
        const uint2 m = s_mv[(t * N + (uint32_t)from) * 4u + dm];
        qr = m.x & 3u;
        qf = m.y & 3u;
        const uint32_t wr = me[(R::kIdx + qr) * BLOCK], wf = me[(R::kIdx + R::kPat + qf) * BLOCK];
        nr = wr + (uint32_t)((int32_t)m.x >> 8);
        nf = wf + (uint32_t)((int32_t)m.y >> 8);
        oldr = wr >> 24;
        oldf = wf >> 24;
        child = (m.x >> 4) & 15u;
      } else {
        const uint2 ma = s_mv[t * N + (uint32_t)blank], mf = s_mv[t * N + (uint32_t)from];
        qr = ma.x >> 28;
        qf = ma.y >> 28;
        nr = me[(R::kIdx + qr) * BLOCK] + (ma.x - mf.x);
        nf = me[(R::kIdx + R::kPat + qf) * BLOCK] + (ma.y - mf.y);
        oldr = mb[R::kVal * 4 * BLOCK + qr];
        oldf = mb[(R::kVal + 1) * 4 * BLOCK + qf];
        child = s_rem[(uint32_t)from * 4u + dm];
      }
      // undoing lanes read entry 0 of the first table: one sector for all of
      // them, and the warp stays on one path
      const uint32_t tr = lookup(!gen ? 0u : W == 4 ? nr & 0x3FFFFFu : nr);
      const uint32_t tf = lookup(!gen ? 0u : W == 4 ? nf & 0x3FFFFFu : nf);
      vr = gen ? tr : vr;
      vf = gen ? tf : vf;
      nhr = hr + (int)(vr - oldr);
      nhf = hf + (int)(vf - oldf);
    } else {
      const uint32_t m = s_md[(t * N + (uint32_t)from) * 4u + dm];
      child = m & 15u;
      nhr = hr + (int)((m >> 3) & 2u) - 1;
    }
    const int nh = PDB ? max(nhr, nhf) : nhr, h0 = PDB ? max(hr, hf) : hr;
    int ev = kStepOn;
    if (!gen || nh <= budget - k) {  // else: generated, not entered
      if (PDB) {
        me[(R::kIdx + qr) * BLOCK] = W == 4 ? nr + ((vr - oldr) << 24) : nr;
        me[(R::kIdx + R::kPat + qf) * BLOCK] = W == 4 ? nf + ((vf - oldf) << 24) : nf;
        if (W == 5) {
          mb[R::kVal * 4 * BLOCK + qr] = (uint8_t)vr;
          mb[(R::kVal + 1) * 4 * BLOCK + qf] = (uint8_t)vf;
        }
        hf = nhf;
      }
      hr = nhr;
      mb[boff] = (uint8_t)t;
      boff = foff;
      blank = from;
      const uint32_t up = rem | (3u - dm) << 4 | (!MULTI && nh > h0 ? kHarder : 0u);
      if (gen && (R::kDeep == 0 || lev < R::kShared)) {
        mb[at] = (uint8_t)up;
        if (PDB) {
          mb[at + 4u * BLOCK * R::kPlane] = (uint8_t)oldr;
          mb[at + 8u * BLOCK * R::kPlane] = (uint8_t)oldf;
        }
      }
      rem = gen ? child : e & 15u;
      k = gen ? lev + 1 : lev;
      if (gen && (nh == 0 || lev >= krare)) {
        if (R::kDeep > 0 && lev >= R::kShared) deep[lev - R::kShared] = up | oldr << 8 | oldf << 16;
        const bool full = lev >= min(R::kMaxLev - 1, kMaxPath - plen);  // no room for a path that long
        if (nh == 0 && !full) record_goal();
        // split task with `splitk` levels left: this child (already counted
        // as generated) becomes a task of its own with one level fewer
        // (published outside the step loop), so a heavy root is split
        // breadth-first by many lanes; the lane then steps back
        if (splitk && lev == 0) ev = kStepEmit;
        if (full) {
          set_error(SP_ERR_STACK_OVERFLOW, (uint32_t)(plen + lev));
          ev = kStepDone;
        }
      }
    }
    return ev;
  };

  // Give the untried moves of the shallowest open level (slack >= min_slack)
  // to a waiting lane.  Returns the level donated, or -1.
  auto find_donation = [&](uint32_t &mask_out) -> int {
    // resume at the first level not yet seen exhausted (`lo`): a level only
    // loses untried moves during a task, so the walk never needs to look
    // below it again, and has nothing left when it has stepped back past it
    if (k < lo) return -1;
    int j = lo, found = -1;
    const int last = min(k, budget + 1 - P.min_slack);
    for (; j <= last; ++j) {
      const uint32_t e = j == k ? rem : level_get(j);
      if (e & 15u) {
        mask_out = e & 15u;
        found = j;
        break;
      }
      if (e & kHarder) lo_slack -= 2;
    }
    lo = min(j, k);
    return found;
  };

  for (;;) {
    const long long t_iter = clock64();
    // pending work of the previous loop: instance advances, then owed indices
    if (MULTI) {
      unsigned pend = __ballot_sync(FULL, events & kAdvance);
      while (pend) {
        // all lanes read the instance in s_cold0 and the loads and goals of the
        // tasks whose end the marked lane has seen, and write the s_hist that
        // the advance before used
        __threadfence();
        __syncwarp();
        const int src = __ffs(pend) - 1;
        pend &= pend - 1u;
        warp_advance(P, s_cold0[(tid & ~31) + src], s_hist[tid >> 5]);
        if (lane == src) {
          events &= ~kAdvance;
          __threadfence();
          atomicSub(&ctl->outstanding, 1u);
        }
      }
    }
    if ((events & kDebt) && ld_acquire(&P.seq[s_cold1[tid] & (P.cap - 1u)]) == s_cold1[tid]) {
      const uint32_t debt = s_cold1[tid];
      Task *D = &P.tasks[debt & (P.cap - 1u)];
      D->sub = s_cold2[tid];
      D->plen = 0;
      D->mask = 0;  // no first move: the claimant finishes it at once
      D->flags = 0;
      st_release(&P.seq[debt & (P.cap - 1u)], debt + 1u);
      events &= ~kDebt;
    }
    // 0. pool state from the block's cached copy (one global poll per block
    //    per poll_ns; a stale copy only delays, never corrupts, decisions:
    //    outstanding == 0 is final, tail and head only grow)
    uint32_t hd = 0, tl = 0, out = 0, hb = 0;
    int32_t err = 0;
    if (lane == 0) {
      volatile uint32_t *vp = (volatile uint32_t *)s_pool;
      const unsigned long long now = globaltimer();
      if (now - *(volatile unsigned long long *)&s_pool_t > P.poll_ns) {
        s_pool_t = now;
        vp[0] = ld_volatile(&ctl->head);
        vp[1] = ld_volatile(&ctl->tail);
        vp[2] = (uint32_t)ld_volatile(&ctl->error);
        vp[3] = ld_volatile(&ctl->outstanding);
        vp[4] = ld_volatile(&ctl->heartbeat);
      }
      hd = vp[0];
      tl = vp[1];
      err = (int32_t)vp[2];
      out = vp[3];
      hb = vp[4];
    }
    hd = __shfl_sync(FULL, hd, 0);
    tl = __shfl_sync(FULL, tl, 0);
    err = __shfl_sync(FULL, err, 0);
    out = __shfl_sync(FULL, out, 0);
    if (err) break;
    // 1. idle lanes claim pool indices, one atomic per warp
    const unsigned need = __ballot_sync(FULL, state == 0);
    if (need) {
      const int leader = __ffs(need) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(&ctl->head, (uint32_t)__popc(need));
      base = __shfl_sync(FULL, base, leader);
      if (state == 0) {
        slot = base + (uint32_t)__popc(need & ((1u << lane) - 1u));
        state = 1;
      }
    }
    // 2. a claimed index becomes a task once its producer published it; only
    //    indices already reserved (below the cached tail) are polled
    if (state == 1 && slot < tl && ld_acquire(&P.seq[slot & (P.cap - 1u)]) == slot + 1u) {
      if (take_task()) state = 2;
      else if (!MULTI || !(events & kBulkHeld)) finish_task();
    }
    if (MULTI) {
      unsigned held = __ballot_sync(FULL, events & kBulkHeld);
      const bool any = held != 0;
      __syncwarp();  // the holders' words are read by all lanes
      while (held) {
        const int src = (tid & ~31) + __ffs(held) - 1;
        held &= held - 1u;
        const uint32_t first = s_lane[R::kSub][src], hdr = s_lane[R::kSplit][src];
        const uint32_t n = hdr & 0xFFu;
        uint32_t t0 = 0;
        if (lane == 0) t0 = atomicAdd(&ctl->tail, n);
        t0 = __shfl_sync(FULL, t0, 0);
        if ((uint32_t)lane < n) {
          uint32_t root = first + (uint32_t)lane, kk = 0;
          if (hdr >> 8 & 0xFFu) {
            // the order is relative to the instance's first root
            const uint32_t e = __ldcg(&P.order[root]);
            root = P.inst_sub_base[P.subs[root].inst] + (e & 0x3FFFFFFu);
            kk = e >> 26;
          }
          publish_root(P, t0 + (uint32_t)lane, root, 0, 0xF, kk | (hdr >> 16 & 0x40u));
        }
        __syncwarp();
      }
      events &= ~kBulkHeld;
      if (any) continue;  // the holders claim again
    }
    // 3. nobody in the warp is searching: finished, failed or waiting
    const unsigned act = __ballot_sync(FULL, state == 2);
    if (!act) {
      if (out == 0) break;
      if (lane == 0) {
        const unsigned long long now = globaltimer();
        if (out != ws.last_out || tl != ws.last_tail || hb != ws.last_hb || ws.last_change == 0) {
          ws.last_out = out;
          ws.last_tail = tl;
          ws.last_hb = hb;
          ws.last_change = now;
        } else if (now - ws.last_change > P.timeout_ns) {
          set_error(SP_ERR_TIMEOUT, out);
        }
      }
      const unsigned backoff = ws.backoff;  // doubled up to SP_MAX_BACKOFF_NS
      __nanosleep(backoff);
      __syncwarp();
      if (lane == 0) {
        ws.backoff = min(backoff * 2u, (unsigned)SP_MAX_BACKOFF_NS);
        ws.idle += (unsigned long long)(clock64() - t_iter);
      }
      __syncwarp();
      continue;
    }
    if (lane == 0) {
      ws.backoff = 256;
      ws.last_change = 0;  // a new idle spell starts its own no-progress clock
      if ((++ws.beat & 127u) == 0u) atomicAdd(&ctl->heartbeat, 1u);
    }
    // 4. search
    // the warp steps together: every lane stays in the loop until none
    // searches, and the vote brings them back together
    int ev = state == 2 ? kStepOn : kStepIdle;
    uint32_t taken = 0;
    // A round's passes are a quarter longer than the device loop's, where the
    // next iteration waits for the last one's tasks (32 / 40 / 48 steps: 100
    // random 15-puzzles 17.4 / 16.9 / 16.9 ms, 2048 24-puzzle roots 11.8 / 11.3
    // / 11.2, 50 24-puzzles 12.7 / 12.9 / 12.9).
    // While as many lanes wait as are three quarters of 768 per SM (of a
    // round's 1024, 9 in 16), they are half as long: issue slots are free and
    // what counts is how fast work spreads.  Against other rules on the same
    // inputs, the other rule first, in ms:
    //   never in the device loop: one random 15-puzzle 1.54 and 1.46, 50
    //     24-puzzles 7.77 and 7.51, 100 Manhattan walks 8.78 and 8.80;
    //   in rounds of 1024 from three lanes in four on: one random 15-puzzle
    //     1.84 and 1.83, 100 of them 11.93 and 11.87, 4096 mixed ones 174.7 and
    //     174.1;
    //   from half of all lanes on: 24-puzzles 9.18 and 9.29, walks 7.97 and 7.80.
    int steps = MULTI ? P.steps : P.steps + P.steps / 4;
    if ((int32_t)(hd - tl) > (int32_t)(48u * P.spread)) steps = (P.steps + 1) / 2;
    for (int s = 0; s < steps; ++s) {
      const bool go = ev == kStepOn && (rem | (uint32_t)k) != 0u;  // else: nothing left of the task
      if (!__any_sync(FULL, go)) break;
      if (go) {
        ++taken;
        ev = step();
      }
    }
    if (ev == kStepOn && (rem | (uint32_t)k) == 0u) ev = kStepDone;
    taken = __reduce_add_sync(FULL, taken);
    if (lane == 0) {
      ws.slots += 32ull * (unsigned long long)steps;
      ws.steps += taken;
    }
    if (state == 2) {
      if (cnt >= (1u << 30)) flush_count();  // long before the 32-bit count wraps
      if (ev == kStepEmit) {
        // the split is advisory: with a debt outstanding or the ring half
        // full, the lane searches the subtree itself
        bool emitted = false;
        if (!(events & kDebt) && (int32_t)(tl - hd) <= (int32_t)(P.cap >> 1)) {
          atomicAdd(&ctl->outstanding, 1u);
          if (MULTI) atomicAdd(&P.inst_out[cur_inst & 0x7FFFFFFFu], 1u);  // the lane's own task keeps it >= 1
          const uint32_t t = atomicAdd(&ctl->tail, 1u);
          if (slot_free(t, 4096)) {
            publish_node(t, k, rem, (splitk - 1u) | (MULTI ? (cur_inst >> 31) << 6 : 0u));
            emitted = true;
          } else {
            atomicAdd(&s_stat[1], 1u);
            events |= kDebt;
            s_cold1[tid] = t;
            s_cold2[tid] = sub;
          }
        }
        if (emitted) rem = 0;
      }
      if (ev == kStepDone) finish_task();
    }
    // 5. donate while fewer than `reserve` tasks are queued (tail - head)
    if (P.donate && hd + P.reserve > tl) {
      uint32_t dmask = 0;
      int lev = (state == 2) ? find_donation(dmask) : -1;
      if (lev >= 0 && plen + lev > kMaxPath) lev = -1;  // prefix would not fit a record
      // donors: the lanes with about the largest parts, at most `allowed` of
      // them (more when the shortfall is large).  A part's size goes by its
      // node's slack and the moves left at it: two of slack are worth six moves.
      // In the device loop, where iterations are small and the next one waits
      // for their last task, it goes by the level in the task alone, which
      // spreads the newest tasks first.
      // Rounds, by level / moves left / 1, 2, 3 or 8 slack + moves left: 16384
      // 24-puzzle roots 84.5 / 71.1 / 71.3 / 70.1 / 69.9 / - ms, 2048 of them
      // by Manhattan 22.0 / 12.9 / 12.1 / 11.8 / 11.7 / 12.1, 100 random
      // 15-puzzles 19.1 / 18.3 / 17.5 / 17.4 / 17.3 / 18.8 (a task then holds
      // 40 % more nodes).  The device loop on 50 24-puzzles by level 2.3, by
      // moves left 2.9, by both 2.6.
      constexpr int kScoreSlack = 3;
      constexpr unsigned kNear = MULTI ? 1u : 4u;
      const unsigned key = lev < 0 ? 0xFFFFFFFFu
                           : MULTI ? (unsigned)lev
                                   : (1u << 24) - (unsigned)(kScoreSlack * min(lo_slack, 1 << 16) + min(budget, 1 << 16) - lev);
      const unsigned best = __reduce_min_sync(FULL, key);
      const uint32_t shortfall = hd + P.reserve - tl;
      const unsigned allowed = min((unsigned)SP_MAX_DONORS, 1u + shortfall / P.spread);
      const unsigned cand = __ballot_sync(FULL, lev >= 0 && key <= best + kNear);
      const unsigned rank = __popc(cand & ((1u << lane) - 1u));
      const bool donor = ((cand >> lane) & 1u) && rank < allowed && !(events & kDebt);
      const unsigned donors = __ballot_sync(FULL, donor);
      if (lane == 0) {
        atomicAdd(&s_stat[2], 1u);  // hungry polls
        if (donors) atomicAdd(&s_stat[4], 1u);
      }
      uint32_t tbase = 0;
      const int lead = donors ? __ffs(donors) - 1 : 0;
      if (donors && lane == lead) {
        atomicAdd(&ctl->outstanding, (uint32_t)__popc(donors));
        tbase = atomicAdd(&ctl->tail, (uint32_t)__popc(donors));
      }
      tbase = __shfl_sync(FULL, tbase, lead);
      // The lead lane's count comes before what any donor, or the claimant of
      // what it publishes, takes off again, so that `outstanding` never reads 0
      // while work is left: a warp barrier orders memory among the warp's lanes
      // (a shuffle does not), a record's release and acquire the rest.
      __syncwarp();
      if (donor) {
        // the reserved index's ring slot is free once the slot's previous
        // occupant (index t - cap, claimed long before) was copied out, which
        // in practice it already is -- wait a bounded time, else keep the
        // branch and owe the index a null task
        atomicAdd(&s_stat[0], 1u);
        if (MULTI) atomicAdd(&P.inst_out[cur_inst & 0x7FFFFFFFu], 1u);  // the donor's own task keeps it >= 1
        const uint32_t t = tbase + (uint32_t)__popc(donors & ((1u << lane) - 1u));
        const bool ok = slot_free(t, 4096);
        if (!ok) {
          atomicAdd(&s_stat[1], 1u);
          events |= kDebt;
          s_cold1[tid] = t;
          s_cold2[tid] = sub;
        }
        if (ok) {
          publish_node(t, lev, dmask, MULTI ? (cur_inst >> 31) << 6 : 0u);
          atomicAdd(&ctl->donated, 1ull);
          if (lev == k) rem = 0;
          else level_cut(lev);
        }
      }
    }
  }
  // efficiency counters
  if (lane == 0) {
    atomicAdd(&ctl->counters[0], ws.steps);
    atomicAdd(&ctl->counters[1], ws.slots);
    atomicAdd(&ctl->counters[2], ws.idle);
    atomicAdd(&ctl->counters[3], (unsigned long long)clock64() - ws.begin);
  }
  __syncthreads();
  if (tid < 5) atomicAdd(&ctl->counters[4 + tid], (unsigned long long)s_stat[tid]);
}

template <int W, bool PDB, int BLOCK, int WORDS, bool MULTI>
__global__ void __launch_bounds__(BLOCK, blocks_on_sm(W, PDB, MULTI, BLOCK)) search_round_kernel(RoundParams P) {
  search_round<W, PDB, BLOCK, WORDS, MULTI>(P);
}

// A round in one block per SM.
template <int W, bool PDB>
__global__ void __launch_bounds__(big_block(W, PDB), 1) search_sm_kernel(RoundParams P) {
  search_round<W, PDB, big_block(W, PDB), W == 4 ? 6 : 10, false>(P);
}

// Reset the ring (seq[s] = s: slot s free for index s) and publish the round's
// tasks at indices [0, n) (seq = index + 1): the pieces of split roots first,
// which the pre-pass has left in their slots, then the host's direct tasks
// (whole roots), which the host orders by decreasing predicted size.
__global__ void pool_init_kernel(Task *tasks, const uint32_t *n_emit, const uint32_t *direct, uint32_t n_direct,
                                 uint32_t *seq, uint32_t cap, PoolCtl *ctl, const SubRoot *subs,
                                 const int32_t *inst_iter) {
  const uint32_t ne = n_emit ? *n_emit : 0u;
  const uint32_t n = min(ne + n_direct, cap);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
    if (i >= ne && i < n) {  // a whole root: every first move
      Task *t = &tasks[i];
      const uint32_t sub = direct[i - ne];
      t->mask = 0xF;
      t->sub = sub;
      t->plen = 0;
      t->flags = inst_iter ? (uint8_t)((inst_iter[subs[sub].inst] & 1) << 6) : (uint8_t)0;
    }
    seq[i] = i < n ? i + 1u : i;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->head = 0;
    ctl->tail = n;
    ctl->outstanding = n;
    ctl->error = (ne + n_direct > cap) ? SP_ERR_CAPACITY : 0;
    ctl->donated = 0;
    ctl->heartbeat = 0;
    for (int c = 0; c < 16; ++c) ctl->counters[c] = 0;
  }
}

// One breadth-first level of the split pre-pass: each input node (a root, or
// a piece of one, at f <= limit) is expanded; every legal non-reverse child
// is counted as generated, exactly as the depth-first search would count it,
// and children within the limit go on to the next level or, at the last
// level, become pool tasks.  flags = levels still to expand.
// Four threads a node, one per move; bound by latency (a few thousand nodes a
// level, up to ten levels one after the other): a thread reads its node, sums
// the child's pattern indices from one record per cell and appends with one
// atomic per warp: a level 22 -> 9 us.
template <int W, bool PDB>
__global__ void __launch_bounds__(128) split_level_kernel(SplitArgs A) {
  constexpr int N = W * W;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t total = 4u * *A.n_in;
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t x0 = blockIdx.x * blockDim.x + threadIdx.x - lane; x0 < total; x0 += step) {
    const uint32_t x = x0 + lane, i = min(x, total - 1u) >> 2;
    const int d = (int)(x & 3u);
    const bool valid = x < total;
    uint4 b0, b1;
    uint32_t sub, levels, mv;
    int plen = 0, budget;
    if (A.roots) {
      const uint2 r = __ldg(A.roots + i);
      sub = r.x;
      levels = r.y;
      const uint4 *rec = reinterpret_cast<const uint4 *>(&A.subs[sub]);
      b0 = __ldg(rec);
      b1 = __ldg(rec + 1);
      budget = __ldg(A.inst_limit + b1.w) - (int)((b1.z >> 16) & 0xFFu) - 1;
      mv = step_legal<W>((int)((b1.z >> 8) & 0xFFu));
      if ((b1.z >> 24) != kNoPre) mv &= ~(1u << (3 - (b1.z >> 24)));
    } else {
      const uint4 *rec = reinterpret_cast<const uint4 *>(&A.in[i]);
      b0 = __ldg(rec);
      b1 = __ldg(rec + 1);
      const uint32_t meta = __ldg(reinterpret_cast<const uint32_t *>(rec + 2));
      sub = b1.w;
      plen = (int)(meta & 0xFFu);
      levels = (meta >> 8) & 0xFFu;
      budget = (int)meta >> 16;
      mv = b1.z >> 24;
    }
    const int blank = (int)((b1.z >> 8) & 0xFFu);
    if (valid && d == 0 && mv) atomicAdd(&A.sub_nodes[sub], (unsigned long long)__popc(mv));
    const bool has = valid && ((mv >> d) & 1u);
    // the child's board: the tile at `src` slides into the blank's cell
    const uint32_t w[7] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z};
    uint32_t nw[7] = {0, 0, 0, 0, 0, 0, 0};
    const int src = has ? blank + step_delta<W>((uint32_t)d) : blank;
    uint32_t moved = 0;
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (c == src) moved = (w[c / 4] >> (8 * (c % 4))) & 0xFFu;
    uint64_t ra = 0, rb = 0, fa = 0, fb = 0;
    int h = 0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const uint32_t t = c == src ? 0u : c == blank ? moved : (w[c / 4] >> (8 * (c % 4))) & 0xFFu;
      nw[c / 4] |= t << (8 * (c % 4));
      if (PDB) {
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
        hr += __ldcg(A.pdb + (sum_field<W>(ra, rb, p) | base));
        hf += __ldcg(A.pdb + (sum_field<W>(fa, fb, p) | base));
      }
      h = max(hr, hf);
    }
    bool keep = has && h <= budget;
    if (keep && plen >= kMaxPath) {
      atomicCAS(A.error, 0, SP_ERR_STACK_OVERFLOW);
      keep = false;
    }
    const uint32_t *path = A.roots ? nullptr : A.in[i].path;
    auto child_path = [&](int q) -> uint32_t {  // word q of the child's path
      uint32_t v = 16 * q < plen ? __ldg(path + q) : 0u;
      if (q == plen >> 4) {
        const int sh = 2 * (plen & 15);
        v = (v & ~(3u << sh)) | (uint32_t)d << sh;
      }
      return v;
    };
    if (keep && h == 0) {  // a goal at the child: record it like the search does
      const SubRoot *root = &A.subs[sub];
      Solution *S = &A.sol[root->inst];
      atomicMax(&S->best, 0xFFFFFFFFu - ((uint32_t)root->g + (uint32_t)plen + 1u));
      if (atomicCAS(&S->flag, 0u, 1u) == 0u) {
        S->sub = sub;
        S->len = (uint32_t)(plen + 1);
        for (int q = 0; 16 * q <= plen; ++q) S->path[q] = child_path(q);
        __threadfence();
      }
    }
    const bool further = levels > 1u;
    Task *dst = nullptr;
#pragma unroll
    for (int kind = 0; kind < 2; ++kind) {  // to the next level, to the pool
      const bool mine = keep && further == (kind == 0);
      const unsigned got = __ballot_sync(FULL, mine);
      if (!got) continue;
      const int leader = __ffs(got) - 1;
      uint32_t at = 0;
      if (lane == leader) at = atomicAdd(kind == 0 ? A.n_next : A.n_out, (uint32_t)__popc(got));
      at = __shfl_sync(FULL, at, leader) + __popc(got & ((1u << lane) - 1u));
      if (!mine) continue;
      if (at < (kind == 0 ? A.cap_next : A.cap_out)) dst = (kind == 0 ? A.next : A.out) + at;
      else atomicCAS(A.error, 0, SP_ERR_CAPACITY);
    }
    if (dst) {
      uint4 *out = reinterpret_cast<uint4 *>(dst);
      const uint32_t child = step_legal<W>(src) & ~(1u << (3 - d));
      out[0] = make_uint4(nw[0], nw[1], nw[2], nw[3]);
      out[1] = make_uint4(nw[4], nw[5], (nw[6] & 0xFFu) | (uint32_t)src << 8 | child << 24, sub);
      *reinterpret_cast<uint32_t *>(out + 2) =
          (uint32_t)(plen + 1) | (levels - 1u) << 8 | (uint32_t)min(budget - 1, kMaxBudget) << 16;
      for (int q = 0; 16 * q <= plen; ++q) dst->path[q] = child_path(q);
    }
  }
}

cudaError_t launch_split_level(int w, bool pdb, int num_sms, const SplitArgs &A, cudaStream_t st) {
  const int grid = num_sms * 8, block = 128;
  if (w == 4) {
    if (pdb) split_level_kernel<4, true><<<grid, block, 0, st>>>(A);
    else split_level_kernel<4, false><<<grid, block, 0, st>>>(A);
  } else {
    if (pdb) split_level_kernel<5, true><<<grid, block, 0, st>>>(A);
    else split_level_kernel<5, false><<<grid, block, 0, st>>>(A);
  }
  note_launch();
  return cudaGetLastError();
}

// Host launchers (template kernels stay in this translation unit).
struct SearchShape {
  void (*kern)(RoundParams) = nullptr;
  int grid = 0, block = 0;
};
template <bool MULTI>
static cudaError_t search_shape(int w, bool pdb, int block, int blocks_per_sm, int num_sms, SearchShape *out) {
  void (*kern)(RoundParams) = nullptr;
#define SP_PICK(W, PD, B, WD) \
  if (w == W && pdb == PD && block == B) kern = search_round_kernel<W, PD, B, WD, MULTI>;
  SP_PICK(4, false, 256, 6)
  SP_PICK(4, true, 256, 6)
  SP_PICK(5, false, 256, 10)
  SP_PICK(5, true, 256, 10)
  SP_PICK(4, false, 128, 6)
  SP_PICK(4, true, 128, 6)
  SP_PICK(5, false, 128, 10)
  SP_PICK(5, true, 128, 10)
#undef SP_PICK
  if (!MULTI && block == 256 && blocks_per_sm <= 0) {  // one block per SM
    block = big_block(w, pdb);
    if (w == 4) kern = pdb ? search_sm_kernel<4, true> : search_sm_kernel<4, false>;
    else kern = pdb ? search_sm_kernel<5, true> : search_sm_kernel<5, false>;
  }
  if (!kern) return cudaErrorInvalidValue;
  int per_sm = blocks_per_sm;
  if (per_sm <= 0) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
  }
  *out = SearchShape{kern, num_sms * per_sm, block};
  return cudaSuccess;
}

static cudaError_t search_shape(int w, bool pdb, int block, int blocks_per_sm, int num_sms, bool multi,
                                SearchShape *out) {
  return multi ? search_shape<true>(w, pdb, block, blocks_per_sm, num_sms, out)
               : search_shape<false>(w, pdb, block, blocks_per_sm, num_sms, out);
}

cudaError_t search_lanes(int w, bool pdb, int block, int blocks_per_sm, int num_sms, bool multi, uint32_t *lanes) {
  SearchShape x;
  const cudaError_t e = search_shape(w, pdb, block, blocks_per_sm, num_sms, multi, &x);
  if (e == cudaSuccess) *lanes = (uint32_t)(x.grid * x.block);
  return e;
}

cudaError_t launch_search(int w, bool pdb, int block, int blocks_per_sm, int num_sms, bool multi, const RoundParams &P,
                          cudaStream_t st) {
  SearchShape x;
  const cudaError_t e = search_shape(w, pdb, block, blocks_per_sm, num_sms, multi, &x);
  if (e != cudaSuccess) return e;
  x.kern<<<x.grid, x.block, 0, st>>>(P);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_pool_init(Task *tasks, const uint32_t *n_emit, const uint32_t *direct, uint32_t n_direct,
                             uint32_t *seq, uint32_t cap, PoolCtl *ctl, const SubRoot *subs, const int32_t *inst_iter,
                             cudaStream_t st) {
  const uint32_t blocks = std::min<uint32_t>((cap + 255) / 256, 152u * 32u);
  pool_init_kernel<<<blocks, 256, 0, st>>>(tasks, n_emit, direct, n_direct, seq, cap, ctl, subs, inst_iter);
  note_launch();
  return cudaGetLastError();
}

}  // namespace sp
