// Learned load balancer on the GPU: layer-1 gather-sum, tcgen05 GEMMs with
// fused epilogues, Adam.  See lbm.h for the model.
//
// GEMM shape: C[M x 256] = A[M x K] . B[256 x K]^T with A and B bf16, K-major
// (K contiguous), fp32 accumulation in tensor memory.  One CTA of 8 warps
// computes one 128-row tile over a K range:
//   * thread 0 streams 64-wide K chunks of A (128 x 64) and B (256 x 64) into
//     shared memory with TMA (128-byte swizzle), two stages, completion on an
//     mbarrier, and issues four tcgen05.mma (M=128, N=256, K=16) per chunk;
//     tcgen05.commit frees a stage once its MMAs have read it;
//   * warp 0 allocates 256 TMEM columns (the 128 x 256 fp32 accumulator);
//   * after the last commit every warp reads half of the columns of its 32
//     accumulator rows with tcgen05.ld (32x32b) and runs the epilogue.
// The training step is four such GEMMs in three launches (dZ1 and dW2 do not
// depend on each other and fill half of the SMs each); with two warps per 32
// accumulator rows and 16-byte reductions they take 49 us for 8192 24-puzzle
// rows, 112 before:
//   forward   Z2 = H1 . W2^T          epilogue: ReLU, layer 3, loss, dL/dy,
//                                     dH2 = dy w3 (Z2 > 0), d/dw3, d/db2
//   backward  dZ1 = dH2 . W2          epilogue: dH1 = dZ1 (H1 > 0), d/db1
//   dW2 = dH2^T . H1                  (split K over the batch, fp32 atomics)
//   dW1 = X^T . dH1                   (X = the one-hot input, ditto)
// Every mbarrier wait is bounded (2 s of %globaltimer); on expiry the CTA
// records an error, drains its copies in flight (bounded), frees its tensor
// memory and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/slide.h"
#include "lbm.h"
#include "sp_defs.h"
#include "sp_kernels.h"

namespace sp {
namespace lbm {

namespace {

constexpr int H = kHidden;
constexpr int BM = 128;                      // accumulator rows per CTA (TMEM lanes)
constexpr int BK = 64;                       // K per stage: one 128-byte swizzle row of bf16
constexpr int STAGES = 2;
constexpr int A_STAGE = BM * BK * 2;         // 16 KB
constexpr int B_STAGE = H * BK * 2;          // 32 KB
constexpr int SMEM_TILES = STAGES * (A_STAGE + B_STAGE);
constexpr int SMEM_BYTES = SMEM_TILES + 1024 /* alignment slack */ + 128 /* barriers, TMEM address */ +
                           2 * BM * 4 /* partial predictions */;
constexpr int kGemmThreads = 256;            // two warps per 32 accumulator rows, half of the columns each
// kind::f16 instruction descriptor: D f32 (bits 4-5 = 1), A bf16 (7-9 = 1),
// B bf16 (10-12 = 1), both K-major (15, 16 = 0), N >> 3 at 17-22, M >> 4 at 24-28
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(H >> 3) << 17) |
                            ((uint32_t)(BM >> 4) << 24);

enum { EPI_F32 = 0, EPI_F32_ATOMIC = 1, EPI_FWD = 2, EPI_BWD1 = 3, EPI_INFER = 4 };

struct EpiArgs {
  float *C;          // EPI_F32 / EPI_F32_ATOMIC: C[row * 256 + col]
  int m_valid;       // rows >= m_valid are padding
  int ldt;           // leading dimension of the transposed bf16 outputs (the batch)
  float inv_b;       // 1 / batch rows, for the mean loss
  const float *b2, *w3, *b3;
  const float *target;
  float *y;
  __nv_bfloat16 *dH2, *dH2T;      // forward-train outputs
  const __nv_bfloat16 *H1;        // backward: ReLU mask of layer 1
  __nv_bfloat16 *dH1T;            // backward output
  float *gw3, *gb2, *gb3, *gb1, *loss;
  int *err;
  unsigned long long wait_ns;  // limit of every mbarrier wait (0: 2 s)
  int starve_kc1;              // self-test only: K chunk starve_kc1 - 1 gets no copies (0: none)
};

// ---- PTX wrappers ---------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false after limit_ns without the phase completing.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
  unsigned long long t0 = 0;
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u) {
      const unsigned long long now = gtimer();
      if (!t0) t0 = now;
      else if (now - t0 > limit_ns) return false;
    }
  }
}
__device__ __forceinline__ void tma_load_2d(const CUtensorMap *map, uint32_t dst, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(holder), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// 32 consecutive fp32 accumulator columns of this thread's row.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of a K-major tile written by TMA with the
// 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart (SBO),
// descriptor version 1, layout type 2 (128-byte swizzle).  The tile base is
// 1024-byte aligned; a K step of 16 elements inside the row adds 32 bytes.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;                       // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((1024u >> 4) & 0x3FFFu) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;                       // version
  d |= (uint64_t)2 << 61;                       // 128-byte swizzle
  return d;
}

// In lane l: the sum over the warp's 32 lanes of v[l] (v is consumed).
__device__ __forceinline__ float warp_colsum(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o];
      const float keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// 32 bf16 values as four 16-byte stores.
__device__ __forceinline__ void store_bf16x32(__nv_bfloat16 *dst, const float (&v)[32]) {
  uint32_t p[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    p[i] = *reinterpret_cast<const uint32_t *>(&h);
  }
  uint4 *d = reinterpret_cast<uint4 *>(dst);
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
}

// Epilogue of a CTA's 128 x 256 accumulator.  Warp w reads the TMEM lanes
// 32 * (w & 3) .. of its warpgroup's position, and the columns of half w >> 2.
template <int EPI>
__device__ __forceinline__ void epilogue(const EpiArgs &E, uint32_t tmem, int m0, float (*s_y)[BM]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = warp >> 2, in_tile = (warp & 3) * 32 + lane;
  const int row = m0 + in_tile;
  const uint32_t tbase = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const bool valid = row < E.m_valid;
  const int cb = half * (H / 2), ce = cb + H / 2;
  if (EPI == EPI_F32 || EPI == EPI_F32_ATOMIC) {
    for (int c0 = cb; c0 < ce; c0 += 32) {
      float v[32];
      tmem_ld32(tbase + c0, v);
      if (valid) {
        float4 *dst = reinterpret_cast<float4 *>(E.C + (size_t)row * H + c0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 x = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          if (EPI == EPI_F32) dst[j] = x;
          else atomicAdd(dst + j, x);  // one 16-byte reduction
        }
      }
    }
  } else if (EPI == EPI_FWD || EPI == EPI_INFER) {
    float part = 0.f;
    for (int c0 = cb; c0 < ce; c0 += 32) {
      float v[32];
      tmem_ld32(tbase + c0, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float z = v[j] + E.b2[c0 + j];
        if (z > 0.f) part += z * E.w3[c0 + j];
      }
    }
    s_y[half][in_tile] = part;
    __syncthreads();
    const float yv = s_y[0][in_tile] + s_y[1][in_tile] + E.b3[0];
    if (valid && half == 0) E.y[row] = yv;
    if (EPI == EPI_FWD) {
      float dy = 0.f, l = 0.f;
      if (valid) {
        const float d = yv - E.target[row];
        l = d * d;
        dy = 2.f * d * E.inv_b;
      }
      if (half == 0) {
        l = warp_sum(l);
        const float sdy = warp_sum(dy);
        if (lane == 0) {
          atomicAdd(E.loss, l * E.inv_b);
          atomicAdd(E.gb3, sdy);
        }
      }
      for (int c0 = cb; c0 < ce; c0 += 32) {
        float v[32], gw[32], gb[32];
        tmem_ld32(tbase + c0, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float z = v[j] + E.b2[c0 + j];
          const float d = z > 0.f ? dy * E.w3[c0 + j] : 0.f;
          gw[j] = z > 0.f ? dy * z : 0.f;
          gb[j] = d;
          v[j] = d;
        }
        store_bf16x32(E.dH2 + (size_t)row * H + c0, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) E.dH2T[(size_t)(c0 + j) * E.ldt + row] = __float2bfloat16_rn(v[j]);
        const float s1 = warp_colsum(gw, lane);
        const float s2 = warp_colsum(gb, lane);
        atomicAdd(&E.gw3[c0 + lane], s1);
        atomicAdd(&E.gb2[c0 + lane], s2);
      }
    }
  } else if (EPI == EPI_BWD1) {
    for (int c0 = cb; c0 < ce; c0 += 32) {
      float v[32];
      tmem_ld32(tbase + c0, v);
      const uint4 *hp = reinterpret_cast<const uint4 *>(E.H1 + (size_t)row * H + c0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 u = hp[q];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 h2 = *reinterpret_cast<const __nv_bfloat162 *>(&w[e]);
          const int j = q * 8 + e * 2;
          if (!(__low2float(h2) > 0.f)) v[j] = 0.f;
          if (!(__high2float(h2) > 0.f)) v[j + 1] = 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) E.dH1T[(size_t)(c0 + j) * E.ldt + row] = __float2bfloat16_rn(v[j]);
      const float s = warp_colsum(v, lane);
      atomicAdd(&E.gb1[c0 + lane], s);
    }
  }
}

// A GEMM of a launch: its operands, row tiles, and the K chunks of a CTA.
struct GemmArgs {
  int m_tiles, kc_per_cta, kc_total;
  EpiArgs E;
};

// One launch runs GEMM `a` on its first CTAs and, when EPI2 is given, GEMM
// `b` on the others: of two that do not depend on each other and fill half of
// the SMs each.
template <int EPI, int EPI2>
__global__ void __launch_bounds__(kGemmThreads, 1)
    umma_gemm_kernel(const __grid_constant__ CUtensorMap a_a, const __grid_constant__ CUtensorMap a_b,
                     const __grid_constant__ GemmArgs a, const __grid_constant__ CUtensorMap b_a,
                     const __grid_constant__ CUtensorMap b_b, const __grid_constant__ GemmArgs b, int ctas_a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *sA = smem;
  uint8_t *sB = smem + STAGES * A_STAGE;
  uint64_t *bars = (uint64_t *)(smem + SMEM_TILES);  // full[2], done[2], accum
  uint32_t *tmem_holder = (uint32_t *)(bars + 6);
  int *s_fail = (int *)(bars + 7);
  float(*s_y)[BM] = reinterpret_cast<float(*)[BM]>(smem + SMEM_TILES + 128);
  const int warp = threadIdx.x >> 5;
  const bool second = EPI2 >= 0 && (int)blockIdx.x >= ctas_a;
  const CUtensorMap *ta = second ? &b_a : &a_a, *tb = second ? &b_b : &a_b;
  const GemmArgs &G = second ? b : a;
  const EpiArgs &E = G.E;
  const int cta = (int)blockIdx.x - (second ? ctas_a : 0);
  const int m0 = (cta % G.m_tiles) * BM;
  const int kc0 = (cta / G.m_tiles) * G.kc_per_cta;
  const int nk = min(G.kc_per_cta, G.kc_total - kc0);
  const uint32_t full0 = smem_u32(bars), done0 = smem_u32(bars + 2), accum = smem_u32(bars + 4);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 5; ++i) mbar_init(smem_u32(bars + i), 1);
    *s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_holder), 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;

  const unsigned long long limit = E.wait_ns ? E.wait_ns : 2000000000ull;
  if (threadIdx.x == 0) {
    int issued = 0, consumed = 0;
    bool ok = nk > 0;
    // chunk kc's copies; the self-test's starved chunk gets none, so the
    // wait for it runs out (its stage's barrier never completes a phase)
    auto issue = [&](int kc) {
      const int s = kc % STAGES;
      if (kc0 + kc + 1 != E.starve_kc1) {
        mbar_expect_tx(full0 + 8 * s, A_STAGE + B_STAGE);
        tma_load_2d(ta, smem_u32(sA + s * A_STAGE), full0 + 8 * s, (kc0 + kc) * BK, m0);
        tma_load_2d(tb, smem_u32(sB + s * B_STAGE), full0 + 8 * s, (kc0 + kc) * BK, 0);
      }
      ++issued;
    };
    for (int kc = 0; kc < min(nk, STAGES); ++kc) issue(kc);
    for (int kc = 0; kc < nk && ok; ++kc) {
      const int s = kc % STAGES;
      const uint32_t ph = (uint32_t)(kc / STAGES) & 1u;
      if (!mbar_wait(full0 + 8 * s, ph, limit)) {
        ok = false;
        break;
      }
      ++consumed;
      tc_fence_after();
      const uint64_t ad = smem_desc(smem_u32(sA + s * A_STAGE));
      const uint64_t bd = smem_desc(smem_u32(sB + s * B_STAGE));
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
        umma_bf16(tmem, ad + (uint64_t)(kk * 2), bd + (uint64_t)(kk * 2), kIdesc, (kc | kk) ? 1u : 0u);
      umma_commit(done0 + 8 * s);
      if (kc + STAGES < nk) {
        if (!mbar_wait(done0 + 8 * s, ph, limit)) {
          ok = false;
          break;
        }
        issue(kc + STAGES);
      }
    }
    if (!ok) {
      // drain: copies in flight land before the CTA leaves (bounded)
      for (int kc = consumed; kc < issued; ++kc)
        if (kc0 + kc + 1 != E.starve_kc1) mbar_wait(full0 + 8 * (kc % STAGES), (uint32_t)(kc / STAGES) & 1u, limit);
      *s_fail = 1;
      if (E.err) atomicExch(E.err, 1);
    }
    umma_commit(accum);  // arrives once every MMA issued above has completed
  }
  __syncthreads();
  // the same answer for all threads: the epilogue has a barrier
  const bool have = __syncthreads_and(mbar_wait(accum, 0, limit) && !*(volatile int *)s_fail);
  if (!have && E.err) atomicExch(E.err, 1);
  tc_fence_after();

  if (have) {
    if (second) epilogue<EPI2 < 0 ? EPI : EPI2>(E, tmem, m0, s_y);
    else epilogue<EPI>(E, tmem, m0, s_y);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// ---- layer 1: gather-sum of one-hot rows ----------------------------------
struct EmbedArgs {
  const uint8_t *boards;   // row r's tiles at boards + (idx ? idx[r] : r) * bstride
  const uint32_t *idx;
  int bstride;
  const int32_t *slack;
  int n;                   // real rows; rows n..rows-1 are padding (the goal, slack 0)
  int rows;                // a multiple of 128
  const __nv_bfloat16 *W1; // [D][256]
  const float *b1;
  __nv_bfloat16 *H1;       // [rows][256]
  __nv_bfloat16 *H1T;      // [256][ldt] or null
  __nv_bfloat16 *XT;       // [Dpad][ldt] one-hot transposed (zeroed by the caller) or null
  int ldt;
  uint32_t *bad;           // the rows are checked when not null: the first bad row's bad_key, by atomicMax
};

// First bad row of a call (rows in order, a row's slack before its tiles),
// larger for earlier ones; 0: none.
__host__ __device__ inline uint32_t bad_key(int row, bool tiles) { return 0x7FFFFFFFu - 2u * (uint32_t)row - (tiles ? 1u : 0u); }

// A block keeps one half of W1's columns in shared memory (154 KB for the
// 24-puzzle) and streams the rows past it, 64 at a time, two to a warp, four
// columns to a lane: 24 conflict-free 8-byte shared reads per row where the
// version before gathered 24 x 512 bytes from L2.  60000 24-puzzle rows 123
// -> 47 us (60 with 16 warps), a training batch of 8192 35 -> 19 us.  Sums run
// over the tiles in order, like before.
constexpr int kEmbThreads = 1024, kEmbCols = H / 2, kEmbRows = kEmbThreads / 16;
template <int W>
constexpr size_t embed_smem() {
  return (size_t)((W * W - 1) * W * W + 1) * kEmbCols * 2 + kEmbRows * 32 * 2 + kEmbCols * (kEmbRows + 2) * 2;
}
template <int W>
__global__ void __launch_bounds__(kEmbThreads, 1) embed_kernel(EmbedArgs A) {
  constexpr int N = W * W;
  constexpr int D = (N - 1) * N + 1;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) uint8_t e_smem[];
  uint8_t *s_w = e_smem;                                                             // [D][kEmbCols]
  uint16_t *s_feat = reinterpret_cast<uint16_t *>(e_smem + (size_t)D * kEmbCols * 2);  // [row][32]
  __nv_bfloat16 *s_ht = reinterpret_cast<__nv_bfloat16 *>(s_feat + kEmbRows * 32);     // [col][kEmbRows + 2]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = blockIdx.x & 1, pairs = gridDim.x >> 1;
  for (int e = tid; e < D * (kEmbCols / 8); e += kEmbThreads) {
    const int f = e / (kEmbCols / 8), q = e % (kEmbCols / 8);
    reinterpret_cast<uint4 *>(s_w)[e] = __ldg(reinterpret_cast<const uint4 *>(A.W1 + (size_t)f * H + half * kEmbCols) + q);
  }
  const float4 bj = __ldg(reinterpret_cast<const float4 *>(A.b1 + half * kEmbCols) + lane);
  __syncthreads();
  auto cols = [&](int f) -> float4 {
    const uint2 v = *reinterpret_cast<const uint2 *>(s_w + f * (kEmbCols * 2) + lane * 8);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xFFFF0000u));
  };
  const float4 sw = cols(D - 1);
  const int r0 = 2 * warp;  // the warp's rows of a tile: r0, r0 + 1
  // the rows of the next tile are read while this one is summed
  uint32_t next_t[2];
  int next_slack[2];
  auto fetch = [&](int tile) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int row = tile * kEmbRows + r0 + q;
      next_t[q] = (uint32_t)lane;
      next_slack[q] = 0;
      if (row < A.n) {
        const size_t src = A.idx ? (size_t)A.idx[row] : (size_t)row;
        if (lane < N) next_t[q] = A.boards[src * (size_t)A.bstride + lane];
        next_slack[q] = A.slack[row];
      }
    }
  };
  fetch(blockIdx.x >> 1);
  for (int tile = blockIdx.x >> 1; tile < A.rows / kEmbRows; tile += pairs) {
    float4 acc[2];
    const uint32_t tile_t[2] = {next_t[0], next_t[1]};
    const int tile_slack[2] = {next_slack[0], next_slack[1]};
    fetch(tile + pairs);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int row = tile * kEmbRows + r0 + q;
      uint16_t *feat = s_feat + (r0 + q) * 32;
      const uint32_t t = tile_t[q];
      const int slack = tile_slack[q];
      if (row < A.n && A.bad) {
        const uint32_t seen = __reduce_or_sync(FULL, lane < N && t < N ? 1u << t : 0u);
        if (lane == 0 && (slack < 0 || slack > 255)) atomicMax(A.bad, bad_key(row, false));
        else if (lane == 0 && seen != (1u << N) - 1u) atomicMax(A.bad, bad_key(row, true));
      }
      feat[lane] = 0;
      __syncwarp();
      if (lane < N && t > 0 && t < N) feat[t - 1] = (uint16_t)((t - 1) * N + lane);
      __syncwarp();
      const float sf = (float)slack;
      acc[q].x = bj.x + sf * sw.x;
      acc[q].y = bj.y + sf * sw.y;
      acc[q].z = bj.z + sf * sw.z;
      acc[q].w = bj.w + sf * sw.w;
      if (A.XT && half == 0 && row < A.n && lane < N)
        A.XT[(size_t)(lane < N - 1 ? feat[lane] : D - 1) * A.ldt + row] = __float2bfloat16_rn(lane < N - 1 ? 1.f : sf);
    }
#pragma unroll
    for (int t = 0; t < N - 1; ++t) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 v = cols(s_feat[(r0 + q) * 32 + t]);
        acc[q].x += v.x;
        acc[q].y += v.y;
        acc[q].z += v.z;
        acc[q].w += v.w;
      }
    }
    __syncwarp();  // all lanes have read the rows' features: the next tile overwrites them
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      __nv_bfloat162 h[2];
      h[0] = __floats2bfloat162_rn(fmaxf(acc[q].x, 0.f), fmaxf(acc[q].y, 0.f));
      h[1] = __floats2bfloat162_rn(fmaxf(acc[q].z, 0.f), fmaxf(acc[q].w, 0.f));
      const size_t row = (size_t)tile * kEmbRows + r0 + q;
      *reinterpret_cast<uint2 *>(A.H1 + row * H + half * kEmbCols + 4 * lane) = *reinterpret_cast<uint2 *>(h);
      if (A.H1T) {
        s_ht[(4 * lane + 0) * (kEmbRows + 2) + r0 + q] = __low2bfloat16(h[0]);
        s_ht[(4 * lane + 1) * (kEmbRows + 2) + r0 + q] = __high2bfloat16(h[0]);
        s_ht[(4 * lane + 2) * (kEmbRows + 2) + r0 + q] = __low2bfloat16(h[1]);
        s_ht[(4 * lane + 3) * (kEmbRows + 2) + r0 + q] = __high2bfloat16(h[1]);
      }
    }
    if (A.H1T) {
      __syncthreads();
      for (int e = tid; e < kEmbCols * kEmbRows; e += kEmbThreads) {
        const int c = e / kEmbRows, r = e % kEmbRows;
        A.H1T[(size_t)(half * kEmbCols + c) * A.ldt + tile * kEmbRows + r] = s_ht[c * (kEmbRows + 2) + r];
      }
      __syncthreads();
    }
  }
}

// *bad: the batch had a bad row; the model stays as it is.
__global__ void adam_kernel(float *p, const float *g, float *m, float *v, size_t n, float lr, float c1, float c2,
                            const uint32_t *bad) {
  if (*bad) return;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
  }
}

// bf16 copies of the weights: W1 [D][256], W2 [out][in] and W2^T [in][out]
__global__ void refresh_kernel(const float *W1, size_t n1, const float *W2, __nv_bfloat16 *W1b, __nv_bfloat16 *W2b,
                               __nv_bfloat16 *W2Tb) {
  const size_t tot = n1 + (size_t)H * H;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x) {
    if (i < n1) {
      W1b[i] = __float2bfloat16_rn(W1[i]);
    } else {
      const size_t k = i - n1;
      const size_t o = k / H, in = k % H;
      const __nv_bfloat16 b = __float2bfloat16_rn(W2[k]);
      W2b[k] = b;
      W2Tb[in * H + o] = b;
    }
  }
}

// ---- host side -------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

int get_encode(std::string &err) {
  if (g_encode) return SP_OK;
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
          cudaSuccess ||
      !fn || q != cudaDriverEntryPointSuccess) {
    err = "cuTensorMapEncodeTiled is not available from the driver";
    return SP_ERR_CUDA;
  }
  g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  return SP_OK;
}

// 2-D bf16 tensor [rows][k] (k contiguous), boxes of box_rows x 64, 128-byte swizzle.
int make_map(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t k, uint32_t box_rows, std::string &err) {
  int rc = get_encode(err);
  if (rc) return rc;
  if (((uintptr_t)ptr & 15u) || (k % 64) || rows < box_rows) {
    err = "GEMM operand not aligned to the tile shape";
    return SP_ERR_ARG;
  }
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(k * 2)};
  cuuint32_t box[2] = {(cuuint32_t)BK, box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    err = "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
    return SP_ERR_CUDA;
  }
  return SP_OK;
}

// A GEMM and, on the rest of the SMs, another one (m_tiles 0: none).
struct GemmCall {
  CUtensorMap ta, tb;
  int m_tiles = 0, kc_total = 0, splits = 1;
  EpiArgs E{};
};
template <int EPI, int EPI2>
cudaError_t launch_gemms(const GemmCall &x, const GemmCall &y, cudaStream_t st) {
  // per device context: the attribute is cheap to set and is not cached
  cudaError_t e = cudaFuncSetAttribute(umma_gemm_kernel<EPI, EPI2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SMEM_BYTES);
  if (e != cudaSuccess) return e;
  auto args = [](const GemmCall &c, int &ctas) {
    const int splits = std::max(1, std::min(c.splits, c.kc_total));
    const int per = std::max(1, (c.kc_total + splits - 1) / splits);
    ctas = c.m_tiles * ((c.kc_total + per - 1) / per);  // every CTA gets at least one chunk
    return GemmArgs{std::max(1, c.m_tiles), per, c.kc_total, c.E};
  };
  int na = 0, nb = 0;
  const GemmArgs a = args(x, na), b = args(y, nb);
  if (EPI2 < 0) nb = 0;
  umma_gemm_kernel<EPI, EPI2><<<na + nb, kGemmThreads, SMEM_BYTES, st>>>(x.ta, x.tb, a, y.ta, y.tb, b, na);
  note_launch(1);
  return cudaGetLastError();
}
template <int EPI>
cudaError_t launch_gemm(const CUtensorMap &ta, const CUtensorMap &tb, int m_tiles, int kc_total, int splits,
                        const EpiArgs &E, cudaStream_t st) {
  GemmCall c;
  c.ta = ta;
  c.tb = tb;
  c.m_tiles = m_tiles;
  c.kc_total = kc_total;
  c.splits = splits;
  c.E = E;
  return launch_gemms<EPI, -1>(c, c, st);
}

uint64_t splitmix(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

struct Buffers {
  int w = 0, D = 0, Dpad = 0;
  size_t np = 0, oW1 = 0, ob1 = 0, oW2 = 0, ob2 = 0, ow3 = 0, ob3 = 0;
  float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;
  __nv_bfloat16 *W1b = nullptr, *W2b = nullptr, *W2Tb = nullptr;
  int cap = 0;  // batch rows
  uint8_t *boards = nullptr;
  uint32_t *idx = nullptr;
  int32_t *slack = nullptr;
  float *target = nullptr, *y = nullptr;
  // a call's flags behind the gradients (one memset for both): the loss, the
  // GEMMs' wait error, the first bad row (bad_key)
  float *scal = nullptr;
  int *err = nullptr;
  uint32_t *bad = nullptr;
  // pinned: the flags, and the predictions of a call until its rows are known to be good
  uint32_t *h_flags = nullptr;
  float *h_y = nullptr;
  size_t h_y_cap = 0;
  int sms = 0;
  __nv_bfloat16 *H1 = nullptr, *H1T = nullptr, *dH2 = nullptr, *dH2T = nullptr, *dH1T = nullptr, *XT = nullptr;
  void release() {
    void *ps[] = {P, G, M, V, W1b, W2b, W2Tb, boards, idx, slack, target, y, H1, H1T, dH2, dH2T, dH1T, XT};
    for (void *p : ps)
      if (p) cudaFree(p);
    if (h_flags) cudaFreeHost(h_flags);
    if (h_y) cudaFreeHost(h_y);
  }
};
constexpr size_t kFlagWords = 3;  // scal, err, bad
// CTAs over which the weight gradients' K (the batch) is split: each adds its
// 128 x 256 partial sum with 16-byte reductions.  8192 rows, two weight
// gradients: 150 CTAs and scalar atomics 70 us; 100 CTAs 27 us, 32 and 150
// the same within 5 % (32000 rows: 32 CTAs 15 % slower).
constexpr int kSplitCtas = 100;

// The status of a call whose rows had a bad one.
static int bad_row(uint32_t key, std::string &err) {
  const bool tiles = ((0x7FFFFFFFu - key) & 1u) != 0;
  err = tiles ? "tiles are not a permutation" : "slack must lie in 0..255";
  return tiles ? SP_ERR_NOT_PERMUTATION : SP_ERR_ARG;
}

#define LBM_CUDA(x)                                                       \
  do {                                                                    \
    cudaError_t e_ = (x);                                                 \
    if (e_ != cudaSuccess) {                                              \
      err = std::string(#x) + ": " + cudaGetErrorString(e_);              \
      return SP_ERR_CUDA;                                                 \
    }                                                                     \
  } while (0)

Model::Model(int width) : w_(width), b_(new Buffers) {
  Buffers &B = *b_;
  B.w = width;
  B.D = feature_dim(width);
  B.Dpad = feature_dim_padded(width);
  B.np = num_params(width);
  B.oW1 = 0;
  B.ob1 = (size_t)B.D * H;
  B.oW2 = B.ob1 + H;
  B.ob2 = B.oW2 + (size_t)H * H;
  B.ow3 = B.ob2 + H;
  B.ob3 = B.ow3 + H;
}

Model::~Model() {
  b_->release();
  delete b_;
}

int Model::init(uint64_t seed, cudaStream_t st, std::string &err) {
  Buffers &B = *b_;
  std::vector<float> p(B.np, 0.f);
  uint64_t s = seed;
  auto normal = [&]() {
    // Box-Muller on two 53-bit uniforms
    const double u1 = ((splitmix(s) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
    const double u2 = (splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
  };
  const int N = w_ * w_;
  const double s1 = std::sqrt(2.0 / N), s2 = std::sqrt(2.0 / H), s3 = std::sqrt(1.0 / H);
  for (size_t i = 0; i < (size_t)B.D * H; ++i) p[B.oW1 + i] = (float)(normal() * s1);
  for (size_t i = 0; i < (size_t)H * H; ++i) p[B.oW2 + i] = (float)(normal() * s2);
  for (size_t i = 0; i < (size_t)H; ++i) p[B.ow3 + i] = (float)(normal() * s3);
  p[B.ob3] = 8.f;
  return import_params(p.data(), p.size(), st, err);
}

int Model::import_params(const float *src, size_t n, cudaStream_t st, std::string &err) {
  Buffers &B = *b_;
  if (n != B.np) {
    err = "parameter count mismatch";
    return SP_ERR_ARG;
  }
  if (!B.P) {
    LBM_CUDA(cudaMalloc(&B.P, B.np * sizeof(float)));
    LBM_CUDA(cudaMalloc(&B.G, (B.np + kFlagWords) * sizeof(float)));
    B.scal = B.G + B.np;
    B.err = reinterpret_cast<int *>(B.scal + 1);
    B.bad = reinterpret_cast<uint32_t *>(B.scal + 2);
    LBM_CUDA(cudaMallocHost(&B.h_flags, kFlagWords * sizeof(uint32_t)));
    int dev = 0;
    LBM_CUDA(cudaGetDevice(&dev));
    LBM_CUDA(cudaDeviceGetAttribute(&B.sms, cudaDevAttrMultiProcessorCount, dev));
    LBM_CUDA(cudaMalloc(&B.M, B.np * sizeof(float)));
    LBM_CUDA(cudaMalloc(&B.V, B.np * sizeof(float)));
    LBM_CUDA(cudaMalloc(&B.W1b, (size_t)B.D * H * 2));
    LBM_CUDA(cudaMalloc(&B.W2b, (size_t)H * H * 2));
    LBM_CUDA(cudaMalloc(&B.W2Tb, (size_t)H * H * 2));
  }
  LBM_CUDA(cudaMemcpyAsync(B.P, src, B.np * sizeof(float), cudaMemcpyHostToDevice, st));
  LBM_CUDA(cudaMemsetAsync(B.M, 0, B.np * sizeof(float), st));
  LBM_CUDA(cudaMemsetAsync(B.V, 0, B.np * sizeof(float), st));
  refresh_kernel<<<256, 256, 0, st>>>(B.P + B.oW1, (size_t)B.D * H, B.P + B.oW2, B.W1b, B.W2b, B.W2Tb);
  note_launch(1);
  ++launches_;
  LBM_CUDA(cudaGetLastError());
  LBM_CUDA(cudaStreamSynchronize(st));
  adam_t_ = 0;
  ready_ = true;
  return SP_OK;
}

int Model::export_params(float *dst, size_t n, cudaStream_t st, std::string &err) {
  Buffers &B = *b_;
  if (!ready_) {
    err = "model not initialised";
    return SP_ERR_ARG;
  }
  if (n != B.np) {
    err = "parameter count mismatch";
    return SP_ERR_ARG;
  }
  LBM_CUDA(cudaMemcpyAsync(dst, B.P, B.np * sizeof(float), cudaMemcpyDeviceToHost, st));
  LBM_CUDA(cudaStreamSynchronize(st));
  return SP_OK;
}

int Model::ensure_batch(int n, std::string &err) {
  Buffers &B = *b_;
  const int need = (n + BM - 1) / BM * BM;
  if (need <= B.cap) return SP_OK;
  int cap = std::max(need, 1024);
  void *ps[] = {B.boards, B.idx, B.slack, B.target, B.y, B.H1, B.H1T, B.dH2, B.dH2T, B.dH1T, B.XT};
  for (void *p : ps)
    if (p) cudaFree(p);
  B.cap = 0;
  const int N = w_ * w_;
  LBM_CUDA(cudaMalloc(&B.boards, (size_t)cap * N));
  LBM_CUDA(cudaMalloc(&B.idx, (size_t)cap * 4));
  LBM_CUDA(cudaMalloc(&B.slack, (size_t)cap * 4));
  LBM_CUDA(cudaMalloc(&B.target, (size_t)cap * 4));
  LBM_CUDA(cudaMalloc(&B.y, (size_t)cap * 4));
  LBM_CUDA(cudaMalloc(&B.H1, (size_t)cap * H * 2));
  LBM_CUDA(cudaMalloc(&B.H1T, (size_t)cap * H * 2));
  LBM_CUDA(cudaMalloc(&B.dH2, (size_t)cap * H * 2));
  LBM_CUDA(cudaMalloc(&B.dH2T, (size_t)cap * H * 2));
  LBM_CUDA(cudaMalloc(&B.dH1T, (size_t)cap * H * 2));
  LBM_CUDA(cudaMalloc(&B.XT, (size_t)cap * B.Dpad * 2));
  B.cap = cap;
  return SP_OK;
}

template <int W>
static cudaError_t launch_embed_w(const EmbedArgs &A, int sms, cudaStream_t st) {
  // per device context: the attribute is cheap to set and is not cached
  cudaError_t e = cudaFuncSetAttribute(embed_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)embed_smem<W>());
  if (e != cudaSuccess) return e;
  const int grid = std::max(2, std::min(sms / 2 * 2, 2 * (A.rows / kEmbRows)));
  embed_kernel<W><<<grid, kEmbThreads, embed_smem<W>(), st>>>(A);
  note_launch(1);
  return cudaGetLastError();
}
static int launch_embed(int w, const EmbedArgs &A, int sms, cudaStream_t st) {
  const cudaError_t e = w == 4 ? launch_embed_w<4>(A, sms, st) : launch_embed_w<5>(A, sms, st);
  return e == cudaSuccess ? SP_OK : SP_ERR_CUDA;
}

// Layers 2 and 3 of the n rows in H1; predictions and flags come back to the
// pinned buffers, at h_y + off.
int Model::forward_infer(int n, size_t off, cudaStream_t st, std::string &err) {
  Buffers &B = *b_;
  const int rows = (n + BM - 1) / BM * BM;
  CUtensorMap ta, tb;
  int rc = make_map(&ta, B.H1, rows, H, BM, err);
  if (!rc) rc = make_map(&tb, B.W2b, H, H, H, err);
  if (rc) return rc;
  EpiArgs E{};
  E.m_valid = n;
  E.b2 = B.P + B.ob2;
  E.w3 = B.P + B.ow3;
  E.b3 = B.P + B.ob3;
  E.y = B.y;
  E.err = B.err;
  LBM_CUDA(launch_gemm<EPI_INFER>(ta, tb, rows / BM, H / BK, 1, E, st));
  launches_ += 1;
  LBM_CUDA(cudaMemcpyAsync(B.h_y + off, B.y, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
  LBM_CUDA(cudaMemcpyAsync(B.h_flags, B.scal, kFlagWords * 4, cudaMemcpyDeviceToHost, st));
  LBM_CUDA(cudaStreamSynchronize(st));
  if (B.h_flags[1]) {
    err = "tensor-core GEMM wait timed out";
    return SP_ERR_TIMEOUT;
  }
  return B.h_flags[2] ? bad_row(B.h_flags[2], err) : SP_OK;
}

// The common part of predict and predict_subs: rows from `boards` (host
// tiles, or null: device SubRoots chosen by idx).
int Model::predict_rows(const uint8_t *tiles, const SubRoot *d_subs, const uint32_t *idx, const int32_t *slack, int n,
                        float *out, cudaStream_t st, std::string &err) {
  if (!ready_) {
    err = "model not initialised";
    return SP_ERR_ARG;
  }
  Buffers &B = *b_;
  const int N = w_ * w_;
  const int chunk = 1 << 16;
  if (B.h_y_cap < (size_t)n) {
    if (B.h_y) cudaFreeHost(B.h_y);
    B.h_y = nullptr;
    B.h_y_cap = 0;
    const size_t c = std::max<size_t>((size_t)n, 4096);
    LBM_CUDA(cudaMallocHost(&B.h_y, c * sizeof(float)));
    B.h_y_cap = c;
  }
  for (int off = 0; off < n; off += chunk) {
    const int m = std::min(chunk, n - off);
    int rc = ensure_batch(m, err);
    if (rc) return rc;
    LBM_CUDA(cudaMemsetAsync(B.scal, 0, kFlagWords * sizeof(uint32_t), st));
    EmbedArgs A{};
    if (tiles) {
      LBM_CUDA(cudaMemcpyAsync(B.boards, tiles + (size_t)off * N, (size_t)m * N, cudaMemcpyHostToDevice, st));
      A.boards = B.boards;
      A.bstride = N;
      A.bad = B.bad;
    } else {
      LBM_CUDA(cudaMemcpyAsync(B.idx, idx + off, (size_t)m * 4, cudaMemcpyHostToDevice, st));
      A.boards = reinterpret_cast<const uint8_t *>(d_subs);  // SubRoot.board is its first member
      A.idx = B.idx;
      A.bstride = (int)sizeof(SubRoot);
    }
    LBM_CUDA(cudaMemcpyAsync(B.slack, slack + off, (size_t)m * 4, cudaMemcpyHostToDevice, st));
    A.slack = B.slack;
    A.n = m;
    A.rows = (m + BM - 1) / BM * BM;
    A.W1 = B.W1b;
    A.b1 = B.P + B.ob1;
    A.H1 = B.H1;
    A.ldt = A.rows;
    if (launch_embed(w_, A, B.sms, st)) {
      err = "layer-1 kernel launch failed";
      return SP_ERR_CUDA;
    }
    launches_ += 1;
    rc = forward_infer(m, (size_t)off, st, err);
    if (rc) return rc;
  }
  memcpy(out, B.h_y, (size_t)n * sizeof(float));
  return SP_OK;
}

int Model::predict(const uint8_t *tiles, const int32_t *slack, int n, float *out, cudaStream_t st,
                   std::string &err) {
  return predict_rows(tiles, nullptr, nullptr, slack, n, out, st, err);
}

int Model::predict_subs(const SubRoot *d_subs, const uint32_t *idx, const int32_t *slack, int n, float *out,
                        cudaStream_t st, std::string &err) {
  return predict_rows(nullptr, d_subs, idx, slack, n, out, st, err);
}

int Model::train_step(const uint8_t *tiles, const int32_t *slack, const float *target, int n, float lr,
                      bool update, float *loss, float *grads, cudaStream_t st, std::string &err) {
  if (!ready_) {
    err = "model not initialised";
    return SP_ERR_ARG;
  }
  if (n <= 0 || n % BM) {
    err = "training batch must be a positive multiple of 128 rows";
    return SP_ERR_ARG;
  }
  Buffers &B = *b_;
  int rc = ensure_batch(n, err);
  if (rc) return rc;
  const int N = w_ * w_;
  LBM_CUDA(cudaMemcpyAsync(B.boards, tiles, (size_t)n * N, cudaMemcpyHostToDevice, st));
  LBM_CUDA(cudaMemcpyAsync(B.slack, slack, (size_t)n * 4, cudaMemcpyHostToDevice, st));
  LBM_CUDA(cudaMemcpyAsync(B.target, target, (size_t)n * 4, cudaMemcpyHostToDevice, st));
  LBM_CUDA(cudaMemsetAsync(B.G, 0, (B.np + kFlagWords) * sizeof(float), st));
  LBM_CUDA(cudaMemsetAsync(B.XT, 0, (size_t)B.Dpad * n * 2, st));
  EmbedArgs A{};
  A.boards = B.boards;
  A.bstride = N;
  A.slack = B.slack;
  A.n = n;
  A.W1 = B.W1b;
  A.b1 = B.P + B.ob1;
  A.H1 = B.H1;
  A.H1T = B.H1T;
  A.XT = B.XT;
  A.ldt = n;
  A.rows = n;
  A.bad = B.bad;
  if (launch_embed(w_, A, B.sms, st)) {
    err = "layer-1 kernel launch failed";
    return SP_ERR_CUDA;
  }
  CUtensorMap m_a, m_b;
  EpiArgs E{};
  E.ldt = n;
  E.inv_b = 1.f / (float)n;
  E.b2 = B.P + B.ob2;
  E.w3 = B.P + B.ow3;
  E.b3 = B.P + B.ob3;
  E.target = B.target;
  E.y = B.y;
  E.dH2 = B.dH2;
  E.dH2T = B.dH2T;
  E.H1 = B.H1;
  E.dH1T = B.dH1T;
  E.gw3 = B.G + B.ow3;
  E.gb2 = B.G + B.ob2;
  E.gb3 = B.G + B.ob3;
  E.gb1 = B.G + B.ob1;
  E.loss = B.scal;
  E.err = B.err;
  // forward + loss + layer-3 backward
  E.m_valid = n;
  if ((rc = make_map(&m_a, B.H1, n, H, BM, err)) || (rc = make_map(&m_b, B.W2b, H, H, H, err))) return rc;
  LBM_CUDA(launch_gemm<EPI_FWD>(m_a, m_b, n / BM, H / BK, 1, E, st));
  // dZ1 = dH2 . W2 and, beside it, dW2 = dH2^T . H1 (K = the batch, split)
  const int kc = n / BK;
  GemmCall dz, dw;
  dz.m_tiles = n / BM;
  dz.kc_total = H / BK;
  dz.E = E;
  if ((rc = make_map(&dz.ta, B.dH2, n, H, BM, err)) || (rc = make_map(&dz.tb, B.W2Tb, H, H, H, err))) return rc;
  dw.m_tiles = H / BM;
  dw.kc_total = kc;
  dw.splits = kSplitCtas / dw.m_tiles;
  dw.E = E;
  dw.E.C = B.G + B.oW2;
  dw.E.m_valid = H;
  if ((rc = make_map(&dw.ta, B.dH2T, H, n, BM, err)) || (rc = make_map(&dw.tb, B.H1T, H, n, H, err))) return rc;
  LBM_CUDA((launch_gemms<EPI_BWD1, EPI_F32_ATOMIC>(dz, dw, st)));
  // dW1 = X^T . dH1
  E.C = B.G + B.oW1;
  E.m_valid = B.D;
  if ((rc = make_map(&m_a, B.XT, B.Dpad, n, BM, err)) || (rc = make_map(&m_b, B.dH1T, H, n, H, err))) return rc;
  LBM_CUDA(launch_gemm<EPI_F32_ATOMIC>(m_a, m_b, B.Dpad / BM, kc, std::max(1, kSplitCtas / (B.Dpad / BM)), E, st));
  launches_ += 4;
  if (update) {
    ++adam_t_;
    const float c1 = 1.f - std::pow(0.9f, (float)adam_t_), c2 = 1.f - std::pow(0.999f, (float)adam_t_);
    adam_kernel<<<512, 256, 0, st>>>(B.P, B.G, B.M, B.V, B.np, lr, c1, c2, B.bad);
    refresh_kernel<<<256, 256, 0, st>>>(B.P + B.oW1, (size_t)B.D * H, B.P + B.oW2, B.W1b, B.W2b, B.W2Tb);
    note_launch(2);
    launches_ += 2;
    LBM_CUDA(cudaGetLastError());
  }
  // flags first: a batch with a bad row leaves grads untouched, and the model
  // too (adam_kernel)
  LBM_CUDA(cudaMemcpyAsync(B.h_flags, B.scal, kFlagWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  LBM_CUDA(cudaStreamSynchronize(st));
  if (B.h_flags[2]) {
    if (update) --adam_t_;
    return bad_row(B.h_flags[2], err);
  }
  if (grads) {
    LBM_CUDA(cudaMemcpyAsync(grads, B.G, B.np * sizeof(float), cudaMemcpyDeviceToHost, st));
    LBM_CUDA(cudaStreamSynchronize(st));
  }
  if (B.h_flags[1]) {
    err = "tensor-core GEMM wait timed out";
    return SP_ERR_TIMEOUT;
  }
  if (loss) memcpy(loss, &B.h_flags[0], sizeof(float));
  return SP_OK;
}

int Model::gemm_stall_selftest(int starve_chunk, int timeout_ms, int *device_status, cudaStream_t st,
                               std::string &err) {
  constexpr int M = BM, K = 4 * BK;
  if (starve_chunk < 0 || starve_chunk >= K / BK || timeout_ms < 10 || timeout_ms > 2000 || !device_status) {
    err = "selftest needs starve_chunk in [0, 4) and timeout_ms in [10, 2000]";
    return SP_ERR_ARG;
  }
  *device_status = SP_OK;
  void *dA = nullptr, *dB = nullptr, *dC = nullptr;
  int *derr = nullptr;
  int rc = SP_OK;
  do {
    if (cudaMalloc(&dA, (size_t)M * K * 2) || cudaMalloc(&dB, (size_t)H * K * 2) ||
        cudaMalloc(&dC, (size_t)M * H * 4) || cudaMalloc((void **)&derr, sizeof(int))) {
      err = "cudaMalloc failed";
      rc = SP_ERR_CUDA;
      break;
    }
    if (cudaMemsetAsync(dA, 0, (size_t)M * K * 2, st) || cudaMemsetAsync(dB, 0, (size_t)H * K * 2, st) ||
        cudaMemsetAsync(derr, 0, sizeof(int), st)) {
      err = "memset failed";
      rc = SP_ERR_CUDA;
      break;
    }
    CUtensorMap ta, tb;
    if ((rc = make_map(&ta, dA, M, K, BM, err)) || (rc = make_map(&tb, dB, H, K, H, err))) break;
    EpiArgs E{};
    E.C = (float *)dC;
    E.m_valid = M;
    E.err = derr;
    E.wait_ns = (unsigned long long)timeout_ms * 1000000ull;
    E.starve_kc1 = starve_chunk + 1;
    if (launch_gemm<EPI_F32>(ta, tb, 1, K / BK, 1, E, st) != cudaSuccess) {
      err = "GEMM launch failed";
      rc = SP_ERR_CUDA;
      break;
    }
    int herr = 0;
    if (cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st) || cudaStreamSynchronize(st)) {
      err = std::string("GEMM self-test failed: ") + cudaGetErrorString(cudaGetLastError());
      rc = SP_ERR_CUDA;
      break;
    }
    *device_status = herr ? SP_ERR_TIMEOUT : SP_OK;
  } while (0);
  if (dA) cudaFree(dA);
  if (dB) cudaFree(dB);
  if (dC) cudaFree(dC);
  if (derr) cudaFree(derr);
  return rc;
}

int Model::gemm_nt(const uint16_t *A, const uint16_t *Bm, float *C, int M, int N, int K, cudaStream_t st,
                   std::string &err) {
  if (M <= 0 || M % BM || N != H || K <= 0 || K % BK) {
    err = "gemm_nt needs M a multiple of 128, N = 256, K a multiple of 64";
    return SP_ERR_ARG;
  }
  void *dA = nullptr, *dB = nullptr, *dC = nullptr;
  int *derr = nullptr;
  auto cleanup = [&]() {
    if (dA) cudaFree(dA);
    if (dB) cudaFree(dB);
    if (dC) cudaFree(dC);
    if (derr) cudaFree(derr);
  };
  int rc = SP_OK;
  std::string e2;
  do {
    if (cudaMalloc(&dA, (size_t)M * K * 2) || cudaMalloc(&dB, (size_t)N * K * 2) ||
        cudaMalloc(&dC, (size_t)M * N * 4) || cudaMalloc((void **)&derr, sizeof(int))) {
      err = "cudaMalloc failed";
      rc = SP_ERR_CUDA;
      break;
    }
    if (cudaMemcpyAsync(dA, A, (size_t)M * K * 2, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(dB, Bm, (size_t)N * K * 2, cudaMemcpyHostToDevice, st) ||
        cudaMemsetAsync(derr, 0, sizeof(int), st)) {
      err = "copy failed";
      rc = SP_ERR_CUDA;
      break;
    }
    CUtensorMap ta, tb;
    if ((rc = make_map(&ta, dA, M, K, BM, err)) || (rc = make_map(&tb, dB, N, K, H, err))) break;
    EpiArgs E{};
    E.C = (float *)dC;
    E.m_valid = M;
    E.err = derr;
    if (launch_gemm<EPI_F32>(ta, tb, M / BM, K / BK, 1, E, st) != cudaSuccess) {
      err = "GEMM launch failed";
      rc = SP_ERR_CUDA;
      break;
    }
    int herr = 0;
    if (cudaMemcpyAsync(C, dC, (size_t)M * N * 4, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st) || cudaStreamSynchronize(st)) {
      err = std::string("GEMM failed: ") + cudaGetErrorString(cudaGetLastError());
      rc = SP_ERR_CUDA;
      break;
    }
    if (herr) {
      err = "tensor-core GEMM wait timed out";
      rc = SP_ERR_TIMEOUT;
    }
  } while (0);
  cleanup();
  return rc;
}

}  // namespace lbm
}  // namespace sp
