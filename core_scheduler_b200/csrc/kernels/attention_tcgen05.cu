// SPDX-License-Identifier: Apache-2.0
// Self-attention on tcgen05 tensor cores for head dimension 64, causal or not, reading the packed qkv tensor
// [B, T, 3, H, 64] (the c_attn output) directly. Forward: writes [B, T, H*64] plus the per-row log-sum-exp.
//
// One CTA per (batch, head, 128-query block), 192 threads:
//   warp 0     TMA producer: Q once, then K and V tiles of 128 keys (two stages)
//   warp 1     MMA issuer: S = Q K^T (128x128x64, fp32 in TMEM) and O += P V (128x64x128; P is a bf16 A operand in
//              TMEM, V an MN-major operand). The scores of block j+1 are issued as soon as those of block j sit in registers
//   warps 2-5  softmax: one thread per query row reads its row of S once (128 registers), keeps the reference max /
//              running sum, exponentiates on packed pairs and writes P back to TMEM. O accumulates in TMEM across key
//              blocks; a warp rescales its 32 rows of O in place only when a row maximum has grown by more than 2^8 since
//              the reference was taken (probabilities stay below 256, exact after the final division)
// Two CTAs share an SM (81 KB of shared memory, 256 TMEM columns, 154 registers a thread): one's barriers and loads hide
// behind the other's exponentials, 1024 cycles a block and what bounds it. 16 x 1024 tokens, 12 heads, causal: 102 -> 58 us
// against four CTAs with 64-key blocks that read S twice and passed P through shared memory; 2 x 4096, 20 heads
// 289 -> 122. Scores never touch global memory. Every mbarrier wait is bounded (abort flag + status word).
//
// What it replaces in the reference project: at::_scaled_dot_product_flash_attention
// (src/compute/sdpa_flash_attn.cpp:56-60) and the cuDNN-frontend SDPA graph
// (src/compute/sdpa_cudnn.cpp:84-172) together with the split/view glue around them.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdlib>

#include "api.h"
#include "bounds_check.h"
#include "tensor_map.h"

namespace cs::kernels {
namespace {
constexpr int BQ = 128;      // queries per CTA
constexpr int BKV = 128;     // keys per step
constexpr int HD = 64;       // head dimension
constexpr int TILE_BYTES = 128 * HD * 2;      // 16 KB: a 128-row tile
constexpr int THREADS = 192;
constexpr int FWD_CTAS_PER_SM = 2;
constexpr int FWD_STAGES = 2;
constexpr int SMEM_BYTES = TILE_BYTES + FWD_STAGES * 2 * TILE_BYTES + 1024 + 256;  // ~81 KB
constexpr int TMEM_COLS = 256;  // S 128, P 64, O 64
constexpr long long kWaitBudgetCycles = 4000000000LL;

__device__ DeviceStatus g_attn_status;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitBudgetCycles) {
      *abort_flag = 1;
      return false;
    }
  }
}
// One lane of the (converged) warp. The branch it guards must stay free of further branches: with one inside, every
// tcgen05.mma in it takes 85 cycles to issue instead of the 34-64 it executes in.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
// After an abandoned wait: copies into this block's shared memory may still be in flight. Gives them a bounded time to land
// before the block goes away.
__device__ __forceinline__ void abort_grace(volatile int *abort_flag) {
  if (!*abort_flag) return;
  const long long t0 = clock64();
  while (clock64() - t0 < 2000000LL) __nanosleep(1000);
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with the A operand in tensor memory (rows = lanes, two bf16 of K per 32-bit column).
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t desc = 0;
  desc |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  desc |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  desc |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  desc |= static_cast<uint64_t>(1) << 46;
  desc |= static_cast<uint64_t>(2) << 61;  // 128-byte swizzle
  return desc;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// packed fp32 pairs (one instruction, IEEE rounding of each half)
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(F2 x, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&t);
}

// Bits `first` .. 31 of a 32-column mask, for any `first`.
__device__ __forceinline__ uint32_t columns_from(int first) { return first >= 32 ? 0u : (first <= 0 ? ~0u : ~0u << first); }
// Scores outside the mask become -inf. Bit tests on one register cost half of what 32 index comparisons do.
__device__ __forceinline__ void mask_columns(uint32_t (&v)[32], uint32_t keep) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (!((keep >> i) & 1u)) v[i] = 0xff800000u;
}

struct AttnParams {
  __nv_bfloat16 *out;   // [B, T, H*64]
  float *lse;           // [B, H, T]
  int B, T, H;
  float scale_log2e;    // softmax scale * log2(e)
  float scale;
  DeviceStatus *status;
  int causal;           // 1: keys after the query are masked; 0: every query sees every key
  int negate;           // 1: the tensor core forms -Q K^T, and `scale` is the magnitude of a negative softmax scale
};

__global__ void __launch_bounds__(THREADS, FWD_CTAS_PER_SM) attention_fwd_kernel(const __grid_constant__ CUtensorMap map_qkv,
                                                                                 const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_smem = base;                                    // 128 x 64
  const uint32_t kv_smem = q_smem + TILE_BYTES;                    // per stage: K tile, V tile
  const uint32_t bar_base = kv_smem + FWD_STAGES * 2 * TILE_BYTES;
  uint64_t *bars = reinterpret_cast<uint64_t *>(aligned + (bar_base - base));
  enum { Q_FULL = 0, S_FULL, S_EMPTY, P_FULL, O_DONE, K_FULL, V_FULL = K_FULL + FWD_STAGES, K_EMPTY = V_FULL + FWD_STAGES,
         V_EMPTY = K_EMPTY + FWD_STAGES, NUM_BARS = V_EMPTY + FWD_STAGES };
  auto bar = [&](int i) { return bar_base + 8u * i; };
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + NUM_BARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + NUM_BARS + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // every head's longest block of queries first, its shortest last
  const int heads = p.B * p.H;
  const int qb = p.T / BQ - 1 - static_cast<int>(blockIdx.x) / heads;
  const int bh = static_cast<int>(blockIdx.x) % heads;
  const int b = bh / p.H, h = bh - b * p.H;
  const int q0 = qb * BQ;
  const int num_kv = p.causal ? qb + 1 : p.T / BKV;
  const int row_base = b * p.T;

  if (threadIdx.x == 0) {
    mbar_init(bar(Q_FULL), 1);
    mbar_init(bar(S_FULL), 1);
    mbar_init(bar(S_EMPTY), 4);  // one arrival per softmax warp
    mbar_init(bar(P_FULL), 4);
    mbar_init(bar(O_DONE), 1);
    for (int s = 0; s < FWD_STAGES; ++s) {
      mbar_init(bar(K_FULL + s), 1);
      mbar_init(bar(V_FULL + s), 1);
      mbar_init(bar(K_EMPTY + s), 1);
      mbar_init(bar(V_EMPTY + s), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t *>(tmem_slot))),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t s_tmem = tmem_base;             // 128 columns of scores
  const uint32_t p_tmem = tmem_base + BKV;       // 64 columns: probabilities, two bf16 per column
  const uint32_t o_tmem = p_tmem + BKV / 2;      // 64 columns of output accumulator

  if (warp == 0) {
    const int q_col = h * HD, k_col = (p.H + h) * HD, v_col = (2 * p.H + h) * HD;
    if (elect_one()) {
      mbar_expect_tx(bar(Q_FULL), TILE_BYTES);
      tma_load_2d(q_smem, &map_qkv, bar(Q_FULL), q_col, row_base + q0);
    }
    int s = 0;
    uint32_t ph = 0;
    for (int j = 0; j < num_kv; ++j) {
      const uint32_t k_dst = kv_smem + s * 2 * TILE_BYTES;
      if (!mbar_wait_warp(bar(K_EMPTY + s), ph ^ 1u, abort_flag)) break;
      if (elect_one()) {
        mbar_expect_tx(bar(K_FULL + s), TILE_BYTES);
        tma_load_2d(k_dst, &map_qkv, bar(K_FULL + s), k_col, row_base + j * BKV);
      }
      if (!mbar_wait_warp(bar(V_EMPTY + s), ph ^ 1u, abort_flag)) break;
      if (elect_one()) {
        mbar_expect_tx(bar(V_FULL + s), TILE_BYTES);
        tma_load_2d(k_dst + TILE_BYTES, &map_qkv, bar(V_FULL + s), v_col, row_base + j * BKV);
      }
      if (++s == FWD_STAGES) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 1) {
    // S = Q K^T: M=128, N=128, both operands K-major. O += P V: M=128, N=64, A (= P) from TMEM, B (= V) MN-major.
    const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | (p.negate ? 1u << 13 : 0u) | (static_cast<uint32_t>(BKV >> 3) << 17) | (8u << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (static_cast<uint32_t>(HD >> 3) << 17) | (8u << 24);
    // descriptors are built once; a k-step or a stage only advances the 16-byte-unit address field
    const uint64_t d_q = smem_desc(q_smem, 16, 1024), d_k = smem_desc(kv_smem, 16, 1024);
    const uint64_t d_v = smem_desc(kv_smem + TILE_BYTES, 8192, 1024);
    constexpr uint64_t kStepK = 32 >> 4, kStepMN = 2048 >> 4, kStage = (2 * TILE_BYTES) >> 4;
    bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_flag);
    int ks = 0, vs = 0;
    uint32_t kph = 0, vph = 0;
    auto issue_s = [&](int j) -> bool {
      if (!mbar_wait_warp(bar(K_FULL + ks), kph, abort_flag)) return false;
      if (!mbar_wait_warp(bar(S_EMPTY), (j & 1) ^ 1u, abort_flag)) return false;  // softmax of block j-1 has read S
      fence_after();
      const uint64_t dk = d_k + ks * kStage;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) umma(s_tmem, d_q + k * kStepK, dk + k * kStepK, idesc_s, k > 0 ? 1u : 0u);
        umma_commit(bar(S_FULL));
        umma_commit(bar(K_EMPTY + ks));
      }
      if (++ks == FWD_STAGES) {
        ks = 0;
        kph ^= 1u;
      }
      return true;
    };
    if (ok) ok = issue_s(0);
    for (int j = 0; ok && j < num_kv; ++j) {
      if (j + 1 < num_kv) ok = issue_s(j + 1);  // as soon as the softmax warps hold the scores of block j
      if (!ok) break;
      if (!mbar_wait_warp(bar(V_FULL + vs), vph, abort_flag)) break;
      if (!mbar_wait_warp(bar(P_FULL), j & 1, abort_flag)) break;
      fence_after();
      const uint64_t dv = d_v + vs * kStage;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)  // 16 keys: 8 columns of P, 2 KB of the MN-major V
          umma_ts(o_tmem, p_tmem + k * 8, dv + k * kStepMN, idesc_o, (j | k) ? 1u : 0u);
        umma_commit(bar(O_DONE));
        umma_commit(bar(V_EMPTY + vs));
      }
      if (++vs == FWD_STAGES) {
        vs = 0;
        vph ^= 1u;
      }
    }
  } else {
    const int q = warp & 3;
    const int r = q * 32 + lane;  // query row inside the block
    const int q_idx = q0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    float m_run = -INFINITY, l_run = 0.f;  // m_run: the maximum the exponents refer to (may lag the true one)
    bool ok = true;
    for (int j = 0; j < num_kv; ++j) {
      const uint32_t ph = j & 1;
      ok = mbar_wait_warp(bar(S_FULL), ph, abort_flag);
      if (!ok) break;
      fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(s_tmem + c * 32 + lane_addr, v[c]);
      tmem_wait_ld();
      // the scores sit in registers: the tensor core may start the next block's
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(S_EMPTY));
      if (p.causal && j == qb) {  // the diagonal block: key i of it is visible from row i on
#pragma unroll
        for (int c = 0; c < 4; ++c) mask_columns(v[c], ~columns_from(r + 1 - c * 32));
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) mx[(i >> 1) & 3] = fmaxf(fmaxf(mx[(i >> 1) & 3], __uint_as_float(v[c][i])), __uint_as_float(v[c][i + 1]));
      const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      // Move the reference maximum only when it lags by more than 2^8 (always on the first block).
      const bool grow = j == 0 || (m_blk - m_run) * p.scale_log2e > 8.0f;
      float alpha = 1.0f;
      if (grow) {
        alpha = fast_exp2((m_run - m_blk) * p.scale_log2e);  // first block: exp2(-inf) = 0
        m_run = m_blk;
        l_run *= alpha;
      }
      const float shift = -m_run * p.scale_log2e;
      const F2 scale2 = f2(p.scale_log2e, p.scale_log2e), shift2 = f2(shift, shift);
      F2 sum[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
      uint32_t pk[4][16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float a, d;
          f2_split(f2_fma(f2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), scale2, shift2), a, d);
          a = fast_exp2(a);
          d = fast_exp2(d);
          sum[i & 1] = f2_add(sum[i & 1], f2(a, d));
          pk[c][i] = pack2(a, d);
        }
        if (c == 0 && j > 0) {
          // P V of block j-1 has read P and completed O before either is touched again
          ok = mbar_wait_warp(bar(O_DONE), ph ^ 1u, abort_flag);
          if (!ok) break;
          fence_after();
          if (__any_sync(0xffffffffu, grow)) {  // rescale this warp's 32 rows of O in place
#pragma unroll 1
            for (int cc = 0; cc < 4; ++cc) {
              uint32_t ov[16];
              tmem_ld16(o_tmem + cc * 16 + lane_addr, ov);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tmem_st16(o_tmem + cc * 16 + lane_addr, ov);
            }
          }
        }
        tmem_st16(p_tmem + c * 16 + lane_addr, pk[c]);
      }
      if (!ok) break;
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(P_FULL));
      float a, d;
      f2_split(f2_add(sum[0], sum[1]), a, d);
      l_run += a + d;
    }
    // the last block's P V completes the accumulator
    const bool done = ok && mbar_wait_warp(bar(O_DONE), (num_kv - 1) & 1, abort_flag);
    if (__all_sync(0xffffffffu, done && !*abort_flag)) {
      fence_after();
      uint32_t o[2][32];
      tmem_ld32(o_tmem + lane_addr, o[0]);
      tmem_ld32(o_tmem + 32 + lane_addr, o[1]);
      tmem_wait_ld();
      const bool row_in_range = CS_IN_BOUNDS(kKidAttention, (static_cast<long long>(row_base + q_idx) * p.H + h) * HD + HD - 1,
                                             static_cast<long long>(p.B) * p.T * p.H * HD);
      const float inv = 1.f / l_run;
      __nv_bfloat16 *dst = p.out + (static_cast<long long>(row_base + q_idx) * p.H + h) * HD;
      if (row_in_range) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const uint32_t(&w8)[32] = o[g >> 2];
          const int at = (g & 3) * 8;
          uint4 w;
          w.x = pack2(__uint_as_float(w8[at + 0]) * inv, __uint_as_float(w8[at + 1]) * inv);
          w.y = pack2(__uint_as_float(w8[at + 2]) * inv, __uint_as_float(w8[at + 3]) * inv);
          w.z = pack2(__uint_as_float(w8[at + 4]) * inv, __uint_as_float(w8[at + 5]) * inv);
          w.w = pack2(__uint_as_float(w8[at + 6]) * inv, __uint_as_float(w8[at + 7]) * inv);
          *reinterpret_cast<uint4 *>(dst + g * 8) = w;
        }
        p.lse[(static_cast<long long>(b) * p.H + h) * p.T + q_idx] = m_run * p.scale + __logf(l_run);
      }
    }
  }

  abort_grace(abort_flag);
  fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    p.status->code = 1;
    p.status->kernel_id = 3;
    p.status->block = blockIdx.x;
    p.status->detail = 0;
  }
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------ backward ----
// dQ, dK, dV of attention from the packed qkv, the forward output, its gradient and the per-row log-sum-exp; results go
// straight into the packed dqkv [B, T, 3, H, 64].
//
// Three launches: (1) per-row constants, delta[b,h,t] = sum_d dO*O; (2) kDKV = true: a 128-key block keeps K_j, V_j
// resident and streams 64-query tiles (Q_i, dO_i), accumulating dV_j and dK_j in TMEM; (3) kDKV = false: a 128-query
// block keeps Q_i, dO_i resident and streams 64-key tiles (K_j, V_j), accumulating dQ_i in TMEM. No atomics,
// deterministic. Per streamed tile:
//   S' = R1 C1^T, dP' = R2 C2^T              (128 x 64 x 64 each, fp32 in TMEM; rows = resident side)
//   P' = exp(scale S' - lse), dS' = P' (dP' - delta)   (softmax warps; the factor `scale` of dS is applied to dK and dQ)
//   [dV += P' C2]   acc += dS' C1            (128 x 64 x 64; P' and dS' stay in TMEM as bf16 A operands over S' and dP',
//                                             C as MN-major operands)
// One persistent CTA per SM owns all 512 TMEM columns: three score buffers of 128 columns and the accumulators. Three
// groups of four softmax warps take the tiles in turn, a buffer each. What a tile costs besides its exponentials (barriers,
// TMEM latency, the MMAs before and after it: about 1200 cycles) overlaps with the other groups' tiles, which leaves a tile
// bound by 640 cycles of tensor core (dK/dV; 512 for dQ) or 512 of the exponential unit. All sixteen warps on one 128-column
// tile, the score buffer of the next one ready, ran in step with each other and needed 2250 cycles for 128 columns, two CTAs
// an SM with 64-column tiles 2800. The accumulators are drained by four warps of their own while the next block is under
// way, across whose boundary the pipeline runs on; resident tiles are double-buffered. 16 x 1024 tokens, 12 heads, causal:
// dK/dV 138 -> 78 us, dQ 91 -> 53; 2 x 4096, 20 heads 343 -> 161 and 231 -> 127.
constexpr int BC = 64;                          // streamed rows per step
constexpr int C_TILE_BYTES = BC * HD * 2;       // 8 KB
constexpr int BWD_GROUPS = 3;                   // softmax groups and score buffers
constexpr int BWD_STAGES = 6;                   // streamed-tile stages: two tiles and 512 bytes of row constants each
constexpr int BWD_THREADS = 128 + (BWD_GROUPS + 1) * 128;  // TMA warp, two MMA warps, one idle; softmax groups, accumulator group
constexpr int BWD_SMEM_BYTES = 4 * TILE_BYTES + BWD_STAGES * (2 * C_TILE_BYTES + 512) + 1024 + 512;  // ~165 KB
constexpr int BWD_TMEM_COLS = 512;

struct AttnBwdParams {
  __nv_bfloat16 *dqkv;     // [B, T, 3, H, 64]
  const float *neg_lse;    // [B, H, T]: -lse * log2(e)
  const float *neg_delta;  // [B, H, T]: -delta
  int B, T, H;
  float scale;             // factor of dQ and dK
  float scale_log2e;       // magnitude of the scale (never zero) * log2(e)
  DeviceStatus *status;
  int causal;
  int negate;              // as in the forward pass
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ float ld_shared(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void ld_shared_pairs(uint32_t addr, F2 &a, F2 &b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a.v), "=l"(b.v) : "r"(addr));
}

__global__ void __launch_bounds__(256) attention_delta_kernel(const __nv_bfloat16 *__restrict__ out, const __nv_bfloat16 *__restrict__ dout,
                                                              const float *__restrict__ lse, float *__restrict__ delta, int B, int T,
                                                              int H) {
  // eight threads per (b, t, h) row of 64 values
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long row = gid >> 3;
  const int part = static_cast<int>(gid & 7);
  const long long rows = static_cast<long long>(B) * T * H;
  float acc = 0.f;
  if (row < rows) {
    const uint4 a = *reinterpret_cast<const uint4 *>(out + row * HD + part * 8);
    const uint4 g = *reinterpret_cast<const uint4 *>(dout + row * HD + part * 8);
    const __nv_bfloat162 *pa = reinterpret_cast<const __nv_bfloat162 *>(&a);
    const __nv_bfloat162 *pg = reinterpret_cast<const __nv_bfloat162 *>(&g);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pg[i]);
      acc = fmaf(x.x, y.x, acc);
      acc = fmaf(x.y, y.y, acc);
    }
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  if (row < rows && part == 0) {
    const long long bt = row / H;
    const int h = static_cast<int>(row - bt * H);
    const long long b = bt / T;
    const int t = static_cast<int>(bt - b * T);
    // plane 0: delta; plane 1: -lse * log2(e); plane 2: -delta (what the two backward kernels add)
    const long long plane = static_cast<long long>(B) * H * T, at = (b * H + h) * T + t;
    delta[at] = acc;
    delta[plane + at] = lse[at] * -1.4426950408889634f;
    delta[2 * plane + at] = -acc;
  }
}

// One 128-row block of one head: what a CTA works on at a time.
struct BwdItem {
  int b, h, r0, c_first, n_iter;
};
template <bool kDKV>
__device__ __forceinline__ BwdItem bwd_item(const AttnBwdParams &p, int id) {
  // Longest loops of every head first: key block 0 streams all queries, query block T/128-1 streams all keys.
  const int heads = p.B * p.H, blocks = p.T / 128;
  const int order = id / heads, bh = id - order * heads;
  const int rb = kDKV ? order : blocks - 1 - order;
  BwdItem it;
  it.b = bh / p.H;
  it.h = bh - it.b * p.H;
  it.r0 = rb * 128;
  it.c_first = kDKV && p.causal ? 2 * rb : 0;  // streamed tiles: queries r0 .. T (kDKV) or keys 0 .. r0+128
  it.n_iter = kDKV ? 2 * blocks - it.c_first : 2 * (p.causal ? rb + 1 : blocks);
  return it;
}
// The k-th block of this CTA. Blocks come in order of falling length and are dealt out back and forth, so that no CTA gets
// the longest one of every round.
__device__ __forceinline__ int bwd_deal(int k) { return k * gridDim.x + ((k & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x); }

// barriers that the softmax groups use
constexpr int BWD_SDP_FULL = 6, BWD_PDS_FULL = BWD_SDP_FULL + BWD_GROUPS, BWD_C_FULL = BWD_PDS_FULL + 2 * BWD_GROUPS;

// What a softmax group of dK/dV does under a causal mask in a CTA with a query whose log-sum-exp is not finite. -inf for a masked
// score does not survive that, and the query's NaN would reach the keys it cannot see: here masked elements are cleared after the
// exponential. A function of its own, eight columns at a time: in the loop that every other CTA runs, the second mask cost
// registers and spills (dK/dV of 2 x 4096 tokens, 20 heads: 157 us without it, 166 with it there, 161 so).
__device__ __noinline__ void careful_dkdv(const AttnBwdParams &p, uint32_t s_tmem, uint32_t vec_smem, uint32_t bar_base,
                                          volatile int *abort_flag, int g, int r, int items) {
  const uint32_t dp_tmem = s_tmem + BC;
  const int lane = r & 31;
  int next = g, s = g;
  uint32_t cph = 0, parity = 0;
  for (int k = 0, id; (id = bwd_deal(k)) < items; ++k) {
    const int n_iter = bwd_item<true>(p, id).n_iter;
    for (; next < n_iter; next += BWD_GROUPS) {
      if (!mbar_wait_warp(bar_base + 8u * (BWD_C_FULL + s), cph, abort_flag)) return;
      if (!mbar_wait_warp(bar_base + 8u * (BWD_SDP_FULL + g), parity, abort_flag)) return;
      parity ^= 1u;
      fence_after();
      const uint32_t vec = vec_smem + s * 512;
#pragma unroll 1
      for (int c = 0; c < BC; c += 8) {
        uint32_t sv[8], dv[8], pp[4], dd[4];
        tmem_ld8(s_tmem + c, sv);
        tmem_ld8(dp_tmem + c, dv);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          float pr[2], ds[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t at = vec + (c + i + j) * 4;
            const bool seen = next * BC + c + i + j >= r;  // tiles start at the block's own rows
            pr[j] = seen ? fast_exp2(fmaf(__uint_as_float(sv[i + j]), p.scale_log2e, ld_shared(at))) : 0.f;
            ds[j] = seen ? pr[j] * (__uint_as_float(dv[i + j]) + ld_shared(at + 256)) : 0.f;
          }
          pp[i >> 1] = pack2(pr[0], pr[1]);
          dd[i >> 1] = pack2(ds[0], ds[1]);
        }
        // over the scores of columns up to c / 2 + 3, which this warp has read
        tmem_st4(s_tmem + c / 2, pp);
        tmem_st4(dp_tmem + c / 2, dd);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_base + 8u * (BWD_PDS_FULL + g));
      s += BWD_GROUPS;
      if (s >= BWD_STAGES) {
        s -= BWD_STAGES;
        cph ^= 1u;
      }
    }
    next -= n_iter;
  }
}

template <bool kDKV>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap qkv_r, const __grid_constant__ CUtensorMap qkv_c,
                     const __grid_constant__ CUtensorMap do_r, const __grid_constant__ CUtensorMap do_c,
                     const __grid_constant__ AttnBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
  constexpr int STAGES = BWD_STAGES, GROUPS = BWD_GROUPS;
  const uint32_t r_smem = base;                            // two buffers of the resident operands of S' and dP'
  const uint32_t c_smem = r_smem + 4 * TILE_BYTES;         // per stage: C1 tile, C2 tile
  const uint32_t vec_smem = c_smem + STAGES * 2 * C_TILE_BYTES;  // per stage: -lse[64], -delta[64] of the streamed queries
  const uint32_t bar_base = vec_smem + STAGES * 512;
  uint64_t *bars = reinterpret_cast<uint64_t *>(aligned + (bar_base - base));
  enum { R_FULL = 0, R_EMPTY = 2, ACC_FULL = 4, ACC_EMPTY, SDP_FULL = BWD_SDP_FULL, PDS_FULL = BWD_PDS_FULL, PDS_EMPTY = PDS_FULL + GROUPS,
         C_FULL = BWD_C_FULL,
         C_EMPTY = C_FULL + STAGES, NUM_BARS = C_EMPTY + STAGES };
  auto bar = [&](int i) { return bar_base + 8u * i; };
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + NUM_BARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + NUM_BARS + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int items = p.B * p.H * (p.T / 128);

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(R_FULL + s), 1);
      mbar_init(bar(R_EMPTY + s), 1);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar(C_FULL + s), 1);
      mbar_init(bar(C_EMPTY + s), 1);
    }
    for (int g = 0; g < GROUPS; ++g) {
      mbar_init(bar(SDP_FULL + g), 1);
      mbar_init(bar(PDS_FULL + g), 4);  // one arrival per warp of the group
      mbar_init(bar(PDS_EMPTY + g), 1);
    }
    mbar_init(bar(ACC_FULL), 1);
    mbar_init(bar(ACC_EMPTY), 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t *>(tmem_slot))),
                 "r"(BWD_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // buffer g: S' in 64 columns (P' later in the first 32), dP' in the next 64 (dS' later in their first 32)
  const uint32_t acc1_tmem = tmem_base + GROUPS * 2 * BC;  // dV (kDKV only)
  const uint32_t acc2_tmem = acc1_tmem + HD;               // dK or dQ

  if (warp == 0) {
    int s = 0, rbuf = 0;
    uint32_t ph = 0, rph = 0;
    bool ok = true;
    for (int k = 0, id; ok && (id = bwd_deal(k)) < items; ++k) {
      const BwdItem it = bwd_item<kDKV>(p, id);
      const int q_col = it.h * HD, k_col = (p.H + it.h) * HD, v_col = (2 * p.H + it.h) * HD, row_base = it.b * p.T;
      ok = mbar_wait_warp(bar(R_EMPTY + rbuf), rph ^ 1u, abort_flag);
      if (!ok) break;
      const uint32_t r1 = r_smem + rbuf * 2 * TILE_BYTES;
      if (elect_one()) {
        mbar_expect_tx(bar(R_FULL + rbuf), 2 * TILE_BYTES);
        tma_load_2d(r1, &qkv_r, bar(R_FULL + rbuf), kDKV ? k_col : q_col, row_base + it.r0);
        tma_load_2d(r1 + TILE_BYTES, kDKV ? &qkv_r : &do_r, bar(R_FULL + rbuf), kDKV ? v_col : q_col, row_base + it.r0);
      }
      rbuf ^= 1;
      if (rbuf == 0) rph ^= 1u;
      const long long vec_row = (static_cast<long long>(it.b) * p.H + it.h) * p.T;
      for (int t = 0; t < it.n_iter; ++t) {
        const int c0 = (it.c_first + t) * BC;
        ok = mbar_wait_warp(bar(C_EMPTY + s), ph ^ 1u, abort_flag);
        if (!ok) break;
        const uint32_t c1 = c_smem + s * 2 * C_TILE_BYTES, c2 = c1 + C_TILE_BYTES;
        if (elect_one()) {
          if (kDKV) {
            mbar_expect_tx(bar(C_FULL + s), 2 * C_TILE_BYTES + 512);
            tma_load_2d(c1, &qkv_c, bar(C_FULL + s), q_col, row_base + c0);
            tma_load_2d(c2, &do_c, bar(C_FULL + s), q_col, row_base + c0);
            bulk_load(vec_smem + s * 512, p.neg_lse + vec_row + c0, 256, bar(C_FULL + s));
            bulk_load(vec_smem + s * 512 + 256, p.neg_delta + vec_row + c0, 256, bar(C_FULL + s));
          } else {
            mbar_expect_tx(bar(C_FULL + s), 2 * C_TILE_BYTES);
            tma_load_2d(c1, &qkv_c, bar(C_FULL + s), k_col, row_base + c0);
            tma_load_2d(c2, &qkv_c, bar(C_FULL + s), v_col, row_base + c0);
          }
        }
        if (++s == STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // S' and dP' of every tile, as soon as its buffer is free: M=128, N=64, both operands K-major
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BC >> 3) << 17) | (8u << 24);
    const uint32_t idesc_s = idesc | (p.negate ? 1u << 13 : 0u);
    // descriptors are built once; a k-step, a stage or a buffer only advances the 16-byte-unit address field
    const uint64_t d_r1 = smem_desc(r_smem, 16, 1024), d_r2 = smem_desc(r_smem + TILE_BYTES, 16, 1024);
    const uint64_t d_c1 = smem_desc(c_smem, 16, 1024), d_c2 = smem_desc(c_smem + C_TILE_BYTES, 16, 1024);
    constexpr uint64_t kStage = (2 * C_TILE_BYTES) >> 4, kBuffer = (2 * TILE_BYTES) >> 4, kStepK = 32 >> 4;
    int s = 0, g = 0, rbuf = 0;
    uint32_t cph = 0, gph = 0, rph = 0;
    bool ok = true;
    for (int k = 0, id; ok && (id = bwd_deal(k)) < items; ++k) {
      const int n_iter = bwd_item<kDKV>(p, id).n_iter;
      ok = mbar_wait_warp(bar(R_FULL + rbuf), rph, abort_flag);
      if (!ok) break;
      const uint64_t rt = rbuf * kBuffer;
      for (int t = 0; t < n_iter; ++t) {
        ok = mbar_wait_warp(bar(C_FULL + s), cph, abort_flag) && mbar_wait_warp(bar(PDS_EMPTY + g), gph ^ 1u, abort_flag);
        if (!ok) break;
        fence_after();
        const uint64_t at = s * kStage;
        const uint32_t s_tmem = tmem_base + g * 2 * BC;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) umma(s_tmem, d_r1 + rt + kk * kStepK, d_c1 + at + kk * kStepK, idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) umma(s_tmem + BC, d_r2 + rt + kk * kStepK, d_c2 + at + kk * kStepK, idesc, kk > 0 ? 1u : 0u);
          umma_commit(bar(SDP_FULL + g));
        }
        if (++s == STAGES) {
          s = 0;
          cph ^= 1u;
        }
        if (++g == GROUPS) {
          g = 0;
          gph ^= 1u;
        }
      }
      if (ok && elect_one()) umma_commit(bar(R_EMPTY + rbuf));
      rbuf ^= 1;
      if (rbuf == 0) rph ^= 1u;
    }
  } else if (warp == 2) {
    // accumulators: M=128, N=64, A (P', dS') from TMEM, B MN-major. A warp of its own: issuing blocks while the pipe is
    // full, and one warp's waits for the two kinds of products cost as much as the products.
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (static_cast<uint32_t>(HD >> 3) << 17) | (8u << 24);
    const uint64_t d_c1 = smem_desc(c_smem, 8192, 1024), d_c2 = smem_desc(c_smem + C_TILE_BYTES, 8192, 1024);
    constexpr uint64_t kStage = (2 * C_TILE_BYTES) >> 4, kStepMN = 2048 >> 4;
    int s = 0, g = 0;
    uint32_t gph = 0, item_parity = 0;
    bool ok = true;
    for (int k = 0, id; ok && (id = bwd_deal(k)) < items; ++k) {
      const int n_iter = bwd_item<kDKV>(p, id).n_iter;
      ok = mbar_wait_warp(bar(ACC_EMPTY), item_parity ^ 1u, abort_flag);  // the accumulators of the block before have been read
      item_parity ^= 1u;
      if (!ok) break;
      for (int t = 0; t < n_iter; ++t) {
        ok = mbar_wait_warp(bar(PDS_FULL + g), gph, abort_flag);
        if (!ok) break;
        fence_after();
        const uint64_t at = s * kStage;
        const uint32_t p_tmem = tmem_base + g * 2 * BC, ds_tmem = p_tmem + BC;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BC / 16; ++kk) {
            if (kDKV) umma_ts(acc1_tmem, p_tmem + kk * 8, d_c2 + at + kk * kStepMN, idesc, (t | kk) ? 1u : 0u);
            umma_ts(acc2_tmem, ds_tmem + kk * 8, d_c1 + at + kk * kStepMN, idesc, (t | kk) ? 1u : 0u);
          }
          umma_commit(bar(PDS_EMPTY + g));
          umma_commit(bar(C_EMPTY + s));
        }
        if (++s == STAGES) s = 0;
        if (++g == GROUPS) {
          g = 0;
          gph ^= 1u;
        }
      }
      if (ok && elect_one()) umma_commit(bar(ACC_FULL));
    }
  } else if (warp >= 4 && warp < 4 + 4 * GROUPS) {
    const int q = warp & 3;          // TMEM lane quarter this warp may access
    const int g = (warp - 4) >> 2;   // softmax group: tiles g, g + GROUPS, ...
    const int r = q * 32 + lane;     // row of the resident block
    const uint32_t s_tmem = tmem_base + g * 2 * BC + (static_cast<uint32_t>(q * 32) << 16), dp_tmem = s_tmem + BC;
    // Does any query on the diagonal of this CTA's blocks have a log-sum-exp that is not finite? Asked while the first tiles are on
    // their way, by every warp for itself.
    bool finite = true;
    if (kDKV && p.causal) {
      for (int k0 = 0; bwd_deal(k0) < items; k0 += 4) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // all loads of a step in flight; past the last block the step's first once more
          const int id = bwd_deal(k0 + u);
          const BwdItem it = bwd_item<kDKV>(p, id < items ? id : bwd_deal(k0));
          v[u] = __ldg(reinterpret_cast<const float4 *>(p.neg_lse + (static_cast<long long>(it.b) * p.H + it.h) * p.T + it.r0) + lane);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)  // 0 * x is zero for finite x only
          finite &= (0.f * v[u].x + 0.f * v[u].y) + (0.f * v[u].z + 0.f * v[u].w) == 0.f;
      }
      finite = __all_sync(0xffffffffu, finite);
    }
    if (kDKV && !finite) {
      careful_dkdv(p, s_tmem, vec_smem, bar_base, abort_flag, g, r, items);
    } else {
      const F2 scale2 = f2(p.scale_log2e, p.scale_log2e);
      int next = g;        // steps until this group's next tile, counted from the start of a block
      int s = g;           // stage of that tile
      uint32_t cph = 0, parity = 0;
      bool ok = true;
      for (int k = 0, id; ok && (id = bwd_deal(k)) < items; ++k) {
        const BwdItem it = bwd_item<kDKV>(p, id);
        if (next >= it.n_iter) {
          next -= it.n_iter;
          continue;
        }
        float lse_r = 0.f, delta_r = 0.f;
        if (!kDKV) {
          const long long at = (static_cast<long long>(it.b) * p.H + it.h) * p.T + it.r0 + r;
          lse_r = p.neg_lse[at];
          delta_r = p.neg_delta[at];
        }
        const F2 lse_r2 = f2(lse_r, lse_r), delta_r2 = f2(delta_r, delta_r);
        for (; next < it.n_iter; next += GROUPS) {
          if (kDKV) {
            ok = mbar_wait_warp(bar(C_FULL + s), cph, abort_flag);  // -lse / -delta of the streamed queries
            if (!ok) break;
          }
          ok = mbar_wait_warp(bar(SDP_FULL + g), parity, abort_flag);
          if (!ok) break;
          parity ^= 1u;
          fence_after();
          const int c0 = (it.c_first + next) * BC - it.r0;  // first streamed row, relative to the resident block
          // rows are keys and columns queries (kDKV), or rows queries and columns keys: keep key <= query
          const bool masked = p.causal && (kDKV ? c0 < 128 : c0 + BC > 0);
          const uint32_t vec = vec_smem + s * 512;
#pragma unroll
          for (int c = 0; c < 2; ++c) {  // 32 columns at a time
            uint32_t sv[32], dv[32];
            tmem_ld32(s_tmem + c * 32, sv);
            tmem_ld32(dp_tmem + c * 32, dv);
            tmem_wait_ld();
            if (masked) {
              const int first = r - c0 - c * 32;  // dK/dV: columns below it are masked; dQ: columns above it
              mask_columns(sv, kDKV ? columns_from(first) : ~columns_from(first + 1));
            }
            uint32_t pp[16], dd[16];
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              F2 nl[2] = {lse_r2, lse_r2}, nd[2] = {delta_r2, delta_r2};
              if (kDKV) {
                ld_shared_pairs(vec + (c * 32 + i) * 4, nl[0], nl[1]);
                ld_shared_pairs(vec + 256 + (c * 32 + i) * 4, nd[0], nd[1]);
              }
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int e = i + 2 * j;
                float a, d;
                f2_split(f2_fma(f2(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), scale2, nl[j]), a, d);
                const F2 pr = f2(fast_exp2(a), fast_exp2(d));
                const F2 ds = f2_mul(pr, f2_add(f2(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])), nd[j]));
                if (kDKV) {
                  f2_split(pr, a, d);
                  pp[e >> 1] = pack2(a, d);
                }
                f2_split(ds, a, d);
                dd[e >> 1] = pack2(a, d);
              }
            }
            // over the scores of columns 0..31, which this warp has read
            if (kDKV) tmem_st16(s_tmem + c * 16, pp);
            tmem_st16(dp_tmem + c * 16, dd);
          }
          tmem_wait_st();
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(PDS_FULL + g));
          s += GROUPS;
          if (s >= STAGES) {
            s -= STAGES;
            cph ^= 1u;
          }
        }
        next -= it.n_iter;
      }
    }
  } else if (warp >= 4 + 4 * GROUPS) {
    // accumulators -> dqkv: thread = row; dV and dK, or dQ
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    uint32_t parity = 0;
    for (int k = 0, id; (id = bwd_deal(k)) < items; ++k) {
      const BwdItem it = bwd_item<kDKV>(p, id);
      if (!mbar_wait_warp(bar(ACC_FULL), parity, abort_flag)) break;
      parity ^= 1u;
      fence_after();
      const long long row = static_cast<long long>(it.b * p.T + it.r0 + r) * 3 * p.H;
      const bool row_in_range =
          CS_IN_BOUNDS(kKidAttention, (row + 2LL * p.H + it.h) * HD + HD - 1, static_cast<long long>(p.B) * p.T * 3 * p.H * HD);
#pragma unroll
      for (int part = kDKV ? 0 : 2; part < 4; ++part) {  // 32 columns each: dV, dV, dK (dQ), dK (dQ)
        const int which = kDKV ? (part < 2 ? 2 : 1) : 0;
        const float factor = part < 2 ? 1.f : p.scale;
        uint32_t v[32];
        tmem_ld32((part < 2 ? acc1_tmem : acc2_tmem) + (part & 1) * 32 + lane_addr, v);
        tmem_wait_ld();
        if (part == 3) {
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(ACC_EMPTY));
        }
        __nv_bfloat16 *dst = p.dqkv + (row + static_cast<long long>(which) * p.H + it.h) * HD + (part & 1) * 32;
        if (row_in_range) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 w;
            w.x = pack2(__uint_as_float(v[i * 8 + 0]) * factor, __uint_as_float(v[i * 8 + 1]) * factor);
            w.y = pack2(__uint_as_float(v[i * 8 + 2]) * factor, __uint_as_float(v[i * 8 + 3]) * factor);
            w.z = pack2(__uint_as_float(v[i * 8 + 4]) * factor, __uint_as_float(v[i * 8 + 5]) * factor);
            w.w = pack2(__uint_as_float(v[i * 8 + 6]) * factor, __uint_as_float(v[i * 8 + 7]) * factor);
            *reinterpret_cast<uint4 *>(dst + i * 8) = w;
          }
        }
      }
    }
  }

  abort_grace(abort_flag);
  fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    p.status->code = 1;
    p.status->kernel_id = kDKV ? 4 : 5;
    p.status->block = blockIdx.x;
    p.status->detail = 0;
  }
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(BWD_TMEM_COLS) : "memory");
  }
}

}  // namespace

int attention_status(DeviceStatus *out) {
  return static_cast<int>(cudaMemcpyFromSymbol(out, g_attn_status, sizeof(DeviceStatus)));
}

namespace {
// [rows, cols] bf16 row-major viewed through 64-column boxes of `box_rows` rows.
bool attn_map(CUtensorMap *out, const void *ptr, int64_t cols, int64_t rows, int box_rows) {
  return get_tensor_map(ptr, static_cast<uint64_t>(cols), static_cast<uint64_t>(rows), static_cast<uint64_t>(cols), HD,
                        static_cast<uint32_t>(box_rows), out);
}
DeviceStatus *attn_status_ptr() {
  static DeviceStatus *ptr = [] {
    void *p = nullptr;
    cudaGetSymbolAddress(&p, g_attn_status);
    return static_cast<DeviceStatus *>(p);
  }();
  return ptr;
}
}  // namespace

namespace {
// The running maximum, -inf for masked scores and the lag of the reference want a positive scale: a negative one is its magnitude
// with the products negated, and zero the smallest normal number, which leaves every finite score at exp(0).
float scale_magnitude(float scale) {
  const float magnitude = std::fabs(scale);
  return magnitude < FLT_MIN ? FLT_MIN : magnitude;
}
}  // namespace

int attention_forward_packed(stream_t stream, const void *qkv, void *out, float *lse, int64_t B, int64_t T, int64_t H, int64_t D,
                             float scale, int causal) {
  if (D != HD || T % BQ != 0 || B <= 0 || H <= 0 || T <= 0) return -1;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 15) return -1;
  static const bool disabled = std::getenv("CS_DISABLE_TCGEN05_ATTENTION") != nullptr;
  if (disabled) return -1;
  CUtensorMap map_qkv;
  if (!attn_map(&map_qkv, qkv, 3 * H * D, B * T, BQ)) return -1;
  static const bool attr_set =
      cudaFuncSetAttribute(attention_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) == cudaSuccess;
  if (!attr_set) return -1;
  AttnParams p{};
  p.out = static_cast<__nv_bfloat16 *>(out);
  p.lse = lse;
  p.B = static_cast<int>(B);
  p.T = static_cast<int>(T);
  p.H = static_cast<int>(H);
  p.negate = scale < 0.f ? 1 : 0;
  p.scale = scale_magnitude(scale);
  p.scale_log2e = p.scale * 1.4426950408889634f;
  p.status = attn_status_ptr();
  p.causal = causal ? 1 : 0;
  attention_fwd_kernel<<<static_cast<unsigned>(T / BQ * H * B), THREADS, SMEM_BYTES, static_cast<cudaStream_t>(stream)>>>(map_qkv, p);
  return finish_launch(1);
}

int attention_backward_packed(stream_t stream, const void *qkv, const void *out, const void *dout, const float *lse, float *delta,
                              void *dqkv, int64_t B, int64_t T, int64_t H, int64_t D, float scale, int causal) {
  if (D != HD || T % 128 != 0 || B <= 0 || H <= 0 || T <= 0) return -1;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) |
       reinterpret_cast<uintptr_t>(dqkv) | reinterpret_cast<uintptr_t>(lse) | reinterpret_cast<uintptr_t>(delta)) & 15)
    return -1;
  static const bool disabled = std::getenv("CS_DISABLE_TCGEN05_ATTENTION") != nullptr;
  if (disabled) return -1;
  CUtensorMap qkv_r, qkv_c, do_r, do_c;
  if (!attn_map(&qkv_r, qkv, 3 * H * D, B * T, 128) || !attn_map(&qkv_c, qkv, 3 * H * D, B * T, BC) ||
      !attn_map(&do_r, dout, H * D, B * T, 128) || !attn_map(&do_c, dout, H * D, B * T, BC))
    return -1;
  static const bool attr_set =
      cudaFuncSetAttribute(attention_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM_BYTES) == cudaSuccess &&
      cudaFuncSetAttribute(attention_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM_BYTES) == cudaSuccess;
  if (!attr_set) return -1;
  auto s = static_cast<cudaStream_t>(stream);
  const long long threads = B * T * H * 8;
  attention_delta_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, s>>>(
      static_cast<const __nv_bfloat16 *>(out), static_cast<const __nv_bfloat16 *>(dout), lse, delta, static_cast<int>(B),
      static_cast<int>(T), static_cast<int>(H));
  AttnBwdParams p{};
  p.dqkv = static_cast<__nv_bfloat16 *>(dqkv);
  p.neg_lse = delta + B * H * T;        // plane 1 of the workspace: -lse * log2(e)
  p.neg_delta = delta + 2 * B * H * T;  // plane 2: -delta
  p.B = static_cast<int>(B);
  p.T = static_cast<int>(T);
  p.H = static_cast<int>(H);
  p.scale = scale;
  p.scale_log2e = scale_magnitude(scale) * 1.4426950408889634f;
  p.negate = scale < 0.f ? 1 : 0;
  p.status = attn_status_ptr();
  p.causal = causal ? 1 : 0;
  const int64_t items = T / 128 * H * B;
  static const int sm_count = [] {
    int dev = 0, n = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }();
  const auto grid = static_cast<unsigned>(items < sm_count ? items : sm_count);
  attention_bwd_kernel<true><<<grid, BWD_THREADS, BWD_SMEM_BYTES, s>>>(qkv_r, qkv_c, do_r, do_c, p);
  attention_bwd_kernel<false><<<grid, BWD_THREADS, BWD_SMEM_BYTES, s>>>(qkv_r, qkv_c, do_r, do_c, p);
  return finish_launch(3);
}
CS_DEFINE_BOUNDS_GETTER(bounds_report_attention)
}  // namespace cs::kernels
