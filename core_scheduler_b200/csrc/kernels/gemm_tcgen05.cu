// SPDX-License-Identifier: Apache-2.0
// bf16 GEMM on the 5th-generation tensor cores (tcgen05) with fp32 accumulators in tensor
// memory (TMEM), operands staged in shared memory by TMA, and fused epilogues.
//
//   D[M,N] = A * B^T     kTN: A [M,K] and B [N,K] row-major (K contiguous)   forward
//                        kNT: A [K,M] and B [K,N] row-major (M/N contiguous) weight gradient
//                        kTM: A [M,K] row-major, B [K,N] row-major           input gradient (dY * W)
//
// Structure (one persistent CTA per SM, 320 threads; clusters of two CTAs share a 256-row tile):
//   warp 0      TMA producer: cp.async.bulk.tensor tiles -> shared-memory ring of five to seven stages
//   warp 1      allocates TMEM and issues tcgen05.mma (leader CTA); two accumulators, so that the epilogue of
//               tile i overlaps the main loop of tile i+1
//   warps 2-9   epilogue: tcgen05.ld the accumulator (each warp owns a 32-row lane quadrant and half of the
//               columns), apply the fused op, TMA-store to global memory
// Shared-memory tiles use the 128-byte swizzle; the K-major operands of kTN are described to
// the MMA with SBO = 1024 B (8 rows x 128 B), the MN-major operands of kNT with LBO = 8192 B
// (next 64-element block) and SBO = 1024 B (next 8 k-rows).
// Every mbarrier wait is bounded: a wait that runs out raises an abort flag, the CTA drains,
// frees its TMEM and returns; the host sees DeviceStatus.code != 0.
//
// What it replaces in the reference project: the cuBLAS calls behind at::linear / at::matmul in
// src/compute/linear.cpp:178-207,245,286-296 and the cuDNN-frontend fused graphs of
// src/compute/gelu_linear_cudnn.cpp:123-311 (GELU+matmul, matmul+GELU', GELU+wgrad), plus the
// log_softmax pass of src/compute/cross_entropy.cpp:57-63 (folded into the classifier epilogue).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "api.h"
#include "bounds_check.h"
#include "collectives.h"
#include "tensor_map.h"

namespace cs::kernels {
namespace {
constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr long long kWaitBudgetCycles = 4000000000LL;  // ~2 s at 2 GHz

struct KParams {
  const void *bias;
  float *stats;
  long long stats_len;  // floats in `stats`
  long long m, n, n_valid;
  int layout, epilogue;
  int m_tiles, n_tiles, splits, kb_total, kb_per_split;
  int group_m;         // pair kernel: row tiles that are walked together before the next column tile
  int atomic_out;     // fp32 output accumulated with red.global.add (split-K or accumulate mode)
  unsigned lbo_mn, sbo_mn, kstep_mn;  // MN-major descriptor parameters (bytes)
  int peer_mode;       // 0 none, 1 = A row blocks come from peers, 2 = D row blocks go to peers,
                       // 3 = A is local but arrives in row chunks announced by flags (all-gather in flight)
  int peer_rank, peer_count;
  int rows_per_peer;
  const uint32_t *ready_flags;  // peer_mode 3: word [owner * 8 + chunk] reaches ready_epoch when that chunk has landed
  uint32_t ready_epoch;
  int ready_chunks;             // chunks per owner (rows_per_peer / ready_chunks rows each, a multiple of 256)
  DeviceStatus *status;
};

struct PeerMaps {
  CUtensorMap m[8];
};

__device__ DeviceStatus g_gemm_status;

// ------------------------------------------------------------------------- PTX helpers ----
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
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
// Bounded wait: false when the budget ran out or another role already aborted.
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
// The tensor-core and TMA instructions take their operands from uniform registers. In a branch that one lane took on its own
// (`if (lane == 0)`) the compiler has to move every operand there again for each instruction: 79 cycles an MMA and 220
// cycles a k-block of TMA loads were measured, more than the tensor core needs for a tile of 128 columns. So a role's whole
// warp walks its loop in step and elects a lane only around the instructions themselves, without another branch inside
// (one there brings the 85 cycles back); waits are voted on, which keeps the control flow uniform when one is abandoned.
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
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_ld_32x32b_x32(uint32_t taddr, uint32_t (&v)[32]) {
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
__device__ __forceinline__ void tcgen05_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor (tcgen05): start address, leading/stride byte offsets in
// 16-byte units, descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t desc = 0;
  desc |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  desc |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  desc |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  desc |= static_cast<uint64_t>(1) << 46;  // version
  desc |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return desc;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&t);
}

struct TileCoord {
  int m0, n0, kb_begin, kb_end, n_tile;
};
// ----------------------------------------------------- epilogue through shared memory + TMA ----
// The accumulator rows a thread reads from TMEM are 64-byte pieces of different output rows;
// storing them directly makes every store instruction touch 32 half-filled sectors. Instead each
// epilogue warp stages 32 rows x 128 bytes in shared memory (128-byte swizzle, conflict-free
// for 16-byte accesses) and one lane issues a TMA store (or, for fp32 gradients, a TMA
// reduce-add) of that box: full 128-byte lines, bounds clipped by the tensor map.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap *map, uint32_t src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

constexpr int EPI_BUF_BYTES = 4096;  // 32 rows x 128 bytes
constexpr int EPI_STAGING_BYTES = EPI_WARPS * 2 * EPI_BUF_BYTES;

struct EpilogueStaging {
  uint32_t base;  // shared-memory address of this warp's two staging boxes
  uint32_t next;  // byte offset of the one the next fill uses
};

// Claims a staging box: the TMA operation that last read it (two fills ago) must have finished
// reading shared memory.
__device__ __forceinline__ uint32_t staging_acquire(EpilogueStaging &st, int lane) {
  if (lane == 0) bulk_wait_read_1();
  __syncwarp();
  const uint32_t b = st.base + st.next;
  st.next ^= EPI_BUF_BYTES;
  return b;
}
// 16-byte piece `piece` (0..7) of row `lane` inside a swizzled 32 x 128-byte box.
__device__ __forceinline__ uint32_t staging_addr(uint32_t box, int lane, int piece) {
  return box + lane * 128 + ((piece ^ (lane & 7)) << 4);
}
// Makes the box visible to the async proxy and lets lane 0 issue the store / reduce.
__device__ __forceinline__ void staging_release(const CUtensorMap *map, uint32_t box, int c0, int c1, bool in_range, bool reduce,
                                                int lane) {
  fence_async_smem();
  __syncwarp();
  if (lane == 0) {
    if (in_range) {
      if (reduce)
        tma_reduce_add_2d(map, box, c0, c1);
      else
        tma_store_2d(map, box, c0, c1);
    }
    bulk_commit();  // an empty group keeps the acquire/commit pairing uniform
  }
}

// Packed fp32 pairs: sm_100 issues two fp32 FMAs per lane with one instruction, which halves what the GELU and
// softmax epilogues spend on issue slots. Same IEEE rounding as the scalar operations.
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
__device__ __forceinline__ F2 f2_unpack_bf16(uint32_t u) { return f2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The same approximation as gelu_math.h (Abramowitz & Stegun 7.1.26), two elements at a time. With
// u = (1 - erf(|x|/sqrt2)) / 2 = h(t) e,  t = 1 / (1 + 0.3275911 |x|/sqrt2),  e = exp(-x^2/2):
//   GELU(x)  = max(x, 0) - |x| u            GELU'(x) = 1/2 + copysign(1/2 - u, x) + x e / sqrt(2 pi)
// h is half the published polynomial. Without the "1 +" of the direct form there is no cancellation for x < 0.
__device__ __forceinline__ void gelu_tail_pair(F2 ax, F2 x, F2 &h, F2 &e) {
  float d0, d1, t0, t1, q0, q1;
  f2_split(f2_fma(ax, f2(0.3275911f * 0.70710678118654752440f, 0.3275911f * 0.70710678118654752440f), f2(1.f, 1.f)), d0, d1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(d1));
  const F2 t = f2(t0, t1);
  F2 poly = f2_fma(f2(0.5f * 1.061405429f, 0.5f * 1.061405429f), t, f2(0.5f * -1.453152027f, 0.5f * -1.453152027f));
  poly = f2_fma(poly, t, f2(0.5f * 1.421413741f, 0.5f * 1.421413741f));
  poly = f2_fma(poly, t, f2(0.5f * -0.284496736f, 0.5f * -0.284496736f));
  poly = f2_fma(poly, t, f2(0.5f * 0.254829592f, 0.5f * 0.254829592f));
  h = f2_mul(poly, t);
  f2_split(f2_mul(f2_mul(x, x), f2(-0.5f * 1.4426950408889634f, -0.5f * 1.4426950408889634f)), q0, q1);
  e = f2(ex2_approx(q0), ex2_approx(q1));
}
// |x| for the tails, where both are zero from 14 on: the bound keeps 0 * inf out of them.
__device__ __forceinline__ F2 gelu_abs(float a, float b) { return f2(fminf(fabsf(a), 64.f), fminf(fabsf(b), 64.f)); }
__device__ __forceinline__ uint32_t gelu_pack(float a, float b) {
  const F2 x = f2(a, b), ax = gelu_abs(a, b);
  F2 h, e;
  gelu_tail_pair(ax, x, h, e);
  float w0, w1, e0, e1;
  f2_split(f2_mul(ax, h), w0, w1);
  f2_split(e, e0, e1);
  return pack_bf16(fmaf(-w0, e0, fmaxf(a, 0.f)), fmaf(-w1, e1, fmaxf(b, 0.f)));
}
__device__ __forceinline__ F2 gelu_grad_pair(F2 x) {
  F2 h, e;
  float h0, h1, e0, e1, x0, x1;
  f2_split(x, x0, x1);
  gelu_tail_pair(gelu_abs(x0, x1), x, h, e);
  f2_split(h, h0, h1);
  f2_split(e, e0, e1);
  const F2 c = f2(0.5f + copysignf(fmaf(-h0, e0, 0.5f), x0), 0.5f + copysignf(fmaf(-h1, e1, 0.5f), x1));
  return f2_fma(f2_mul(x, f2(0.39894228040143267794f, 0.39894228040143267794f)), e, c);
}

__device__ __forceinline__ void ld_shared_v4(uint32_t addr, uint32_t (&w)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}

template <int EPI>
constexpr bool epi_uses_aux = EPI == kEpiResidualBf16 || EPI == kEpiDGelu;
template <int EPI>
constexpr bool epi_is_f32 = EPI == kEpiStoreF32;
// Columns of the tile one epilogue warp handles: half the tile, but never less than one 128-byte box.
template <int TN, int EPI>
constexpr int epi_cols = epi_is_f32<EPI> ? TN / 2 : (TN >= 128 ? TN / 2 : 64);

// Auxiliary operand (residual / pre-activation) of one warp's part of a tile: TMA-loaded into the warp's staging boxes,
// where the result overwrites it. A thread that reads its own row from global memory instead touches 32 rows per load
// instruction. Called by lane 0, with every earlier store of the warp out of the boxes.
template <int TN, int EPI>
__device__ __forceinline__ void aux_prefetch(const CUtensorMap *map_aux, uint32_t box, uint32_t aux_bar, int row0, int col0) {
#pragma unroll
  for (int g = 0; g < epi_cols<TN, EPI> / 64; ++g) {
    mbar_expect_tx(aux_bar + 8u * g, EPI_BUF_BYTES);
    tma_load_2d(box + g * EPI_BUF_BYTES, map_aux, aux_bar + 8u * g, col0 + g * 64, row0);
  }
}

// One warp's share of a finished accumulator of the pair kernel: 32 rows of lane quadrant q, epi_cols() columns. What the
// epilogue does is a template parameter: the softmax and GELU forms are bound by issue slots (13 K cycles a tile with
// everything decided at run time, against 6 K cycles of tensor-core work for K = 768), and so is what they overlap with.
// The TMEM load of the next 32 columns is in flight while the current ones are processed, and the accumulator goes back to
// the MMA warp (`release`) as soon as its last column sits in registers.
template <int TN, int EPI, typename Release>
__device__ __forceinline__ bool epilogue_pair_tile(const KParams &p, const CUtensorMap *map_d, const CUtensorMap *map_d2, int m0, int n0,
                                                   int n_tile, uint32_t tmem_acc, int q, int half, int lane, EpilogueStaging &st,
                                                   int store_row_base, uint32_t aux_bar, uint32_t aux_parity, volatile int *abort_flag,
                                                   Release release) {
  constexpr int COLS = epi_cols<TN, EPI>;
  constexpr int CHUNKS = COLS / 32;
  const int row0 = m0 + q * 32;
  const bool rows_in_range = row0 < p.m;
  const int col_base = COLS * half;
  const uint32_t taddr = tmem_acc + col_base + (static_cast<uint32_t>(q * 32) << 16);
  uint32_t acc[2][32];
  tcgen05_ld_32x32b_x32(taddr, acc[0]);
  float run_max = -INFINITY, run_sum = 0.f;  // softmax partials
  uint32_t box = 0;
#pragma unroll
  for (int ch = 0; ch < CHUNKS; ++ch) {
    uint32_t(&v)[32] = acc[ch & 1];
    tcgen05_wait_ld();
    if (ch + 1 < CHUNKS) {
      tcgen05_ld_32x32b_x32(taddr + (ch + 1) * 32, acc[(ch + 1) & 1]);
    } else {
      release();
    }
    const int gcol = n0 + col_base + ch * 32;
    if constexpr (epi_is_f32<EPI>) {
      box = staging_acquire(st, lane);
#pragma unroll
      for (int g = 0; g < 8; ++g) st_shared_v4(staging_addr(box, lane, g), v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
      staging_release(map_d, box, gcol, row0 - store_row_base, rows_in_range && gcol < p.n, p.atomic_out || p.epilogue == kEpiAccumF32, lane);
    } else {
      const int sub = ch & 1;  // two 32-column chunks share one 64-column (128-byte) box
      if (EPI != kEpiDGelu && EPI != kEpiCrossEntropy && p.bias && gcol < p.n) {
        const uint4 *bp = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(p.bias) + gcol);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (gcol + g * 8 + 8 > p.n) break;
          const uint4 b = __ldg(bp + g);
          const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float s0, s1;
            f2_split(f2_add(f2(__uint_as_float(v[g * 8 + 2 * i]), __uint_as_float(v[g * 8 + 2 * i + 1])), f2_unpack_bf16(w[i])), s0, s1);
            v[g * 8 + 2 * i] = __float_as_uint(s0);
            v[g * 8 + 2 * i + 1] = __float_as_uint(s1);
          }
        }
      }
      if constexpr (epi_uses_aux<EPI>) {
        if (sub == 0) {
          box = st.base + (ch >> 1) * EPI_BUF_BYTES;
          if (!mbar_wait_warp(aux_bar + 8u * (ch >> 1), aux_parity, abort_flag)) {
            tcgen05_wait_ld();  // no load may be outstanding when the kernel unwinds
            return false;
          }
        }
        // all loads, all arithmetic, all stores: sixteen independent pairs hide each other's latency
        uint32_t w[4][4];
#pragma unroll
        for (int g = 0; g < 4; ++g) ld_shared_v4(staging_addr(box, lane, sub * 4 + g), w[g]);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const F2 a = f2_unpack_bf16(w[i >> 2][i & 3]);
          const F2 x = f2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
          float s0, s1;
          f2_split(EPI == kEpiResidualBf16 ? f2_add(x, a) : f2_mul(x, gelu_grad_pair(a)), s0, s1);
          w[i >> 2][i & 3] = pack_bf16(s0, s1);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) st_shared_v4(staging_addr(box, lane, sub * 4 + g), w[g][0], w[g][1], w[g][2], w[g][3]);
      } else {
        uint32_t packed[16], activated[EPI == kEpiGeluDual ? 16 : 1];
#pragma unroll
        for (int i = 0; i < 16; ++i) packed[i] = pack_bf16(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        if constexpr (EPI == kEpiGeluDual) {
#pragma unroll
          for (int i = 0; i < 16; ++i) activated[i] = gelu_pack(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        }
        if (sub == 0) {
          if constexpr (EPI == kEpiGeluDual) {  // both boxes, whose stores have had the time of the arithmetic above
            if (lane == 0) bulk_wait_read_0();
            __syncwarp();
            box = st.base;
          } else {
            box = staging_acquire(st, lane);
          }
        }
#pragma unroll
        for (int g = 0; g < 4; ++g)
          st_shared_v4(staging_addr(box, lane, sub * 4 + g), packed[4 * g], packed[4 * g + 1], packed[4 * g + 2], packed[4 * g + 3]);
        if constexpr (EPI == kEpiGeluDual) {
#pragma unroll
          for (int g = 0; g < 4; ++g)
            st_shared_v4(staging_addr(box + EPI_BUF_BYTES, lane, sub * 4 + g), activated[4 * g], activated[4 * g + 1], activated[4 * g + 2],
                         activated[4 * g + 3]);
        }
        if constexpr (EPI == kEpiCrossEntropy) {
          // Running (max, sum-exp) over the valid columns, on the logits as stored (bf16). Exponents are differences to the
          // maximum times log2(e), not a product minus a product: the maximum stays the bf16 value it is, and neither
          // rounding nor overflow of the products gets into the sum.
          constexpr float kLog2e = 1.4426950408889634f;
          const long long left = p.n_valid - gcol;  // valid columns of this chunk
          auto raise = [&](float cmax) {
            if (cmax > run_max) {
              run_sum *= ex2_approx((run_max - cmax) * kLog2e);  // first chunk: 0 * exp2(-inf) = 0
              run_max = cmax;
            }
          };
          if (left >= 32) {
            __nv_bfloat162 mx = *reinterpret_cast<__nv_bfloat162 *>(&packed[0]);
#pragma unroll
            for (int i = 1; i < 16; ++i) mx = __hmax2(mx, *reinterpret_cast<__nv_bfloat162 *>(&packed[i]));
            const float cmax = fmaxf(__low2float(mx), __high2float(mx));
            raise(cmax);
            if (run_max > -INFINITY) {
              const F2 scale = f2(kLog2e, kLog2e), shift = f2(-run_max, -run_max);
              F2 s0 = f2(0.f, 0.f), s1 = f2(0.f, 0.f);
#pragma unroll
              for (int i = 0; i < 16; i += 2) {
                float a, b, c, d;
                f2_split(f2_mul(f2_add(f2_unpack_bf16(packed[i]), shift), scale), a, b);
                f2_split(f2_mul(f2_add(f2_unpack_bf16(packed[i + 1]), shift), scale), c, d);
                s0 = f2_add(s0, f2(ex2_approx(a), ex2_approx(b)));
                s1 = f2_add(s1, f2(ex2_approx(c), ex2_approx(d)));
              }
              float a, b;
              f2_split(f2_add(s0, s1), a, b);
              run_sum += a + b;
            } else if (cmax != cmax) {
              run_sum = cmax;  // nothing but NaN so far: no maximum, but not an empty chunk either
            }
          } else if (left > 0) {
            float cmax = -INFINITY, nan = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float x = __uint_as_float(i & 1 ? packed[i >> 1] & 0xffff0000u : packed[i >> 1] << 16);
              if (i < left) {
                cmax = fmaxf(cmax, x);
                if (x != x) nan = x;
              }
            }
            raise(cmax);
            if (run_max > -INFINITY) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float x = __uint_as_float(i & 1 ? packed[i >> 1] & 0xffff0000u : packed[i >> 1] << 16);
                if (i < left) run_sum += ex2_approx((x - run_max) * kLog2e);
              }
            } else if (nan != nan) {
              run_sum = nan;
            }
          }
        }
      }
      if (sub == 1) {
        const int c0 = gcol - 32;
        const bool in_range = rows_in_range && c0 < p.n;
        staging_release(map_d, box, c0, row0 - store_row_base, in_range, false, lane);
        if constexpr (EPI == kEpiGeluDual) staging_release(map_d2, box + EPI_BUF_BYTES, c0, row0 - store_row_base, in_range, false, lane);
      }
    }
  }
  if constexpr (EPI == kEpiCrossEntropy) {
    const long long row = row0 + lane;
    const long long at = (row * (2LL * p.n_tiles) + 2LL * n_tile + half) * 2;
    if (row < p.m && CS_IN_BOUNDS(kKidGemmEpilogue, at + 1, p.stats_len)) {
      float *stp = p.stats + at;
      stp[0] = run_max;
      stp[1] = run_sum;
    }
  }
  return true;
}

// ===================================================================================
// A thread-block cluster of two CTAs on neighbouring SMs computes one 256 x TN tile with tcgen05.mma.cta_group::2. CTA r of
// the pair loads rows [128r, 128r+128) of the A tile and its half of the B tile (plain TMA loads, no multicast): 32 KB a CTA
// for each 256x256x64 block, where a CTA on its own would move 48 KB for 128x256x64. One row tile of up to 128 rows runs
// with the second CTA's half empty.
// The leader CTA (cluster rank 0) issues the MMAs for the pair; barriers:
//   full[s]       in the leader: the leader's producer arrives with the byte count of both
//                 CTAs, both CTAs' TMA loads complete on it
//   empty[s]      in each CTA: tcgen05.commit multicasts the arrival to both
//   tmem_full[b]  in each CTA (multicast commit); tmem_empty[b] in the leader, counted by the
//                 epilogue warps of both CTAs
// ===================================================================================
constexpr int BM2 = 256;
constexpr int BARS2_BYTES = 512;
// Per tile width TN (256, 128 or 64 columns): this CTA's half of the B tile, one stage, and as many stages as fit beside the
// epilogue's 64 KB.
template <int TN>
struct Pair {
  static constexpr int B_BYTES = TN / 2 * BK * 2;
  static constexpr int STAGE = A_BYTES + B_BYTES;              // 32 / 24 / 20 KB
  static constexpr int STAGES = TN == 256 ? 5 : (TN == 128 ? 6 : 7);
  static constexpr int SMEM = STAGES * STAGE + EPI_STAGING_BYTES + 1024 + BARS2_BYTES;
  static constexpr int TMEM = 2 * TN;                          // two accumulators
};
static_assert(Pair<256>::SMEM <= 232448 && Pair<128>::SMEM <= 232448 && Pair<64>::SMEM <= 232448, "227 KB of shared memory per block");

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t cta) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(cta));
  return out;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster_addr, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ void tcgen05_mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int TN>
__device__ __forceinline__ TileCoord tile_coord2(const KParams &p, int tile) {
  const int mn = p.m_tiles * p.n_tiles;
  const int split = tile / mn;
  const int rem = tile - split * mn;
  // groups of group_m row tiles walk all column tiles together (see the choice of group_m)
  const int group = rem / (p.group_m * p.n_tiles);
  const int in_group = rem - group * p.group_m * p.n_tiles;
  const int group_rows = min(p.group_m, p.m_tiles - group * p.group_m);
  int n_tile = in_group / group_rows;
  int m_tile = group * p.group_m + in_group - n_tile * group_rows;
  if (p.peer_mode == 3) {
    // Rows arrive chunk by chunk from every owner at once: walk the row tiles in arrival order (chunk 0 of every
    // owner starting with this rank, then chunk 1, ...) and finish all column tiles of a row tile before the next.
    const int order = rem / p.n_tiles;
    n_tile = rem - order * p.n_tiles;
    const int per_peer = p.rows_per_peer / BM2;
    const int per_chunk = per_peer / p.ready_chunks;
    const int chunk = order / (p.peer_count * per_chunk);
    const int within = order - chunk * (p.peer_count * per_chunk);
    const int owner = (within / per_chunk + p.peer_rank) % p.peer_count;
    m_tile = owner * per_peer + chunk * per_chunk + (within % per_chunk);
  } else if (p.peer_mode) {
    // walk the owners' blocks in ring order so that no two ranks hammer the same peer: gathering starts with the
    // rows this rank owns (local data is consumed while remote traffic ramps up), scattering with the next rank's
    // rows (remote traffic starts at once, the local block comes last)
    const int per_peer = p.rows_per_peer / BM2;
    m_tile = (m_tile + (p.peer_rank + (p.peer_mode == 2 ? 1 : 0)) * per_peer) % p.m_tiles;
  }
  TileCoord c;
  c.m0 = m_tile * BM2;
  c.n0 = n_tile * TN;
  c.n_tile = n_tile;
  c.kb_begin = split * p.kb_per_split;
  c.kb_end = min(p.kb_total, c.kb_begin + p.kb_per_split);
  return c;
}

// 128 registers per thread (the two wide forms with both GELU outputs spill 16 and 24 bytes at it): the SM's four register
// files are filled by warps, and a partition that holds three of this block's ten warps then still has room for two warps of a
// light kernel (collectives, AdamW), so those really run beside a resident GEMM block instead of waiting for it to retire.
// map_aux: auxiliary operand in output boxes (epilogues that have one); map_d2: second output (kEpiGeluDual).
template <int TN, int EPI>
__global__ void __maxnreg__(128)
gemm2_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
             const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_d2,
             const __grid_constant__ PeerMaps peer_maps, const KParams p) {
  constexpr int STAGES2 = Pair<TN>::STAGES, STAGE2_BYTES = Pair<TN>::STAGE;
  constexpr bool kAux = epi_uses_aux<EPI>;
  const CUtensorMap &map_aux = map_d2;  // an epilogue has an auxiliary operand or a second output, never both
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t staging_base = smem_base + STAGES2 * STAGE2_BYTES;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem_aligned + STAGES2 * STAGE2_BYTES + EPI_STAGING_BYTES);
  const uint32_t bar_base = staging_base + EPI_STAGING_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES2 + s); };
  auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * STAGES2 + b); };
  auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES2 + 2 + b); };
  auto aux_bar = [&](int w) { return bar_base + 8u * (2 * STAGES2 + 4 + 2 * w); };  // two per epilogue warp
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + 2 * STAGES2 + 4 + 2 * EPI_WARPS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * STAGES2 + 5 + 2 * EPI_WARPS);
  static_assert((2 * STAGES2 + 6 + 2 * EPI_WARPS) * 8 <= BARS2_BYTES, "barrier area");

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const bool leader = cta == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int total_tiles = p.m_tiles * p.n_tiles * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tmem_full_bar(b), 1);
      mbar_init(tmem_empty_bar(b), 2 * (epi_cols<TN, EPI> == TN ? EPI_WARPS / 2 : EPI_WARPS));  // warps that read it
    }
    if (kAux)
      for (int w = 0; w < 2 * EPI_WARPS; ++w) mbar_init(aux_bar(0) + 8u * w, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t *>(tmem_slot))),
                 "r"(Pair<TN>::TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across the pair
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp == 0) {
    // ---------------------------------------------- TMA producer (one per CTA) ----
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int ready_key = -1;
    for (int tile = pair; ok && tile < total_tiles; tile += num_pairs) {
      const TileCoord c = tile_coord2<TN>(p, tile);
      const int m0 = c.m0 + static_cast<int>(cta) * 128;         // this CTA's rows of A / D
      const int nb0 = c.n0 + static_cast<int>(cta) * (TN / 2);   // this CTA's rows of the B tile
      const CUtensorMap *rows_map = &map_a;
      int row = m0;
      if (p.peer_mode == 1) {  // all-gather fused into the load: this tile's rows live in their owner's memory
        const int owner = m0 / p.rows_per_peer;
        rows_map = &peer_maps.m[owner];
        row = m0 - owner * p.rows_per_peer;
      }
      if (p.peer_mode == 3) {
        // the rows of this tile are written by the all-gather that runs beside this kernel: wait for their chunk
        const int owner = c.m0 / p.rows_per_peer;
        const int chunk = (c.m0 - owner * p.rows_per_peer) / (p.rows_per_peer / p.ready_chunks);
        const int key = owner * 8 + chunk;
        if (key != ready_key) {
          const uint32_t *flag = p.ready_flags + key;
          const long long t0 = clock64();
          for (;;) {
            uint32_t seen;
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
            if (static_cast<int32_t>(seen - p.ready_epoch) >= 0) break;
            if (*abort_flag || clock64() - t0 > kWaitBudgetCycles) {
              *abort_flag = 1;
              ok = false;
              break;
            }
            __nanosleep(100);
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          // the chunk was written by other GPUs through the generic proxy; the loads below go through the async proxy
          asm volatile("fence.proxy.async.global;" ::: "memory");
          ready_key = key;
        }
      }
      for (int kb = c.kb_begin; kb < c.kb_end; ++kb) {
        if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        const uint32_t a_dst = smem_base + stage * STAGE2_BYTES;
        const uint32_t b_dst = a_dst + A_BYTES;
        const uint32_t full_leader = mapa_shared(full_bar(stage), 0);
        if (leader && elect_one()) mbar_expect_tx(full_bar(stage), 2 * STAGE2_BYTES);
        if (p.layout == kTN) {
          if (elect_one()) {
            tma_load_2d_pair(a_dst, rows_map, full_leader, kb * BK, row);
            tma_load_2d_pair(b_dst, &map_b, full_leader, kb * BK, nb0);
          }
        } else if (p.layout == kNT) {
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < 2; ++j) tma_load_2d_pair(a_dst + j * 8192, &map_a, full_leader, m0 + j * 64, kb * BK);
#pragma unroll
            for (int j = 0; j < TN / 128; ++j) tma_load_2d_pair(b_dst + j * 8192, &map_b, full_leader, nb0 + j * 64, kb * BK);
          }
        } else {
          if (elect_one()) {
            tma_load_2d_pair(a_dst, rows_map, full_leader, kb * BK, row);
#pragma unroll
            for (int j = 0; j < TN / 128; ++j) tma_load_2d_pair(b_dst + j * 8192, &map_b, full_leader, nb0 + j * 64, kb * BK);
          }
        }
        if (++stage == STAGES2) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (leader CTA only) ----
    if (leader) {
      const uint32_t a_major = p.layout == kNT ? 1u : 0u;
      const uint32_t b_major = p.layout == kTN ? 0u : 1u;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (a_major << 15) | (b_major << 16) |
                             (static_cast<uint32_t>(TN >> 3) << 17) | (static_cast<uint32_t>(BM2 >> 4) << 24);
      // descriptors of stage 0; a stage or a k-step further only moves the 16-byte-unit address field
      const uint64_t desc_a = make_smem_desc(smem_base, a_major ? p.lbo_mn : 16u, a_major ? p.sbo_mn : 1024u);
      const uint64_t desc_b = make_smem_desc(smem_base + A_BYTES, b_major ? p.lbo_mn : 16u, b_major ? p.sbo_mn : 1024u);
      const uint32_t kstep_a = (a_major ? p.kstep_mn : static_cast<uint32_t>(UMMA_K * 2)) >> 4;
      const uint32_t kstep_b = (b_major ? p.kstep_mn : static_cast<uint32_t>(UMMA_K * 2)) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < total_tiles; tile += num_pairs) {
        const TileCoord c = tile_coord2<TN>(p, tile);
        if (!mbar_wait_warp(tmem_empty_bar(acc), acc_phase ^ 1u, abort_flag)) break;
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TN;
        for (int kb = c.kb_begin; kb < c.kb_end; ++kb) {
          if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint64_t da = desc_a + static_cast<uint32_t>(stage * (STAGE2_BYTES >> 4));
          const uint64_t db = desc_b + static_cast<uint32_t>(stage * (STAGE2_BYTES >> 4));
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              tcgen05_mma_pair(d_tmem, da + k * kstep_a, db + k * kstep_b, idesc, (kb > c.kb_begin || k > 0) ? 1u : 0u);
            tcgen05_commit_pair(empty_bar(stage));
          }
          if (kb + 1 == c.kb_end && elect_one()) tcgen05_commit_pair(tmem_full_bar(acc));
          if (++stage == STAGES2) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------- epilogue (each CTA) ----
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    EpilogueStaging st;
    st.base = staging_base + (warp - 2) * 2 * EPI_BUF_BYTES;
    st.next = 0;
    constexpr int COLS = epi_cols<TN, EPI>;
    const bool has_part = half * COLS < TN;  // a 64-column tile has work for one half of the warps only
    uint32_t aux_parity = 0;
    auto prefetch = [&](int tile) {
      if (kAux && lane == 0 && tile < total_tiles) {
        const TileCoord c = tile_coord2<TN>(p, tile);
        aux_prefetch<TN, EPI>(&map_aux, st.base, aux_bar(warp - 2), c.m0 + static_cast<int>(cta) * 128 + q * 32, c.n0 + half * COLS);
      }
    };
    if (has_part) {
      if constexpr (kAux) prefetch(pair);
      for (int tile = pair; tile < total_tiles; tile += num_pairs) {
        const TileCoord c = tile_coord2<TN>(p, tile);
        const int m0_cta = c.m0 + static_cast<int>(cta) * 128;
        if (!mbar_wait_warp(tmem_full_bar(acc), acc_phase, abort_flag)) break;
        tcgen05_fence_after();
        auto release = [&] {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(tmem_empty_bar(acc), 0));
        };
        const CUtensorMap *out = &map_d;
        int store_base = 0;
        if (p.peer_mode == 2) {  // reduce-scatter fused into the epilogue: this tile goes to the owner of its rows
          const int owner = m0_cta / p.rows_per_peer;
          out = &peer_maps.m[owner];
          store_base = owner * p.rows_per_peer;
        }
        if (!epilogue_pair_tile<TN, EPI>(p, out, &map_d2, m0_cta, c.n0, c.n_tile, tmem_base + acc * TN, q, half, lane, st, store_base,
                                         aux_bar(warp - 2), aux_parity, abort_flag, release))
          break;
        if constexpr (kAux) {
          if (lane == 0) bulk_wait_read_0();  // the boxes are free again: fetch the next tile's operand behind its main loop
          prefetch(tile + num_pairs);
          aux_parity ^= 1u;
        }
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    // the shared memory must outlive the stores that read it; stores into peers are complete before the block ends
    if (lane == 0) {
      if (p.peer_mode == 2)
        bulk_wait_all();
      else
        bulk_wait_read_0();
    }
  }

  // ------------------------------------------------------------------------- teardown ----
  abort_grace(abort_flag);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer may still be signalling our barriers or reading our shared memory
  if (threadIdx.x == 0 && *abort_flag) {
    p.status->code = 1;
    p.status->kernel_id = 2;
    p.status->block = blockIdx.x;
    p.status->detail = p.layout;
  }
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Pair<TN>::TMEM) : "memory");
  }
}

}  // namespace

// ------------------------------------------------------------------ host: tensor maps ----
bool get_tensor_map(const void *ptr, uint64_t inner, uint64_t outer, uint64_t stride_elems, uint32_t box_inner,
                    uint32_t box_outer, CUtensorMap *out, int elem_bytes) {
  static const TensorMapEncodeFn encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      return static_cast<TensorMapEncodeFn>(nullptr);
    }
    return reinterpret_cast<TensorMapEncodeFn>(fn);
  }();
  static TensorMapCache cache;
  return cache.get(encode, TensorMapKey{ptr, inner, outer, stride_elems * elem_bytes, box_inner, box_outer, elem_bytes}, out);
}

namespace {
// Row tiles walked together (group_m): the pairs in flight then cover a block of group_m x (pairs / group_m) tiles, and a
// row panel of A is read from memory once per sweep over the columns. A that stays in L2 as a whole (32 MB of 126 MB, the
// rest is the other operand and the output passing through) is walked column tile by column tile, so that B streams
// through once; otherwise blocks of eight, which reads the larger operand of every classifier product once instead of
// once per column tile.
int choose_group_m(int64_t m, int64_t k, int m_tiles) {
  return m * k * 2 <= (32LL << 20) ? m_tiles : 8;
}

template <int TN, int EPI>
cudaError_t launch_pair(cudaStream_t s, int grid, const CUtensorMap &a, const CUtensorMap &b, const CUtensorMap &d, const CUtensorMap &d2,
                        const PeerMaps &peers, const KParams &p) {
  static const cudaError_t attr_set = cudaFuncSetAttribute(gemm2_kernel<TN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, Pair<TN>::SMEM);
  if (attr_set != cudaSuccess) return attr_set;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = Pair<TN>::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm2_kernel<TN, EPI>, a, b, d, d2, peers, p);
}
template <int TN>
cudaError_t launch_pair_epi(int epi, cudaStream_t s, int grid, const CUtensorMap &a, const CUtensorMap &b, const CUtensorMap &d,
                            const CUtensorMap &d2, const PeerMaps &peers, const KParams &p) {
  switch (epi) {
    case kEpiStoreBf16: return launch_pair<TN, kEpiStoreBf16>(s, grid, a, b, d, d2, peers, p);
    case kEpiResidualBf16: return launch_pair<TN, kEpiResidualBf16>(s, grid, a, b, d, d2, peers, p);
    case kEpiGeluDual: return launch_pair<TN, kEpiGeluDual>(s, grid, a, b, d, d2, peers, p);
    case kEpiDGelu: return launch_pair<TN, kEpiDGelu>(s, grid, a, b, d, d2, peers, p);
    default: break;
  }
  if constexpr (TN == 256) {  // choose_tile_n narrows bf16 outputs only, and not the classifier's
    if (epi == kEpiStoreF32 || epi == kEpiAccumF32) return launch_pair<TN, kEpiStoreF32>(s, grid, a, b, d, d2, peers, p);
    if (epi == kEpiCrossEntropy) return launch_pair<TN, kEpiCrossEntropy>(s, grid, a, b, d, d2, peers, p);
  }
  return cudaErrorInvalidValue;
}

// Weight gradients have few output tiles and a long reduction: split K so that every SM has work; partial sums meet in the
// fp32 output through vector atomics. The split count whose tile total fills whole waves of the pairs best, with at least 8
// k-blocks per split; ties go to fewer splits (fewer reduce-adds).
int64_t choose_splits(int64_t tiles, int64_t k_blocks, int pairs) {
  int64_t best = 1;
  double best_eff = 0.0;
  for (int64_t sp = 1; sp <= k_blocks / 8 || sp == 1; ++sp) {
    const int64_t total = tiles * sp, waves = (total + pairs - 1) / pairs;
    const double eff = static_cast<double>(total) / (static_cast<double>(waves) * pairs);
    if (eff > best_eff + 0.02) {
      best_eff = eff;
      best = sp;
    }
    if (total >= 4 * pairs || sp == 64) break;
  }
  return best;
}

// Width of the pair kernel's tile. A k-block of 64 costs a pair 2 TN cycles of tensor core or 256 + TN cycles of operand
// traffic (64 bytes a cycle and SM, what the 8192^3 product sustains), whichever is more; a narrower tile pays only where
// the wide ones leave pairs without work. Measured with 256 / 128 / 64 columns: 1536x768x3072 21.2 / 13.6 / 13.4 us,
// 1536x2304x768 10.8 / 10.6 / 12.0, 3000x5120x1280 42.0 / 43.5 / 57.2, 16384x768x3072 60.5 / 65.9 / 92.6.
//
// An input gradient (kTM) runs beside the weight gradient of its layer, which is as large the other way round. Where that
// leaves pairs free and 256-column tiles fit into them, narrower ones that do not only make the two take turns: forward and
// backward of 1200 x 1024 x 3072 take 43 us with 40 narrow tiles beside 48, 37 with 20 wide ones (1500 x 768 x 2304: 38 and 32.5).
int choose_tile_n(const GemmArgs &a, int pairs, bool fixed) {
  if (fixed) return 256;
  int best = 256;
  double best_cost = 0;
  int64_t beside = INT64_MAX;  // tiles that narrowing may lead to
  if (a.layout == kTM) {
    const int64_t blocks = (a.k + BM2 - 1) / BM2 * ((a.n + BN - 1) / BN);
    const int64_t free_pairs = pairs - blocks * choose_splits(blocks, (a.m + BK - 1) / BK, pairs);
    if ((a.m + BM2 - 1) / BM2 * ((a.n + BN - 1) / BN) <= free_pairs) beside = free_pairs;
  }
  for (int tn = 256; tn >= 64; tn /= 2) {
    if (tn == 64 && a.layout != kTN) break;  // an MN-major half tile of 32 columns is no whole swizzle atom
    const int64_t tiles = ((a.m + BM2 - 1) / BM2) * ((a.n + tn - 1) / tn);
    if (tn < 256 && tiles > beside) break;
    const int64_t waves = (tiles + pairs - 1) / pairs;
    const double cost = static_cast<double>(waves) * (2 * tn > 256 + tn ? 2 * tn : 256 + tn);
    if (tn == 256 || cost < 0.95 * best_cost) {
      best = tn;
      best_cost = cost;
    }
  }
  return best;
}
}  // namespace

int64_t gemm_ce_stat_tiles(int64_t n) { return 2 * ((n + BN - 1) / BN); }  // one (max, sum) pair per 128-column half tile

int gemm_status(DeviceStatus *out) {
  return static_cast<int>(cudaMemcpyFromSymbol(out, g_gemm_status, sizeof(DeviceStatus)));
}
int gemm_status_reset() {
  DeviceStatus zero{};
  return static_cast<int>(cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(DeviceStatus)));
}

int gemm_bf16(stream_t stream, const GemmArgs &a) {
  auto s = static_cast<cudaStream_t>(stream);
  if (a.m <= 0 || a.n <= 0 || a.k <= 0) return -1;
  if (a.n % 8 != 0 || a.ldd % 8 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0) return -1;
  if ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b) | reinterpret_cast<uintptr_t>(a.d)) & 15) return -1;
  if (!a.b || (!a.a && !(a.peer_count > 1 && a.a_peers[0])) || (!a.d && !(a.peer_count > 1 && a.d_peers[0]))) return -1;
  if (a.aux && (reinterpret_cast<uintptr_t>(a.aux) & 15)) return -1;
  if (a.d2 && (reinterpret_cast<uintptr_t>(a.d2) & 15)) return -1;
  if (a.bias && (reinterpret_cast<uintptr_t>(a.bias) & 15)) return -1;
  const bool f32_out = a.epilogue == kEpiStoreF32 || a.epilogue == kEpiAccumF32;
  if (a.layout != kNT && a.k % 8 != 0) return -1;
  if (a.layout < 0 || a.layout > kTM) return -1;
  if (a.layout == kNT && (a.m % 8 != 0)) return -1;
  if (f32_out && a.n % 4 != 0) return -1;
  if (a.m > 0x7fffffffLL || a.n > 0x7fffffffLL || a.k > 0x7fffffffLL) return -1;
  static const bool disabled = std::getenv("CS_DISABLE_TCGEN05_GEMM") != nullptr;
  if (disabled) return -1;

  static const int sm_count = [] {
    int dev = 0, n = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }();
  const bool peers_used = a.peer_count > 1;
  const int tn = choose_tile_n(a, sm_count / 2, peers_used || f32_out || a.epilogue == kEpiCrossEntropy);
  const uint32_t b_box_rows = static_cast<uint32_t>(tn / 2);
  PeerMaps peer_maps{};
  int peer_mode = 0;
  int rows_per_peer = 0;
  if (a.peer_count > 1) {
    if (a.peer_count > 8 || a.m % a.peer_count != 0) return -1;
    rows_per_peer = static_cast<int>(a.m / a.peer_count);
    if (rows_per_peer % BM2 != 0) return -1;
    if (a.a_peers[0]) {
      if (a.layout == kNT) return -1;
      peer_mode = 1;
      for (int j = 0; j < a.peer_count; ++j)
        if (!a.a_peers[j] || (reinterpret_cast<uintptr_t>(a.a_peers[j]) & 15) ||
            !get_tensor_map(a.a_peers[j], a.k, rows_per_peer, a.lda, BK, BM, &peer_maps.m[j]))
          return -1;
    } else if (a.d_peers[0]) {
      if (a.epilogue != kEpiAccumF32 && a.epilogue != kEpiStoreBf16) return -1;
      peer_mode = 2;
      const bool f32 = a.epilogue == kEpiAccumF32;
      for (int j = 0; j < a.peer_count; ++j)
        if (!a.d_peers[j] || (reinterpret_cast<uintptr_t>(a.d_peers[j]) & 15) ||
            !get_tensor_map(a.d_peers[j], a.n, rows_per_peer, a.ldd, f32 ? 32 : 64, 32, &peer_maps.m[j], f32 ? 4 : 2))
          return -1;
    } else if (a.ready_flags) {
      if (a.layout == kNT || a.ready_chunks < 1 || a.ready_chunks > 8 || rows_per_peer % (BM2 * a.ready_chunks) != 0) return -1;
      peer_mode = 3;
    }
  }
  CUtensorMap map_a, map_b;
  if (peer_mode == 1) {
    map_a = peer_maps.m[0];
  } else if (a.layout == kNT) {
    if (!get_tensor_map(a.a, a.m, a.k, a.lda, 64, BK, &map_a)) return -1;
  } else {
    if (!get_tensor_map(a.a, a.k, a.m, a.lda, BK, BM, &map_a)) return -1;
  }
  if (a.layout == kTN) {
    if (!get_tensor_map(a.b, a.k, a.n, a.ldb, BK, b_box_rows, &map_b)) return -1;
  } else {
    if (!get_tensor_map(a.b, a.n, a.k, a.ldb, 64, BK, &map_b)) return -1;
  }
  CUtensorMap map_d{}, map_d2{};
  // output boxes of the TMA-store epilogue: 32 rows x 128 bytes
  if (peer_mode == 2) {
    map_d = peer_maps.m[0];
  } else if (f32_out) {
    if (!get_tensor_map(a.d, a.n, a.m, a.ldd, 32, 32, &map_d, 4)) return -1;
  } else {
    if (!get_tensor_map(a.d, a.n, a.m, a.ldd, 64, 32, &map_d)) return -1;
  }
  map_d2 = map_d;
  if ((a.epilogue == kEpiResidualBf16 || a.epilogue == kEpiDGelu) && !get_tensor_map(a.aux, a.n, a.m, a.ldd, 64, 32, &map_d2)) return -1;
  if (a.epilogue == kEpiGeluDual && !get_tensor_map(a.d2, a.n, a.m, a.ldd, 64, 32, &map_d2)) return -1;

  KParams p{};
  p.bias = a.bias;
  p.stats = a.stats;
  p.stats_len = a.stats_len;
  p.m = a.m;
  p.n = a.n;
  p.n_valid = a.n_valid > 0 ? a.n_valid : a.n;
  p.layout = a.layout;
  p.epilogue = a.epilogue;
  p.m_tiles = static_cast<int>((a.m + BM2 - 1) / BM2);
  p.n_tiles = static_cast<int>((a.n + tn - 1) / tn);
  p.group_m = choose_group_m(a.m, a.k, p.m_tiles);
  p.kb_total = static_cast<int>((a.k + BK - 1) / BK);
  p.splits = 1;
  if (f32_out) {
    p.splits = static_cast<int>(choose_splits(static_cast<int64_t>(p.m_tiles) * p.n_tiles, p.kb_total, sm_count / 2));
  }
  p.kb_per_split = (p.kb_total + p.splits - 1) / p.splits;
  p.splits = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;
  p.atomic_out = 0;
  if (f32_out && p.splits > 1) {
    p.atomic_out = 1;
    if (a.epilogue == kEpiStoreF32) {
      // every split adds into a zeroed output
      const cudaError_t e = cudaMemset2DAsync(a.d, static_cast<size_t>(a.ldd) * 4, 0, static_cast<size_t>(a.n) * 4,
                                              static_cast<size_t>(a.m), s);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
  }
  p.peer_mode = peer_mode;
  p.peer_rank = a.peer_rank;
  p.peer_count = a.peer_count;
  p.rows_per_peer = rows_per_peer;
  if (peer_mode == 2) {
    p.splits = 1;  // the cross-rank sum happens in (or after) the destination
    p.kb_per_split = p.kb_total;
    p.atomic_out = f32_out ? 1 : 0;
  }
  p.ready_flags = a.ready_flags;
  p.ready_epoch = a.ready_epoch;
  p.ready_chunks = a.ready_chunks;
  // MN-major operand descriptors: next 64-element block 8192 B on, next 8 k-rows 1024 B on, one UMMA_K step = 16 k-rows
  p.lbo_mn = 8192;
  p.sbo_mn = 1024;
  p.kstep_mn = 2048;
  static DeviceStatus *status_ptr = [] {
    void *ptr = nullptr;
    cudaGetSymbolAddress(&ptr, g_gemm_status);
    return static_cast<DeviceStatus *>(ptr);
  }();
  p.status = status_ptr;

  const int total_tiles = p.m_tiles * p.n_tiles * p.splits;
  // a GEMM that waits for chunks of an all-gather in flight leaves SMs free for that gather's blocks
  const int pairs = (sm_count - (peer_mode == 3 ? kGatherBesideGemmBlocks : 0)) / 2;
  const int grid = 2 * (total_tiles < pairs ? total_tiles : pairs);
  const cudaError_t e = tn == 256   ? launch_pair_epi<256>(a.epilogue, s, grid, map_a, map_b, map_d, map_d2, peer_maps, p)
                        : tn == 128 ? launch_pair_epi<128>(a.epilogue, s, grid, map_a, map_b, map_d, map_d2, peer_maps, p)
                                    : launch_pair_epi<64>(a.epilogue, s, grid, map_a, map_b, map_d, map_d2, peer_maps, p);
  if (e != cudaSuccess) return static_cast<int>(e);
  return finish_launch(1);
}
CS_DEFINE_BOUNDS_GETTER(bounds_report_gemm)
}  // namespace cs::kernels
