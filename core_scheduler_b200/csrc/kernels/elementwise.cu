// SPDX-License-Identifier: Apache-2.0
// Memory-bound sm_100a kernels: AdamW, GELU, residual add, casts/transposes, LayerNorm,
// embedding, cross-entropy helpers and gradient-norm reductions. All are vectorised to 128-bit
// accesses and sized so that a launch covers the 148 SMs with several resident CTAs each.
//
// What they replace in the reference project: src/optimizer/adamw.cu:35-90 (scalar, one
// element per thread, one launch per tensor) and the ATen library calls listed for
// LayerNorm / GeLU / Embedding / CrossEntropy / clip_grad_norm in src/compute/*.cpp.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "api.h"
#include "bounds_check.h"
#include "gelu_math.h"

namespace cs::kernels {
namespace {
std::atomic<int64_t> g_launches{0};
}
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }
int finish_launch(int n) {
  count_launch(n);
  return static_cast<int>(cudaGetLastError());
}
CS_DEFINE_BOUNDS_GETTER(bounds_report_elementwise)
bool bounds_check_enabled() {
#ifdef CS_BOUNDS_CHECK
  return true;
#else
  return false;
#endif
}
int bounds_report(BoundsReport *out, bool reset) {
  *out = BoundsReport{};
  if (!bounds_check_enabled()) return 0;
  int rc = static_cast<int>(cudaDeviceSynchronize());
  if (rc != 0) return rc;
  using Getter = int (*)(BoundsReport *, bool);
  const Getter getters[] = {bounds_report_elementwise, bounds_report_collectives, bounds_report_gemm, bounds_report_attention};
  for (Getter g : getters) {
    BoundsReport r{};
    rc = g(&r, reset);
    if (rc != 0) return rc;
    if (r.code != 0 && out->code == 0) *out = r;
  }
  return 0;
}
namespace {
constexpr int kSmCount = 148;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct alignas(16) Bf16x8 {
  __nv_bfloat162 v[4];
};
__device__ __forceinline__ void unpack(const Bf16x8 &p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ Bf16x8 pack(const float (&f)[8]) {
  Bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}
__device__ __forceinline__ void load8(const void *base, int64_t elem, int dtype, float (&f)[8]) {
  if (dtype == 1) {
    unpack(*reinterpret_cast<const Bf16x8 *>(static_cast<const __nv_bfloat16 *>(base) + elem), f);
  } else {
    const float4 a = *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + elem);
    const float4 b = *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + elem + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
}

int grid_for(int64_t work_items, int threads, int max_ctas_per_sm = 8) {
  const int64_t blocks = (work_items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(kSmCount) * max_ctas_per_sm;
  return static_cast<int>(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}
}  // namespace

// ------------------------------------------------------------------------------- AdamW ----
namespace {
template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

template <typename P, typename G, int VEC>
__global__ void __launch_bounds__(256) adamw_kernel(P *__restrict__ w, const G *__restrict__ g, P *__restrict__ m,
                                                    P *__restrict__ v, P *__restrict__ vmax,
                                                    __nv_bfloat16 *__restrict__ lp, int64_t n, float lr, float b1,
                                                    float b2, float eps, float wd, float ibc1, float ibc2,
                                                    float gscale, const float *__restrict__ clip) {
  const float scale = clip ? gscale * clip[0] : gscale;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x * VEC;
  for (int64_t base = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * VEC; base < n; base += stride) {
    P wv[VEC], mv[VEC], vv[VEC], xv[VEC];
    G gv[VEC];
    const bool full = base + VEC <= n;
    if (!CS_IN_BOUNDS(kKidAdamW, base, n)) continue;
    if (full) {
      // 128-bit (fp32 x4) or 64-bit (16-bit x4) vector accesses
      using PV = typename std::conditional<sizeof(P) == 4, float4, float2>::type;
      using GV = typename std::conditional<sizeof(G) == 4, float4, float2>::type;
      *reinterpret_cast<PV *>(wv) = *reinterpret_cast<const PV *>(w + base);
      *reinterpret_cast<PV *>(mv) = *reinterpret_cast<const PV *>(m + base);
      *reinterpret_cast<PV *>(vv) = *reinterpret_cast<const PV *>(v + base);
      *reinterpret_cast<GV *>(gv) = *reinterpret_cast<const GV *>(g + base);
      if (vmax) *reinterpret_cast<PV *>(xv) = *reinterpret_cast<const PV *>(vmax + base);
    } else {
      for (int i = 0; i < VEC; ++i) {
        if (base + i < n) {
          wv[i] = w[base + i]; mv[i] = m[base + i]; vv[i] = v[base + i]; gv[i] = g[base + i];
          if (vmax) xv[i] = vmax[base + i];
        }
      }
    }
    __nv_bfloat16 lo[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const float grad = to_f<G>(gv[i]) * scale;
      float wt = to_f<P>(wv[i]);
      wt -= lr * wd * wt;
      const float mt = b1 * to_f<P>(mv[i]) + (1.0f - b1) * grad;
      const float vt = b2 * to_f<P>(vv[i]) + (1.0f - b2) * grad * grad;
      const float mhat = mt * ibc1;
      float vhat = vt * ibc2;
      if (vmax) {
        vhat = fmaxf(to_f<P>(xv[i]), vhat);
        xv[i] = from_f<P>(vhat);
      }
      wt -= lr * mhat / (sqrtf(vhat) + eps);
      wv[i] = from_f<P>(wt);
      mv[i] = from_f<P>(mt);
      vv[i] = from_f<P>(vt);
      lo[i] = __float2bfloat16_rn(to_f<P>(wv[i]));
    }
    if (full) {
      using PV = typename std::conditional<sizeof(P) == 4, float4, float2>::type;
      *reinterpret_cast<PV *>(w + base) = *reinterpret_cast<PV *>(wv);
      *reinterpret_cast<PV *>(m + base) = *reinterpret_cast<PV *>(mv);
      *reinterpret_cast<PV *>(v + base) = *reinterpret_cast<PV *>(vv);
      if (vmax) *reinterpret_cast<PV *>(vmax + base) = *reinterpret_cast<PV *>(xv);
      if (lp) *reinterpret_cast<float2 *>(lp + base) = *reinterpret_cast<float2 *>(lo);
    } else {
      for (int i = 0; i < VEC; ++i) {
        if (base + i < n) {
          w[base + i] = wv[i]; m[base + i] = mv[i]; v[base + i] = vv[i];
          if (vmax) vmax[base + i] = xv[i];
          if (lp) lp[base + i] = lo[i];
        }
      }
    }
  }
}

template <typename P, typename G>
int launch_adamw(cudaStream_t s, const AdamWArgs &a) {
  constexpr int VEC = 4;
  // vector accesses need 16-byte (fp32) / 8-byte (16-bit) alignment of every base pointer
  const uintptr_t mask = (reinterpret_cast<uintptr_t>(a.param) | reinterpret_cast<uintptr_t>(a.grad) |
                          reinterpret_cast<uintptr_t>(a.exp_avg) | reinterpret_cast<uintptr_t>(a.exp_avg_sq) |
                          reinterpret_cast<uintptr_t>(a.max_exp_avg_sq) | reinterpret_cast<uintptr_t>(a.lp));
  const int threads = 256;
  if (mask & 15) {
    adamw_kernel<P, G, 1><<<grid_for(a.n, threads), threads, 0, s>>>(
        static_cast<P *>(a.param), static_cast<const G *>(a.grad), static_cast<P *>(a.exp_avg),
        static_cast<P *>(a.exp_avg_sq), static_cast<P *>(a.max_exp_avg_sq), static_cast<__nv_bfloat16 *>(a.lp), a.n,
        a.lr, a.beta1, a.beta2, a.eps, a.weight_decay, a.inv_bias_correction1, a.inv_bias_correction2, a.grad_scale,
        a.clip_coef);
  } else {
    adamw_kernel<P, G, VEC><<<grid_for((a.n + VEC - 1) / VEC, threads), threads, 0, s>>>(
        static_cast<P *>(a.param), static_cast<const G *>(a.grad), static_cast<P *>(a.exp_avg),
        static_cast<P *>(a.exp_avg_sq), static_cast<P *>(a.max_exp_avg_sq), static_cast<__nv_bfloat16 *>(a.lp), a.n,
        a.lr, a.beta1, a.beta2, a.eps, a.weight_decay, a.inv_bias_correction1, a.inv_bias_correction2, a.grad_scale,
        a.clip_coef);
  }
  return finish_launch();
}
}  // namespace

int adamw_step(stream_t stream, const AdamWArgs &a) {
  auto s = static_cast<cudaStream_t>(stream);
  if (a.n == 0) return 0;
  switch (a.param_dtype * 3 + a.grad_dtype) {
    case 0: return launch_adamw<float, float>(s, a);
    case 1: return launch_adamw<float, __nv_bfloat16>(s, a);
    case 2: return launch_adamw<float, __half>(s, a);
    case 4: return launch_adamw<__nv_bfloat16, __nv_bfloat16>(s, a);
    case 3: return launch_adamw<__nv_bfloat16, float>(s, a);
    case 8: return launch_adamw<__half, __half>(s, a);
    case 6: return launch_adamw<__half, float>(s, a);
    default: return static_cast<int>(cudaErrorInvalidValue);
  }
}

// ------------------------------------------------------------------ GELU / add / casts ----
namespace {
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const Bf16x8 *__restrict__ x, Bf16x8 *__restrict__ y, int64_t n8) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (!CS_IN_BOUNDS(kKidElementwise, i, n8)) continue;
    float f[8];
    unpack(x[i], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = gelu_f(f[k]);
    y[i] = pack(f);
  }
}
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const Bf16x8 *__restrict__ dy, const Bf16x8 *__restrict__ x,
                                                       Bf16x8 *__restrict__ dx, int64_t n8) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f[8], g[8];
    unpack(x[i], f);
    unpack(dy[i], g);
#pragma unroll
    for (int k = 0; k < 8; ++k) g[k] *= gelu_grad_f(f[k]);
    dx[i] = pack(g);
  }
}
__global__ void __launch_bounds__(256) add_kernel(const Bf16x8 *__restrict__ a, const Bf16x8 *__restrict__ b,
                                                  Bf16x8 *__restrict__ o, int64_t n8) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f[8], g[8];
    unpack(a[i], f);
    unpack(b[i], g);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] += g[k];
    o[i] = pack(f);
  }
}
__global__ void tail_kernel(const __nv_bfloat16 *a, const __nv_bfloat16 *b, __nv_bfloat16 *o, int64_t begin, int64_t n,
                            int mode) {
  const int64_t i = begin + threadIdx.x;
  if (i >= n) return;
  const float x = __bfloat162float(a[i]);
  if (mode == 0) o[i] = __float2bfloat16_rn(gelu_f(x));
  if (mode == 1) o[i] = __float2bfloat16_rn(x * gelu_grad_f(__bfloat162float(b[i])));  // a = dy, b = x
  if (mode == 2) o[i] = __float2bfloat16_rn(x + __bfloat162float(b[i]));
}
__global__ void __launch_bounds__(256) cast_kernel(const float *__restrict__ src, __nv_bfloat16 *__restrict__ dst, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}
// 32x32 tile transpose through shared memory; src [rows, cols] (fp32 or bf16) -> dst [cols, rows] bf16
template <typename T>
__global__ void __launch_bounds__(256) transpose_kernel(const T *__restrict__ src, __nv_bfloat16 *__restrict__ dst,
                                                        int64_t rows, int64_t cols) {
  __shared__ float tile[32][33];
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 32, c0 = static_cast<int64_t>(blockIdx.x) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t r = r0 + ty + 8 * k, c = c0 + tx;
    if (r < rows && c < cols && CS_IN_BOUNDS(kKidTranspose, r * cols + c, rows * cols)) tile[ty + 8 * k][tx] = to_f<T>(src[r * cols + c]);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t c = c0 + ty + 8 * k, r = r0 + tx;
    if (r < rows && c < cols && CS_IN_BOUNDS(kKidTranspose, c * rows + r, rows * cols)) dst[c * rows + r] = __float2bfloat16_rn(tile[tx][ty + 8 * k]);
  }
}
}  // namespace

int gelu_forward(stream_t stream, const void *x, void *y, int64_t n) {
  auto s = static_cast<cudaStream_t>(stream);
  const int64_t n8 = n / 8;
  if (n8) gelu_fwd_kernel<<<grid_for(n8, 256), 256, 0, s>>>(static_cast<const Bf16x8 *>(x), static_cast<Bf16x8 *>(y), n8);
  if (n % 8)
    tail_kernel<<<1, 8, 0, s>>>(static_cast<const __nv_bfloat16 *>(x), nullptr, static_cast<__nv_bfloat16 *>(y), n8 * 8, n, 0);
  return finish_launch();
}
int gelu_backward(stream_t stream, const void *dy, const void *x, void *dx, int64_t n) {
  auto s = static_cast<cudaStream_t>(stream);
  const int64_t n8 = n / 8;
  if (n8)
    gelu_bwd_kernel<<<grid_for(n8, 256), 256, 0, s>>>(static_cast<const Bf16x8 *>(dy), static_cast<const Bf16x8 *>(x),
                                                      static_cast<Bf16x8 *>(dx), n8);
  if (n % 8)
    tail_kernel<<<1, 8, 0, s>>>(static_cast<const __nv_bfloat16 *>(dy), static_cast<const __nv_bfloat16 *>(x),
                                static_cast<__nv_bfloat16 *>(dx), n8 * 8, n, 1);
  return finish_launch();
}
int add_bf16(stream_t stream, const void *a, const void *b, void *out, int64_t n) {
  auto s = static_cast<cudaStream_t>(stream);
  const int64_t n8 = n / 8;
  if (n8)
    add_kernel<<<grid_for(n8, 256), 256, 0, s>>>(static_cast<const Bf16x8 *>(a), static_cast<const Bf16x8 *>(b),
                                                 static_cast<Bf16x8 *>(out), n8);
  if (n % 8)
    tail_kernel<<<1, 8, 0, s>>>(static_cast<const __nv_bfloat16 *>(a), static_cast<const __nv_bfloat16 *>(b),
                                static_cast<__nv_bfloat16 *>(out), n8 * 8, n, 2);
  return finish_launch();
}
namespace {
__global__ void __launch_bounds__(256) acc_residual_kernel(const float *__restrict__ acc, const Bf16x8 *__restrict__ res,
                                                           Bf16x8 *__restrict__ out, int64_t n8) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f[8];
    load8(acc, i * 8, 0, f);
    if (res) {
      float r[8];
      unpack(res[i], r);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] += r[k];
    }
    out[i] = pack(f);
  }
}
}  // namespace

int add_f32_residual_to_bf16(stream_t stream, const float *acc, const void *residual, void *out, int64_t n) {
  if (n % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  if (n == 0) return 0;
  acc_residual_kernel<<<grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      acc, static_cast<const Bf16x8 *>(residual), static_cast<Bf16x8 *>(out), n / 8);
  return finish_launch();
}

int cast_fp32_to_bf16(stream_t stream, const float *src, void *dst, int64_t n) {
  if (n) cast_kernel<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(src, static_cast<__nv_bfloat16 *>(dst), n);
  return finish_launch();
}
int transpose_cast_to_bf16(stream_t stream, const void *src, int src_dtype, void *dst_t, int64_t rows, int64_t cols) {
  auto s = static_cast<cudaStream_t>(stream);
  dim3 grid(static_cast<unsigned>((cols + 31) / 32), static_cast<unsigned>((rows + 31) / 32));
  if (src_dtype == 0)
    transpose_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float *>(src), static_cast<__nv_bfloat16 *>(dst_t), rows, cols);
  else if (src_dtype == 1)
    transpose_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16 *>(src),
                                                         static_cast<__nv_bfloat16 *>(dst_t), rows, cols);
  else
    return static_cast<int>(cudaErrorInvalidValue);
  return finish_launch();
}

namespace {
__global__ void __launch_bounds__(256) pack_qkv_kernel(const Bf16x8 *__restrict__ q, const Bf16x8 *__restrict__ k,
                                                       const Bf16x8 *__restrict__ v, Bf16x8 *__restrict__ out, int64_t B,
                                                       int64_t H, int64_t T, int d8, int src_bthd) {
  // one thread per 16-byte piece of the output, output-major so that writes are fully coalesced
  const int64_t total = B * T * 3 * H * d8;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t r = i;
    const int c = static_cast<int>(r % d8);
    r /= d8;
    const int64_t h = r % H;
    r /= H;
    const int which = static_cast<int>(r % 3);
    r /= 3;
    const int64_t t = r % T;
    const int64_t b = r / T;
    const Bf16x8 *src = which == 0 ? q : (which == 1 ? k : v);
    const int64_t from = src_bthd ? ((b * T + t) * H + h) * d8 + c : ((b * H + h) * T + t) * d8 + c;
    if (!CS_IN_BOUNDS(kKidPackQkv, from, B * H * T * d8)) continue;
    out[i] = src[from];
  }
}
}  // namespace

int pack_qkv(stream_t stream, const void *q, const void *k, const void *v, void *packed, int64_t B, int64_t H, int64_t T,
             int64_t D, int src_bthd) {
  if (D % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  const int64_t total = B * T * 3 * H * (D / 8);
  if (total == 0) return 0;
  pack_qkv_kernel<<<grid_for(total, 256, 16), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const Bf16x8 *>(q), static_cast<const Bf16x8 *>(k), static_cast<const Bf16x8 *>(v),
      static_cast<Bf16x8 *>(packed), B, H, T, static_cast<int>(D / 8), src_bthd);
  return finish_launch();
}

// --------------------------------------------------------------------------- LayerNorm ----
namespace {
constexpr int kLnWarps = 4;       // rows per CTA iteration
constexpr int kLnRows = 4;        // rows a CTA of the forward column kernel has in flight
constexpr int kLnBwdRows = 2;     // rows a CTA of the backward kernel works on, with as many more on their way

// Rows up to 768 columns and wider than 2048: one warp per row, grid-stride over rows. Lane l owns the 8-element chunks
// l, l+32, ... of the row. The next row (still packed, in its 128-bit load registers) is fetched before the current
// one is reduced, so that loads stay in flight during the shuffles; the grid is one resident wave.
constexpr int ln_row_ctas_per_sm(int chunks) { return chunks <= 3 ? 4 : 2; }
template <int CHUNKS>
__global__ void __launch_bounds__(kLnWarps * 32, CHUNKS <= 3 ? 4 : 1)
ln_fwd_row_kernel(const __nv_bfloat16 *__restrict__ x, const void *__restrict__ gamma, const void *__restrict__ beta, int pdt,
              __nv_bfloat16 *__restrict__ y, float *__restrict__ mean, float *__restrict__ rstd, int64_t rows, int d, float eps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nchunks = d / 8;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kLnWarps;
  int64_t row = static_cast<int64_t>(blockIdx.x) * kLnWarps + warp;
  Bf16x8 cur[CHUNKS], nxt[CHUNKS];
  auto load_row = [&](Bf16x8(&dst)[CHUNKS], int64_t r) {
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int chunk = lane + 32 * c;
      if (chunk < nchunks && CS_IN_BOUNDS(kKidLayerNormFwd, r * d + chunk * 8 + 7, rows * d))
        dst[c] = *reinterpret_cast<const Bf16x8 *>(x + r * d + chunk * 8);
    }
  };
  // gamma and beta of this lane's chunks stay in registers for narrow rows (they would otherwise be
  // re-read from L1 for every row: four times the bytes of the row itself)
  constexpr bool kHoist = CHUNKS <= 3;
  float gw[kHoist ? CHUNKS : 1][8] = {}, bw[kHoist ? CHUNKS : 1][8] = {};
  if (kHoist) {
#pragma unroll
    for (int c = 0; c < (kHoist ? CHUNKS : 1); ++c) {
      const int chunk = lane + 32 * c;
      if (chunk < nchunks) {
        load8(gamma, chunk * 8, pdt, gw[c]);
        if (beta) load8(beta, chunk * 8, pdt, bw[c]);
      }
    }
  }
  if (row < rows) load_row(cur, row);
  while (row < rows) {
    const int64_t next = row + stride;
    if (next < rows) load_row(nxt, next);
    float v[CHUNKS][8];
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (lane + 32 * c < nchunks) {
        unpack(cur[c], v[c]);
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += v[c][k];
      }
    }
    const float mu = warp_sum(sum) / d;
    float sq = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (lane + 32 * c < nchunks) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float t = v[c][k] - mu;
          sq += t * t;
        }
      }
    }
    const float rs = rsqrtf(warp_sum(sq) / d + eps);
    if (lane == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int chunk = lane + 32 * c;
      if (chunk < nchunks) {
        float g[8], b[8], o[8];
        if (kHoist) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            g[k] = gw[kHoist ? c : 0][k];
            b[k] = bw[kHoist ? c : 0][k];
          }
        } else {
          load8(gamma, chunk * 8, pdt, g);
          if (beta) {
            load8(beta, chunk * 8, pdt, b);
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) b[k] = 0.f;
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = (v[c][k] - mu) * rs * g[k] + b[k];
        if (CS_IN_BOUNDS(kKidLayerNormFwd, row * d + chunk * 8 + 7, rows * d)) *reinterpret_cast<Bf16x8 *>(y + row * d + chunk * 8) = pack(o);
      }
    }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) cur[c] = nxt[c];
    row = next;
  }
}

// Rows up to 2048 columns (forward: from 776 on): thread t of a CTA owns columns 8t .. 8t+7 and the CTA takes a group of rows at
// a time. gamma, beta and the dgamma/dbeta partials of eight columns are 16 to 32 registers, whatever the width, where a warp per
// row keeps 2 x 8 partials for each of its d / 256 chunks (167 registers, 12 warps an SM) or re-reads gamma and beta from L1 for
// every row. What a row costs instead is a sum over the CTA's warps: the rows of a group share one halving butterfly, one barrier
// and 256 bytes of shared memory, little enough for a CTA to run beside a resident GEMM block. Forward takes four rows at a time;
// backward two, with the next two on their way while these meet: four without that left no load in flight between the barriers
// and was slower than a warp per row below 1000 columns. Bound by HBM, from cold caches, against a warp per row: 32768 x 1280
// forward 48 -> 44 us, backward with the residual gradient 116 -> 73 (four bf16 tensors, 51 at the copy rate); backward of
// 32768 x 768 49 -> 46, of 32768 x 256 24 -> 17, of 1024 x 768 7.6 -> 5.0.

// Sums each of N values over the warp; afterwards lane l holds the sum of value l / (32 / N). N shuffles in all but the last
// rounds instead of N in each of the five.
template <int N>
__device__ __forceinline__ float warp_sum_many(float (&v)[N], int lane) {
  int half = 16;
#pragma unroll
  for (int n = N; n > 1; n /= 2, half /= 2) {
    const bool upper = (lane & half) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float give = upper ? v[i] : v[i + n / 2], keep = upper ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
    }
  }
  float r = v[0];
#pragma unroll
  for (int o = 16 / N; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
// The same over the CTA; v[i] is replaced by the total of value i. `red` alternates between two buffers, so that one
// barrier per sum is enough.
template <int N>
__device__ __forceinline__ void cta_sum_many(float (&v)[N], float (&red)[8][N], int warp, int lane, int warps) {
  const float mine = warp_sum_many<N>(v, lane);
  if ((lane & (32 / N - 1)) == 0) red[warp][lane / (32 / N)] = mine;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = 0.f;
  for (int w = 0; w < warps; ++w) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += red[w][i];
  }
}

__global__ void __launch_bounds__(256, 4) ln_fwd_kernel(const __nv_bfloat16 *__restrict__ x, const void *__restrict__ gamma,
                                                     const void *__restrict__ beta, int pdt, __nv_bfloat16 *__restrict__ y,
                                                     float *__restrict__ mean, float *__restrict__ rstd, int64_t rows, int d, float eps) {
  __shared__ float red[2][8][kLnRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int col = threadIdx.x * 8;
  const bool active = col < d;
  float g[8], b[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) g[k] = b[k] = 0.f;
  if (active) {
    load8(gamma, col, pdt, g);
    if (beta) load8(beta, col, pdt, b);
  }
  // The mean of equal values has to be that value: rstd, up to eps^-1/2 there, makes a last bit visible. A 32-bit reciprocal is
  // off by up to 2^-25 and the product with it misses; the 64-bit product rounds to the quotient. Divisions instead cost 15 %
  // (their slow path takes registers); this costs 2 %.
  const double mean_factor = 1.0 / d;
  const float inv_d = static_cast<float>(mean_factor);
  const int64_t step = static_cast<int64_t>(gridDim.x) * kLnRows;
  for (int64_t row0 = static_cast<int64_t>(blockIdx.x) * kLnRows; row0 < rows; row0 += step) {
    Bf16x8 xp[kLnRows] = {};
    float s[kLnRows];
#pragma unroll
    for (int r = 0; r < kLnRows; ++r)
      if (active && row0 + r < rows && CS_IN_BOUNDS(kKidLayerNormFwd, (row0 + r) * d + col + 7, rows * d))
        xp[r] = *reinterpret_cast<const Bf16x8 *>(x + (row0 + r) * d + col);
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      float v[8];
      unpack(xp[r], v);
      s[r] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    }
    cta_sum_many<kLnRows>(s, red[0], warp, lane, warps);
    float mu[kLnRows];
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      mu[r] = static_cast<float>(s[r] * mean_factor);
      s[r] = 0.f;
      float v[8];
      unpack(xp[r], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) s[r] = fmaf(v[k] - mu[r], v[k] - mu[r], s[r]);
      if (!active) s[r] = 0.f;
    }
    cta_sum_many<kLnRows>(s, red[1], warp, lane, warps);
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      if (row0 + r >= rows) break;
      const float rs = rsqrtf(s[r] * inv_d + eps);
      if (threadIdx.x == 0) {
        mean[row0 + r] = mu[r];
        rstd[row0 + r] = rs;
      }
      if (active && CS_IN_BOUNDS(kKidLayerNormFwd, (row0 + r) * d + col + 7, rows * d)) {
        float v[8], o[8];
        unpack(xp[r], v);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = (v[k] - mu[r]) * rs * g[k] + b[k];
        *reinterpret_cast<Bf16x8 *>(y + (row0 + r) * d + col) = pack(o);
      }
    }
  }
}

__global__ void __launch_bounds__(256, 2) ln_bwd_kernel(const __nv_bfloat16 *__restrict__ dy, const __nv_bfloat16 *__restrict__ x,
                                                     const void *__restrict__ gamma, int pdt, const float *__restrict__ mean,
                                                     const float *__restrict__ rstd, const __nv_bfloat16 *__restrict__ dres,
                                                     __nv_bfloat16 *__restrict__ dx, float *__restrict__ scratch, int64_t rows, int d) {
  __shared__ float red[2][8][2 * kLnBwdRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int col = threadIdx.x * 8;
  const bool active = col < d;
  float g[8], dg[8], db[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) g[k] = dg[k] = db[k] = 0.f;
  if (active) load8(gamma, col, pdt, g);
  const float inv_d = 1.f / d;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kLnBwdRows;
  int buffer = 0;
  // The next rows are on their way while the sums of the present ones meet.
  Bf16x8 xn[kLnBwdRows] = {}, dn[kLnBwdRows] = {}, rn[kLnBwdRows] = {};
  float mun[kLnBwdRows], rsn[kLnBwdRows];
  auto load = [&](int64_t first) {
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      const int64_t row = first + r;
      const bool in = row < rows;
      if (in && active && CS_IN_BOUNDS(kKidLayerNormBwd, row * d + col + 7, rows * d)) {
        xn[r] = *reinterpret_cast<const Bf16x8 *>(x + row * d + col);
        dn[r] = *reinterpret_cast<const Bf16x8 *>(dy + row * d + col);
        if (dres) rn[r] = *reinterpret_cast<const Bf16x8 *>(dres + row * d + col);
      } else {
        xn[r] = dn[r] = rn[r] = Bf16x8{};
      }
      mun[r] = in ? mean[row] : 0.f;
      rsn[r] = in ? rstd[row] : 0.f;
    }
  };
  int64_t row0 = static_cast<int64_t>(blockIdx.x) * kLnBwdRows;
  load(row0);
  for (; row0 < rows; row0 += step, buffer ^= 1) {
    Bf16x8 xp[kLnBwdRows], dp[kLnBwdRows], rp[kLnBwdRows];
    float mu[kLnBwdRows], rs[kLnBwdRows], s[2 * kLnBwdRows];
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      xp[r] = xn[r];
      dp[r] = dn[r];
      rp[r] = rn[r];
      mu[r] = mun[r];
      rs[r] = rsn[r];
    }
    load(row0 + step);
    {
      float xv[kLnBwdRows][8], dv[kLnBwdRows][8], s1[kLnBwdRows] = {}, s2[kLnBwdRows] = {};
#pragma unroll
      for (int r = 0; r < kLnBwdRows; ++r) {
        unpack(xp[r], xv[r]);
        unpack(dp[r], dv[r]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float tg = 0.f, tb = 0.f;  // the rows meet before the long sums: half as many additions at their magnitude
#pragma unroll
        for (int r = 0; r < kLnBwdRows; ++r) {
          const float xh = (xv[r][k] - mu[r]) * rs[r], gy = dv[r][k] * g[k];
          s1[r] = fmaf(gy, xh, s1[r]);
          s2[r] += gy;
          tg = fmaf(dv[r][k], xh, tg);
          tb += dv[r][k];
        }
        dg[k] += tg;
        db[k] += tb;
      }
#pragma unroll
      for (int r = 0; r < kLnBwdRows; ++r) {
        s[2 * r] = active ? s1[r] : 0.f;
        s[2 * r + 1] = active ? s2[r] : 0.f;
      }
    }
    cta_sum_many<2 * kLnBwdRows>(s, red[buffer], warp, lane, warps);
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      if (row0 + r >= rows || !active) break;
      const float c1 = s[2 * r] * inv_d, c2 = s[2 * r + 1] * inv_d;
      float xv[8], dv[8], o[8];
      unpack(xp[r], xv);
      unpack(dp[r], dv);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = rs[r] * (dv[k] * g[k] - c2 - (xv[k] - mu[r]) * rs[r] * c1);
      if (dres) {
        float t[8];
        unpack(rp[r], t);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] += t[k];
      }
      if (CS_IN_BOUNDS(kKidLayerNormBwd, (row0 + r) * d + col + 7, rows * d))
        *reinterpret_cast<Bf16x8 *>(dx + (row0 + r) * d + col) = pack(o);
    }
  }
  if (active) {
    float4 *mine = reinterpret_cast<float4 *>(scratch + static_cast<int64_t>(blockIdx.x) * 2 * d + col);
    mine[0] = make_float4(dg[0], dg[1], dg[2], dg[3]);
    mine[1] = make_float4(dg[4], dg[5], dg[6], dg[7]);
    mine += d / 4;
    mine[0] = make_float4(db[0], db[1], db[2], db[3]);
    mine[1] = make_float4(db[4], db[5], db[6], db[7]);
  }
}

// Sums the CTAs' partial rows. These are up to 4.6 MB at every width (512 threads an SM with sixteen sums each), so a block takes
// few columns and many rows at once: QUADS groups of four columns, 128 / QUADS rows. 32768 rows of 768: 10.5 -> 4.6 us, where 32
// columns a block left 48 blocks to do it. Four columns (half of a 32-byte sector) are the better choice while eight would leave
// fewer blocks than SMs: 32768 rows of 256 in 7.2 us with eight, 5.2 with four. 128 threads and 128 bytes of shared memory find room
// on an SM that a GEMM block holds; with more of either a launch waited for GEMM blocks to retire.
template <int QUADS>
__global__ void __launch_bounds__(128) ln_bwd_reduce_kernel(const float *__restrict__ scratch, int parts, int d,
                                                            float *__restrict__ dgamma, float *__restrict__ dbeta, int accumulate) {
  __shared__ float4 red[4][QUADS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cq = lane % QUADS;
  const int which = blockIdx.y;  // 0 = dgamma, 1 = dbeta
  const float *src = scratch + static_cast<int64_t>(which) * d + blockIdx.x * (4 * QUADS) + cq * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int p = threadIdx.x / QUADS; p < parts; p += 128 / QUADS) {
    const float4 v = *reinterpret_cast<const float4 *>(src + static_cast<int64_t>(p) * 2 * d);
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
#pragma unroll
  for (int o = QUADS; o <= 16; o <<= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
    acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
  }
  if (lane < QUADS) red[warp][cq] = acc;
  __syncthreads();
  if (threadIdx.x < 4 * QUADS) {
    const int c = blockIdx.x * (4 * QUADS) + threadIdx.x;
    const auto part = [&](int w) { return reinterpret_cast<const float *>(red[w])[threadIdx.x]; };
    const float t = (part(0) + part(1)) + (part(2) + part(3));
    float *out = which == 0 ? dgamma : dbeta;
    out[c] = accumulate ? out[c] + t : t;
  }
}

int ln_threads(int d) { return (d / 8 + 31) / 32 * 32; }
// CTAs of the column kernels: what the SMs hold at `per_sm_threads` threads each (64 registers a thread forward, 128 backward),
// but no more than there are groups of rows or `most`.
int64_t ln_grid(int64_t rows, int d, int group, int per_sm_threads, int64_t most) {
  const int64_t wave = static_cast<int64_t>(kSmCount) * (per_sm_threads / ln_threads(d));
  const int64_t groups = (rows + group - 1) / group, cap = wave < most ? wave : most;
  return groups < cap ? groups : cap;
}
constexpr int kLnBwdThreads = 512, kLnFwdThreads = 1024;  // per SM
int launch_ln_bwd(cudaStream_t s, const void *dy, const void *x, const void *gamma, int pdt, const float *mean, const float *rstd,
                  const void *dres, void *dx, float *dgamma, float *dbeta, int accumulate, float *scratch, int64_t rows, int d,
                  int64_t scratch_rows) {
  const int parts = static_cast<int>(ln_grid(rows, d, kLnBwdRows, kLnBwdThreads, scratch_rows));
  ln_bwd_kernel<<<parts, ln_threads(d), 0, s>>>(static_cast<const __nv_bfloat16 *>(dy), static_cast<const __nv_bfloat16 *>(x), gamma,
                                                pdt, mean, rstd, static_cast<const __nv_bfloat16 *>(dres),
                                                static_cast<__nv_bfloat16 *>(dx), scratch, rows, d);
  const int code = finish_launch();
  if (code != 0) return code;
  if (d / 8 * 2 < kSmCount)
    ln_bwd_reduce_kernel<1><<<dim3(static_cast<unsigned>(d / 4), 2), 128, 0, s>>>(scratch, parts, d, dgamma, dbeta, accumulate);
  else
    ln_bwd_reduce_kernel<2><<<dim3(static_cast<unsigned>(d / 8), 2), 128, 0, s>>>(scratch, parts, d, dgamma, dbeta, accumulate);
  return finish_launch();
}

template <int CHUNKS>
int launch_ln_fwd_rows(cudaStream_t s, const void *x, const void *gamma, const void *beta, int pdt, void *y, float *mean,
                       float *rstd, int64_t rows, int d, float eps) {
  const int64_t blocks = (rows + kLnWarps - 1) / kLnWarps;
  const int64_t wave = static_cast<int64_t>(kSmCount) * ln_row_ctas_per_sm(CHUNKS);
  const int grid = static_cast<int>(blocks > wave ? wave : blocks);
  ln_fwd_row_kernel<CHUNKS><<<grid, kLnWarps * 32, 0, s>>>(static_cast<const __nv_bfloat16 *>(x), gamma, beta, pdt,
                                                            static_cast<__nv_bfloat16 *>(y), mean, rstd, rows, d, eps);
  return finish_launch();
}
}  // namespace

int layernorm_forward(stream_t stream, const void *x, const void *gamma, const void *beta, int param_dtype, void *y,
                      float *mean, float *rstd, int64_t rows, int64_t d, float eps) {
  auto s = static_cast<cudaStream_t>(stream);
  if (d % 8 != 0 || d > 8192 || rows == 0) return rows == 0 ? 0 : static_cast<int>(cudaErrorInvalidValue);
  const int chunks = static_cast<int>((d / 8 + 31) / 32);
  const int di = static_cast<int>(d);
  // The column kernel is the faster one above 768 columns (32768 x 1024: 35 against 39 us, 64 x 1024: 3.5 against 4.2), a warp per
  // row up to there (32768 x 768: 22 against 31, 32768 x 256: 13 against 21, 64 x 256: 2.7 against 3.5; all from cold caches).
  if (chunks <= 2) return launch_ln_fwd_rows<2>(s, x, gamma, beta, param_dtype, y, mean, rstd, rows, di, eps);
  if (chunks <= 3) return launch_ln_fwd_rows<3>(s, x, gamma, beta, param_dtype, y, mean, rstd, rows, di, eps);
  if (chunks > 16) return launch_ln_fwd_rows<32>(s, x, gamma, beta, param_dtype, y, mean, rstd, rows, di, eps);
  if (chunks > 8) return launch_ln_fwd_rows<16>(s, x, gamma, beta, param_dtype, y, mean, rstd, rows, di, eps);
  ln_fwd_kernel<<<static_cast<int>(ln_grid(rows, di, kLnRows, kLnFwdThreads, rows)), ln_threads(di), 0, s>>>(
      static_cast<const __nv_bfloat16 *>(x), gamma, beta, param_dtype, static_cast<__nv_bfloat16 *>(y), mean, rstd, rows, di, eps);
  return finish_launch();
}

int64_t layernorm_backward_scratch_rows(int64_t d) {
  return static_cast<int64_t>(kSmCount) * (kLnBwdThreads / ln_threads(static_cast<int>(d)));
}

int layernorm_backward(stream_t stream, const void *dy, const void *x, const void *gamma, int param_dtype,
                       const float *mean, const float *rstd, const void *grad_residual, void *dx, float *dgamma,
                       float *dbeta, int accumulate, float *scratch, int64_t rows, int64_t d) {
  auto s = static_cast<cudaStream_t>(stream);
  if (d % 8 != 0 || d > 2048) return static_cast<int>(cudaErrorInvalidValue);  // wider rows use the library path
  if (rows == 0) return 0;
  return launch_ln_bwd(s, dy, x, gamma, param_dtype, mean, rstd, grad_residual, dx, dgamma, dbeta, accumulate, scratch, rows,
                       static_cast<int>(d), layernorm_backward_scratch_rows(d));
}

// --------------------------------------------------------------------------- embedding ----
namespace {
// A warp takes 256 columns of a row at a time, so that the id is read once for them, no element pays for a division, and a piece's
// loads do not wait for the piece before. One warp for the whole row was slower at both ends: 16384 x 1280 from fp32 tables 26.4 us,
// 21.3 so; 114 x 1280 5.6 and 3.2 (cold caches). Four CTAs an SM leave room for what runs beside it: embed forward + backward of
// 16384 x 768, one pass after another, 69 us with eight and 64 with four.
__global__ void __launch_bounds__(256) embedding_fwd_kernel(const int64_t *__restrict__ idx, const void *__restrict__ wte,
                                                            const void *__restrict__ wpe, int tdt,
                                                            __nv_bfloat16 *__restrict__ out, int64_t rows,
                                                            int64_t seq_len, int d, int64_t vocab) {
  const int lane = threadIdx.x & 31, pieces = (d + 255) / 256;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5), items = rows * pieces;
  for (int64_t item = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); item < items; item += warps) {
    const int64_t row = items < INT32_MAX ? static_cast<int32_t>(item) / pieces : item / pieces;
    int64_t token = idx[row];
    (void)CS_IN_BOUNDS(kKidEmbeddingFwd, token, vocab);  // diagnostic build: remember the first bad id
    token = token < 0 ? 0 : (token >= vocab ? vocab - 1 : token);  // clamp instead of faulting
    const int64_t pos = !wpe ? 0 : (rows < INT32_MAX && seq_len < INT32_MAX ? static_cast<int32_t>(row) % static_cast<int32_t>(seq_len) : row % seq_len);
    const int col = static_cast<int>(item - row * pieces) * 256 + lane * 8;
    if (col < d) {
      float a[8];
      load8(wte, token * d + col, tdt, a);
      if (wpe) {
        float p[8];
        load8(wpe, pos * d + col, tdt, p);
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] += p[k];
      }
      *reinterpret_cast<Bf16x8 *>(out + row * d + col) = pack(a);
    }
  }
}

// One warp per row (several where rows are few), four columns per atomic: a vector reduction carries four times what a scalar one does through the same
// L2 slot, and text sends a good part of its rows to the same few ids. 16384 rows of 768, ids log-uniform over 50304:
// 143 -> 24 us. kVector: the table is 16-byte aligned.
template <bool kVector, bool kSplit>
__global__ void __launch_bounds__(256) embedding_bwd_wte_kernel(const int64_t *__restrict__ idx,
                                                                const __nv_bfloat16 *__restrict__ dy,
                                                                float *__restrict__ dwte, int64_t rows, int d,
                                                                int64_t vocab, int64_t padding_idx, int segments) {
  const int segs = kSplit ? segments : 1;
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t item = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); item < rows * segs; item += warps) {
    const int64_t row = item / segs;
    const int seg = static_cast<int>(item - row * segs);
    const int64_t token = idx[row];
    if (token != padding_idx) (void)CS_IN_BOUNDS(kKidEmbeddingBwd, token, vocab);
    if (token < 0 || token >= vocab || token == padding_idx) continue;
#pragma unroll 4
    for (int col = (seg * 32 + lane) * 4; col < d; col += 128 * segs) {
      const uint2 raw = *reinterpret_cast<const uint2 *>(dy + row * d + col);
      const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.x));
      const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.y));
      float *dst = dwte + token * d + col;
      if (kVector) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(lo.x), "f"(lo.y), "f"(hi.x), "f"(hi.y) : "memory");
      } else {
        atomicAdd(dst, lo.x);
        atomicAdd(dst + 1, lo.y);
        atomicAdd(dst + 2, hi.x);
        atomicAdd(dst + 3, hi.y);
      }
    }
  }
}

__global__ void __launch_bounds__(256) embedding_bwd_wpe_kernel(const __nv_bfloat16 *__restrict__ dy,
                                                                float *__restrict__ dwpe, int accumulate,
                                                                int64_t batch, int64_t seq_len, int d) {
  const int chunks = d / 8;
  const int64_t total = seq_len * chunks;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / chunks;
    const int chunk = static_cast<int>(i - t * chunks);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t b = 0; b < batch; ++b) {
      float g[8];
      unpack(*reinterpret_cast<const Bf16x8 *>(dy + (b * seq_len + t) * d + chunk * 8), g);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g[k];
    }
    float *dst = dwpe + t * d + chunk * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k] = accumulate ? dst[k] + acc[k] : acc[k];
  }
}
}  // namespace

int embedding_forward(stream_t stream, const int64_t *idx, const void *wte, const void *wpe, int table_dtype, void *out,
                      int64_t rows, int64_t seq_len, int64_t d, int64_t vocab) {
  if (rows == 0) return 0;
  if (d % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  embedding_fwd_kernel<<<grid_for(rows * ((d + 255) / 256) * 32, 256, 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      idx, wte, wpe, table_dtype, static_cast<__nv_bfloat16 *>(out), rows, seq_len, static_cast<int>(d), vocab);
  return finish_launch();
}

namespace {
// Warps per row: a row is split while that leaves each warp a piece and the SMs have fewer than sixteen warps each. 114 rows of
// 1280: 4.5 us with one warp each, 2.7 so (cold caches); 4096 rows of 768 gain nothing from it.
int embedding_segments(int64_t rows, int64_t d, int64_t piece) {
  int segs = 1;
  while (segs * piece < d && rows * segs < 16 * kSmCount) segs *= 2;
  return segs;
}
}  // namespace

int embedding_backward(stream_t stream, const int64_t *idx, const void *dy, float *dwte, float *dwpe, int accumulate_wpe,
                       int64_t rows, int64_t seq_len, int64_t d, int64_t vocab, int64_t padding_idx) {
  auto s = static_cast<cudaStream_t>(stream);
  if (rows == 0) return 0;
  if (d % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  if (dwte) {
    const int segs = embedding_segments(rows, d, 128);
    const bool aligned = (reinterpret_cast<uintptr_t>(dwte) & 15) == 0;
    auto *kernel = segs > 1 ? (aligned ? embedding_bwd_wte_kernel<true, true> : embedding_bwd_wte_kernel<false, true>)
                            : (aligned ? embedding_bwd_wte_kernel<true, false> : embedding_bwd_wte_kernel<false, false>);
    kernel<<<grid_for(rows * segs * 32, 256), 256, 0, s>>>(idx, static_cast<const __nv_bfloat16 *>(dy), dwte, rows, static_cast<int>(d),
                                                           vocab, padding_idx, segs);
  }
  if (dwpe)
    embedding_bwd_wpe_kernel<<<grid_for(seq_len * (d / 8), 256), 256, 0, s>>>(static_cast<const __nv_bfloat16 *>(dy), dwpe,
                                                                             accumulate_wpe, rows / seq_len, seq_len,
                                                                             static_cast<int>(d));
  return finish_launch((dwte ? 1 : 0) + (dwpe ? 1 : 0));
}

// -------------------------------------------------------------------------- column sums ----
namespace {
// Bias gradient: sums of the columns of a bf16 matrix. A block takes 64 columns (128 bytes of each row) and every
// gridDim.y-th group of 32 rows; its 32 row lanes meet in registers and shared memory, and with more than one block per
// column group the partial rows meet in a second, small launch. Terms meet in pairs at each level, so that few additions are made
// at the magnitude of the result. No atomics: the same bits every time. Bound by HBM, from cold caches against the library's
// reduction: 3000 x 5120 18 -> 9 us, 16384 x 768 31 -> 11, 16384 x 50304 272 -> 284 (four rows a step instead of two: 319).
__global__ void __launch_bounds__(256, 8) column_sum_kernel(const __nv_bfloat16 *__restrict__ x, int64_t rows, int64_t n,
                                                         float *__restrict__ out, int accumulate) {
  __shared__ float red[8][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cl = threadIdx.x & 7;
  const int64_t col = static_cast<int64_t>(blockIdx.x) * 64 + cl * 8;
  const int64_t hop = static_cast<int64_t>(gridDim.y) * 32 * n;  // to this thread's next row
  const __nv_bfloat16 *end = x + rows * n;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col < n) {
    for (const __nv_bfloat16 *at = x + (static_cast<int64_t>(blockIdx.y) * 32 + (threadIdx.x >> 3)) * n + col; at < end; at += 2 * hop) {
      Bf16x8 held[2] = {};
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (at + u * hop < end && CS_IN_BOUNDS(kKidElementwise, at + u * hop + 7 - x, rows * n))
          held[u] = *reinterpret_cast<const Bf16x8 *>(at + u * hop);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(held[0].v[i]), b = __bfloat1622float2(held[1].v[i]);
        acc[2 * i] += a.x + b.x;
        acc[2 * i + 1] += a.y + b.y;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 8);
    acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 16);
  }
  if (lane < 8) {
#pragma unroll
    for (int k = 0; k < 8; ++k) red[warp][cl * 8 + k] = acc[k];
  }
  __syncthreads();
  const int64_t c = static_cast<int64_t>(blockIdx.x) * 64 + threadIdx.x;
  if (threadIdx.x < 64 && c < n) {
    const auto part = [&](int w) { return red[w][threadIdx.x]; };
    const float t = ((part(0) + part(1)) + (part(2) + part(3))) + ((part(4) + part(5)) + (part(6) + part(7)));
    float *dst = out + static_cast<int64_t>(blockIdx.y) * n + c;
    *dst = accumulate ? *dst + t : t;
  }
}
__global__ void __launch_bounds__(128) column_sum_merge_kernel(const float *__restrict__ parts, int count, int64_t n,
                                                               float *__restrict__ out, int accumulate) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x;
  if (c >= n) return;
  float t = 0.f;
  for (int p0 = 0; p0 < count; p0 += 8) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = p0 + i < count ? parts[(p0 + i) * n + c] : 0.f;
    t += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  out[c] = accumulate ? out[c] + t : t;
}
}  // namespace

int64_t column_sum_parts(int64_t rows, int64_t n) {
  // four blocks an SM, at least 64 rows each: fewer leave nothing to overlap with the block's own reduction
  const int64_t groups = (n + 63) / 64, want = (4 * kSmCount + groups - 1) / groups, most = (rows + 63) / 64;
  const int64_t parts = want < most ? want : most;
  return parts < 1 ? 1 : (parts > 64 ? 64 : parts);
}
int column_sum(stream_t stream, const void *x, int64_t rows, int64_t n, float *out, int accumulate, float *scratch) {
  auto s = static_cast<cudaStream_t>(stream);
  if (n % 8 != 0 || rows <= 0 || n <= 0 || (reinterpret_cast<uintptr_t>(x) & 15)) return static_cast<int>(cudaErrorInvalidValue);
  const int parts = static_cast<int>(column_sum_parts(rows, n));
  const dim3 grid(static_cast<unsigned>((n + 63) / 64), static_cast<unsigned>(parts));
  const bool split = parts > 1;
  column_sum_kernel<<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16 *>(x), rows, n, split ? scratch : out, split ? 0 : accumulate);
  if (split)
    column_sum_merge_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(scratch, parts, n, out, accumulate);
  return finish_launch(split ? 2 : 1);
}

// ----------------------------------------------------------------------- cross entropy ----
namespace {
// A row's (max, sum-exp) partials, merged by one warp. kHeld pairs a lane are loaded at once and stay in registers for both passes:
// 16 (512 half tiles, 65536 columns), or 2 where 64 half tiles are all there are. With one 4-byte load in flight after another,
// 16384 rows of 394 pairs took 88 us where 16 take 54; 16384 rows of 4 pairs take 9.8 us with 16 and 6.5 with 2.
template <int kHeld>
__device__ __forceinline__ void merge_softmax_partials(const float *st, int n_tiles, int lane, float &mx_out, float &sum_out) {
  const float2 *pairs = reinterpret_cast<const float2 *>(st);
  float2 held[kHeld];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) held[i] = lane + 32 * i < n_tiles ? __ldg(pairs + lane + 32 * i) : make_float2(-INFINITY, 0.f);
#pragma unroll
  for (int i = 0; i < kHeld; ++i) mx = fmaxf(mx, held[i].x);
  for (int t = lane + 32 * kHeld; t < n_tiles; t += 32) mx = fmaxf(mx, pairs[t].x);
  mx = warp_max(mx);
  // a tile without a maximum has the sum 0, or NaN where its logits are
  const auto rescaled = [mx](float2 pair) { return pair.x > -INFINITY ? pair.y * __expf(pair.x - mx) : pair.y; };
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) sum += rescaled(held[i]);
  for (int t = lane + 32 * kHeld; t < n_tiles; t += 32) sum += rescaled(pairs[t]);
  mx_out = mx;
  sum_out = warp_sum(sum);
}

// One warp per row: merge the per-tile (max, sum-exp) partials, emit lse and the row loss.
template <int kHeld>
__global__ void __launch_bounds__(256) ce_finalize_kernel(const float *__restrict__ stats, int64_t n_tiles,
                                                          const __nv_bfloat16 *__restrict__ logits, int64_t ld,
                                                          const int64_t *__restrict__ target, float *__restrict__ lse,
                                                          float *__restrict__ loss_sum, float *__restrict__ count,
                                                          int64_t rows, int64_t ignore_index) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  float row_loss = 0.f, row_valid = 0.f;
  if (row < rows) {
    float mx, sum;
    merge_softmax_partials<kHeld>(stats + row * n_tiles * 2, static_cast<int>(n_tiles), lane, mx, sum);
    const float l = mx + __logf(sum);
    if (lane == 0) {
      lse[row] = l;
      const int64_t tg = target[row];
      if (tg != ignore_index && tg >= 0) (void)CS_IN_BOUNDS(kKidCrossEntropy, tg, ld);
      if (tg != ignore_index && tg >= 0 && tg < ld) {  // a label beyond the row is skipped, never dereferenced
        row_loss = l - __bfloat162float(logits[row * ld + tg]);
        row_valid = 1.f;
      }
    }
  }
  __shared__ float red[2][8];
  if (lane == 0) {
    red[0][threadIdx.x >> 5] = row_loss;
    red[1][threadIdx.x >> 5] = row_valid;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = 0.f, b = 0.f;
    for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) {
      a += red[0][i];
      b += red[1][i];
    }
    if (b > 0.f) {
      atomicAdd(loss_sum, a);
      atomicAdd(count, b);
    }
  }
}
__global__ void ce_mean_kernel(float *loss, const float *count) { loss[0] = loss[0] / fmaxf(count[0], 1.f); }

__global__ void __launch_bounds__(256) ce_backward_kernel(__nv_bfloat16 *__restrict__ logits, int64_t ld,
                                                          const float *__restrict__ lse, const int64_t *__restrict__ target,
                                                          const float *__restrict__ count, float grad_scale, int64_t rows,
                                                          int64_t n, int64_t n_valid, int64_t ignore_index, int64_t col_offset) {
  // One CTA walks whole rows; target and lse are read once per row. An element costs one FMA, one exponential and one
  // multiplication: the target and the end of the valid columns are looked at once per chunk of eight, with 32-bit column
  // numbers, and each thread has several chunks in flight. With both tested per element in 64 bits the kernel was bound by
  // issue slots: 16384 x 50304 in 701 us (0.72 of the copy bandwidth), now 543 (0.93).
  constexpr int kUnroll = 4;
  const int chunks = static_cast<int>(n / 8);
  const float inv = grad_scale / fmaxf(count[0], 1.f);
  const float log2e = 1.4426950408889634f;
  const int64_t left = n_valid - col_offset;  // valid columns of this slice
  const int valid = static_cast<int>(left < 0 ? 0 : (left > n ? n : left));
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const int64_t tg = target[row];
    const bool ignored = tg == ignore_index || tg < 0;
    if (!ignored && col_offset == 0) (void)CS_IN_BOUNDS(kKidCrossEntropy, tg, n_valid);
    const int64_t local = tg - col_offset;
    const int hit = ignored || local < 0 || local >= n ? -1 : static_cast<int>(local);  // column of the target, if it is here
    const float l2 = ignored ? 0.f : lse[row] * log2e;
    Bf16x8 *row_ptr = reinterpret_cast<Bf16x8 *>(logits + row * ld);
    for (int c0 = threadIdx.x; c0 < chunks; c0 += kUnroll * blockDim.x) {
      Bf16x8 v[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int c8 = c0 + u * static_cast<int>(blockDim.x);
        if (c8 < chunks && CS_IN_BOUNDS(kKidCrossEntropy, row * ld + c8 * 8 + 7, rows * ld)) v[u] = row_ptr[c8];
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int c8 = c0 + u * static_cast<int>(blockDim.x), col = c8 * 8;
        if (c8 >= chunks || !CS_IN_BOUNDS(kKidCrossEntropy, row * ld + col + 7, rows * ld)) continue;
        float f[8];
        if (ignored) {
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = 0.f;
        } else {
          unpack(v[u], f);
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = exp2f(fmaf(f[k], log2e, -l2));  // subnormal probabilities are gradients too
          if (col + 8 > valid) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (col + k >= valid) f[k] = 0.f;
          }
          if ((hit >> 3) == c8) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (col + k == hit) f[k] -= 1.f;
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] *= inv;
        }
        row_ptr[c8] = pack(f);
      }
    }
  }
}
}  // namespace

int cross_entropy_finalize(stream_t stream, const float *stats, int64_t n_tiles, const void *logits, int64_t ld,
                           const int64_t *target, float *lse, float *loss, float *count, int64_t rows,
                           int64_t ignore_index) {
  auto s = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(loss, 0, sizeof(float), s);
  cudaMemsetAsync(count, 0, sizeof(float), s);
  const int threads = 256;
  const int64_t blocks = (rows * 32 + threads - 1) / threads;
  auto *kernel = n_tiles <= 64 ? ce_finalize_kernel<2> : ce_finalize_kernel<16>;
  kernel<<<static_cast<unsigned>(blocks), threads, 0, s>>>(stats, n_tiles, static_cast<const __nv_bfloat16 *>(logits), ld, target, lse,
                                                           loss, count, rows, ignore_index);
  ce_mean_kernel<<<1, 1, 0, s>>>(loss, count);
  return finish_launch(2);
}

namespace {
template <int kHeld>
__global__ void __launch_bounds__(256) ce_slice_stats_kernel(const float *__restrict__ stats, int64_t n_tiles,
                                                             const __nv_bfloat16 *__restrict__ logits, int64_t ld,
                                                             const int64_t *__restrict__ target, int64_t col_offset,
                                                             int64_t n_valid_local, float *__restrict__ out, int64_t rows) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  float mx, sum;
  merge_softmax_partials<kHeld>(stats + row * n_tiles * 2, static_cast<int>(n_tiles), lane, mx, sum);
  if (lane == 0) {
    out[row * 2] = (n_valid_local > 0 && (mx > -INFINITY || sum != 0.f)) ? mx + __logf(sum) : -INFINITY;
    const int64_t local = target[row] - col_offset;
    out[row * 2 + 1] = (local >= 0 && local < n_valid_local) ? __bfloat162float(logits[row * ld + local]) : 0.f;
  }
}
}  // namespace

int cross_entropy_slice_stats(stream_t stream, const float *stats, int64_t n_tiles, const void *logits, int64_t ld,
                              const int64_t *target, int64_t col_offset, int64_t n_valid_local, float *out, int64_t rows) {
  if (rows == 0) return 0;
  const int threads = 256;
  const int64_t blocks = (rows * 32 + threads - 1) / threads;
  auto *kernel = n_tiles <= 64 ? ce_slice_stats_kernel<2> : ce_slice_stats_kernel<16>;
  kernel<<<static_cast<unsigned>(blocks), threads, 0, static_cast<cudaStream_t>(stream)>>>(
      stats, n_tiles, static_cast<const __nv_bfloat16 *>(logits), ld, target, col_offset, n_valid_local, out, rows);
  return finish_launch();
}

int cross_entropy_backward_inplace(stream_t stream, void *logits, int64_t ld, const float *lse, const int64_t *target,
                                   const float *count, float grad_scale, int64_t rows, int64_t n, int64_t n_valid,
                                   int64_t ignore_index, int64_t col_offset) {
  if (n % 8 != 0 || ld % 8 != 0) return static_cast<int>(cudaErrorInvalidValue);
  // Four chunks of eight columns a thread, up to 256 threads, and as many CTAs as an SM holds at 64 registers a thread. With 256
  // threads at every width 16384 x 512 took 20.2 us and 3000 x 4000 11.2, now 8.6 and 10.1.
  const int threads = n >= 8192 ? 256 : static_cast<int>((n / 1024 + 1) * 32);
  const int64_t cap = static_cast<int64_t>(kSmCount) * (threads == 256 ? 8 : 1024 / threads);
  ce_backward_kernel<<<static_cast<unsigned>(rows < cap ? rows : cap), threads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16 *>(logits), ld, lse, target, count, grad_scale, rows, n, n_valid, ignore_index, col_offset);
  return finish_launch();
}

// ----------------------------------------------------------------------- gradient norm ----
namespace {
// 16-byte loads where the pointer allows it; the scalar loop covers the tail (or everything).
template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(const T *__restrict__ x, int64_t n, float *__restrict__ out) {
  constexpr int V = 16 / sizeof(T);
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t nv = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / V : 0;
  float acc0 = 0.f, acc1 = 0.f;
  for (int64_t i = gid; i < nv; i += stride) {
    const uint4 raw = *reinterpret_cast<const uint4 *>(x + i * V);
    const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      const float a = to_f<T>(e[k]), b = to_f<T>(e[k + 1]);
      acc0 = fmaf(a, a, acc0);
      acc1 = fmaf(b, b, acc1);
    }
  }
  for (int64_t i = nv * V + gid; i < n; i += stride) {
    const float v = to_f<T>(x[i]);
    acc0 = fmaf(v, v, acc0);
  }
  float acc = warp_sum(acc0 + acc1);
  __shared__ float red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[i];
    atomicAdd(out, t);
  }
}
__global__ void clip_coef_kernel(const float *sumsq, float max_norm, float *coef, float *norm_out) {
  const float norm = sqrtf(sumsq[0]);
  norm_out[0] = norm;
  coef[0] = fminf(1.f, max_norm / (norm + 1e-6f));
}
template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(T *__restrict__ x, int64_t n, const float *__restrict__ coef) {
  const float c = coef[0];
  if (c == 1.f) return;
  constexpr int V = 16 / sizeof(T);
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t nv = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / V : 0;
  for (int64_t i = gid; i < nv; i += stride) {
    uint4 raw = *reinterpret_cast<const uint4 *>(x + i * V);
    T *e = reinterpret_cast<T *>(&raw);
#pragma unroll
    for (int k = 0; k < V; ++k) e[k] = from_f<T>(to_f<T>(e[k]) * c);
    *reinterpret_cast<uint4 *>(x + i * V) = raw;
  }
  for (int64_t i = nv * V + gid; i < n; i += stride) x[i] = from_f<T>(to_f<T>(x[i]) * c);
}
}  // namespace

int sum_squares(stream_t stream, const void *x, int dtype, int64_t n, float *sumsq) {
  auto s = static_cast<cudaStream_t>(stream);
  if (n == 0) return 0;
  if (dtype == 0) sumsq_kernel<float><<<grid_for((n + 3) / 4, 256, 8), 256, 0, s>>>(static_cast<const float *>(x), n, sumsq);
  else if (dtype == 1) sumsq_kernel<__nv_bfloat16><<<grid_for((n + 7) / 8, 256, 8), 256, 0, s>>>(static_cast<const __nv_bfloat16 *>(x), n, sumsq);
  else return static_cast<int>(cudaErrorInvalidValue);
  return finish_launch();
}
int clip_coefficient(stream_t stream, const float *sumsq, float max_norm, float *coef, float *norm_out) {
  clip_coef_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(sumsq, max_norm, coef, norm_out);
  return finish_launch();
}
int scale_by_device_scalar(stream_t stream, void *x, int dtype, int64_t n, const float *coef) {
  auto s = static_cast<cudaStream_t>(stream);
  if (n == 0) return 0;
  if (dtype == 0) scale_kernel<float><<<grid_for((n + 3) / 4, 256, 8), 256, 0, s>>>(static_cast<float *>(x), n, coef);
  else if (dtype == 1) scale_kernel<__nv_bfloat16><<<grid_for((n + 7) / 8, 256, 8), 256, 0, s>>>(static_cast<__nv_bfloat16 *>(x), n, coef);
  else return static_cast<int>(cudaErrorInvalidValue);
  return finish_launch();
}
}  // namespace cs::kernels

// ------------------------------------------------------------- allocation-free entry ----
// LayerNorm backward for callers that cannot allocate (see no_alloc.h). Same kernels as
// layernorm_backward() above; the partial dgamma/dbeta rows go to a file-scope device array.
#include "no_alloc.h"

namespace {
static __device__ __align__(256) float g_noalloc_ln_scratch[CS_NOALLOC_LN_PARTS * 2 * CS_NOALLOC_LN_MAX_D];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
float *g_noalloc_scratch_ptr[kNoAllocMaxDevices] = {};

// In host code `g_noalloc_ln_scratch` is only a handle for the runtime; the address a kernel
// can use has to be asked for, once per device, with that device current.
int noalloc_scratch(float **out) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (device < 0 || device >= kNoAllocMaxDevices) return static_cast<int>(cudaErrorInvalidDevice);
  std::lock_guard<std::mutex> lock{g_noalloc_mutex};
  if (!g_noalloc_scratch_ptr[device]) {
    float *ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_noalloc_ln_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    g_noalloc_scratch_ptr[device] = ptr;
  }
  *out = g_noalloc_scratch_ptr[device];
  return 0;
}
}  // namespace

extern "C" __attribute__((visibility("default"))) int cs_layernorm_backward_noalloc(
    const void *dy, const void *x, const float *gamma, const float *mean, const float *rstd, const void *grad_residual,
    void *dx, float *dgamma, float *dbeta, int accumulate, int64_t rows, int64_t d, void *stream) {
  using namespace cs::kernels;
  if (!dy || !x || !gamma || !mean || !rstd || !dx || !dgamma || !dbeta || rows < 0) return -2;
  if (d <= 0 || d % 8 != 0 || d > CS_NOALLOC_LN_MAX_D) return -1;
  if (rows == 0) return 0;
  float *scratch = nullptr;
  const int rc = noalloc_scratch(&scratch);
  if (rc != 0) return rc;
  auto s = static_cast<cudaStream_t>(stream);
  return launch_ln_bwd(s, dy, x, gamma, 0, mean, rstd, grad_residual, dx, dgamma, dbeta, accumulate, scratch, rows, static_cast<int>(d),
                       CS_NOALLOC_LN_PARTS * CS_NOALLOC_LN_MAX_D / d);  // a narrower row leaves room for more partial rows
}
