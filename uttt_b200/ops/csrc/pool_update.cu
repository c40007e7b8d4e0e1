// Fast-weight master step, fused: one pass instead of ten elementwise / reduction launches.
//
//   u = m + lr * d                         m: fp32 master rows [R, D], d: update direction (bf16 or fp32)
//   restore: n = u / (|u| + 1e-5) * |m|    (rows keep their previous length; language-model rule)
//   unit   : n = u / max(|u|, 1e-12)       (unit rows; view-synthesis rule)
//   none   : n = u
//   w = bf16(n)                            compute copy read by the grouped GEMMs
//
// and its vector-Jacobian product (g = d n + d w):
//   restore: s = |m| / (|u| + eps);  g_u = s g - u (g.u) s / ((|u| + eps) |u|);  g_m = g_u + m (g.u) / ((|u| + eps) |m|)
//   unit   : g_u = g / |u| - u (g.u) / |u|^3;                                     g_m = g_u
//   g_d = lr g_u
// One warp per row of up to 512 elements, four warps beyond; the row lives in registers between the reduction and the
// write.
// Reference behaviour: flame/custom_models/uttt_moe/modeling_recurrent_lact.py:754-825 (dense apply) and the
// row re-normalisation of the view-synthesis blocks.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "common.cuh"
#include "operand.h"

namespace uttt {

constexpr int kPoolMaxV = 4;         // float4 pieces per lane
constexpr int kPoolMaxD = 2048;      // four warps to a row of more than 512 elements, one to a shorter one
enum PoolRenorm { kRestore = 0, kUnit = 1, kNone = 2 };

template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&f)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, float (&f)[4]) {
  float4 v = *reinterpret_cast<const float4*>(p);
  f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&f)[4]) {
  uint2 v = *reinterpret_cast<const uint2*>(p);
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&v.x), b = *reinterpret_cast<__nv_bfloat162*>(&v.y);
  f[0] = __low2float(a); f[1] = __high2float(a); f[2] = __low2float(b); f[3] = __high2float(b);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&f)[4]);
template <>
__device__ __forceinline__ void store4<float>(float* p, const float (&f)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&f)[4]) {
  __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
  uint2 v;
  v.x = *reinterpret_cast<uint32_t*>(&a);
  v.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = v;
}

// Sums of a row held by W warps (W = 4: half of a 256-thread block, with a barrier of its own).  `turn` alternates the
// exchange buffer from one row to the next, so that one barrier per row is enough.
template <int W, int N>
__device__ __forceinline__ void row_sums(float (&v)[N], int& turn) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = warp_sum(v[i]);
  if constexpr (W > 1) {
    static_assert(W == 4);
    __shared__ float part[2][8][N];
    const int warp = threadIdx.x >> 5, first = warp & ~(W - 1);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int i = 0; i < N; ++i) part[turn][warp][i] = v[i];
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + first / W), "n"(32 * W) : "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i] = 0.f;
#pragma unroll
      for (int w = 0; w < W; ++w) v[i] += part[turn][first + w][i];
    }
    turn ^= 1;
  }
}

// Bound by memory.  A row of 1536 elements on one warp needs 12 vectors per lane and array in registers (the backward
// holds three arrays), which left two or three blocks per SM and half the copy rate; on four warps it needs three.
// 24,576 rows of 1536: forward 113 -> 84 us, backward 252 -> 126 us; 196,608 rows of 384, where the backward no longer
// reads the master twice: 287 -> 229 us.
template <typename TD, int W>
__global__ void __launch_bounds__(256) pool_step_fwd_kernel(const float* __restrict__ m, const TD* __restrict__ d,
                                                            float lr, int mode, float* __restrict__ n_out,
                                                            __nv_bfloat16* __restrict__ w_out, long long rows, int D) {
  constexpr int L = 32 * W, MAXV = kPoolMaxV;
  const int lane = threadIdx.x & (L - 1);
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const long long stride = (long long)gridDim.x * blockDim.x / L;
  const int nv = D >> 2;
  int turn = 0;
  for (long long r = first; r < rows; r += stride) {
    const float* mr = m + r * D;
    const TD* dr = d + r * D;
    float u[MAXV][4];
    float su = 0.f, sm = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      int v = lane + L * j;
      if (v < nv) {
        float a[4], b[4];
        load4(mr + v * 4, a);
        load4(dr + v * 4, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          u[j][i] = fmaf(lr, b[i], a[i]);
          su = fmaf(u[j][i], u[j][i], su);
          sm = fmaf(a[i], a[i], sm);
        }
      }
    }
    float s = 1.f;
    if (mode != kNone) {
      float t[2] = {su, sm};
      row_sums<W>(t, turn);
      su = t[0];
      sm = t[1];
      s = (mode == kRestore) ? sqrtf(sm) / (sqrtf(su) + 1e-5f) : 1.f / fmaxf(sqrtf(su), 1e-12f);
    }
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      int v = lane + L * j;
      if (v < nv) {
        float o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = u[j][i] * s;
        store4(n_out + r * D + v * 4, o);
        store4(w_out + r * D + v * 4, o);
      }
    }
  }
}

template <typename TD, int W>
__global__ void __launch_bounds__(256) pool_step_bwd_kernel(const float* __restrict__ m, const TD* __restrict__ d,
                                                            const float* __restrict__ gn,
                                                            const __nv_bfloat16* __restrict__ gw, float lr, int mode,
                                                            float* __restrict__ gm_out, TD* __restrict__ gd_out,
                                                            long long rows, int D) {
  constexpr int L = 32 * W, MAXV = kPoolMaxV;
  const int lane = threadIdx.x & (L - 1);
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const long long stride = (long long)gridDim.x * blockDim.x / L;
  const int nv = D >> 2;
  int turn = 0;
  for (long long r = first; r < rows; r += stride) {
    const float* mr = m + r * D;
    const TD* dr = d + r * D;
    float u[MAXV][4], g[MAXV][4], a[MAXV][4];
    float su = 0.f, sm = 0.f, gu = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      int v = lane + L * j;
      if (v < nv) {
        float b[4];
        load4(mr + v * 4, a[j]);
        load4(dr + v * 4, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) g[j][i] = 0.f;
        if (gn != nullptr) load4(gn + r * D + v * 4, g[j]);
        if (gw != nullptr) {
          float h[4];
          load4(gw + r * D + v * 4, h);
#pragma unroll
          for (int i = 0; i < 4; ++i) g[j][i] += h[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          u[j][i] = fmaf(lr, b[i], a[j][i]);
          su = fmaf(u[j][i], u[j][i], su);
          sm = fmaf(a[j][i], a[j][i], sm);
          gu = fmaf(g[j][i], u[j][i], gu);
        }
      }
    }
    float cg = 1.f, cu = 0.f, cm = 0.f;      // g_u = cg * g - cu * u ;  g_m = g_u + cm * m
    if (mode != kNone) {
      float t[3] = {su, sm, gu};
      row_sums<W>(t, turn);
      su = t[0];
      sm = t[1];
      gu = t[2];
      const float nu = sqrtf(su), nm = sqrtf(sm);
      if (mode == kRestore) {
        const float den = nu + 1e-5f;
        cg = nm / den;
        cu = (nu > 0.f) ? gu * nm / (den * den * nu) : 0.f;
        cm = (nm > 0.f) ? gu / (den * nm) : 0.f;
      } else {
        const float den = fmaxf(nu, 1e-12f);
        cg = 1.f / den;
        cu = (nu > 1e-12f) ? gu / (den * den * den) : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      int v = lane + L * j;
      if (v < nv) {
        float o_m[4], o_d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float t = cg * g[j][i] - cu * u[j][i];
          o_m[i] = (cm != 0.f) ? fmaf(cm, a[j][i], t) : t;
          o_d[i] = lr * t;
        }
        store4(gm_out + r * D + v * 4, o_m);
        store4(gd_out + r * D + v * 4, o_d);
      }
    }
  }
}

static int pool_blocks(long long rows, int rows_per_block) {
  int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  long long want = (rows + rows_per_block - 1) / rows_per_block;
  return (int)std::max<long long>(1, std::min<long long>(want, (long long)sms * 8));
}

bool pool_step_supported(int64_t D) { return D % 4 == 0 && D <= kPoolMaxD; }

// m [.., D] fp32, d same shape (bf16 or fp32) -> (n fp32, w bf16)
std::vector<at::Tensor> pool_step_fwd(at::Tensor m, at::Tensor d, double lr, int64_t mode) {
  c10::cuda::CUDAGuard guard(m.device());
  TORCH_CHECK(m.scalar_type() == at::kFloat && m.is_contiguous() && d.is_contiguous() && d.numel() == m.numel());
  const int D = m.size(-1);
  TORCH_CHECK(pool_step_supported(D));
  m = dense16(m);
  d = dense16(d);
  const long long rows = m.numel() / D;
  auto n = at::empty_like(m);
  auto w = at::empty(m.sizes(), m.options().dtype(at::kBFloat16));
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int blocks = pool_blocks(rows, D <= 512 ? 8 : 2);
  auto go = [&](auto* dp) {
    using TD = std::remove_cv_t<std::remove_pointer_t<decltype(dp)>>;
    if (D <= 512)
      pool_step_fwd_kernel<TD, 1><<<blocks, 256, 0, stream>>>(m.data_ptr<float>(), dp, (float)lr, (int)mode,
                                                              n.data_ptr<float>(),
                                                              reinterpret_cast<__nv_bfloat16*>(w.data_ptr()), rows, D);
    else
      pool_step_fwd_kernel<TD, 4><<<blocks, 256, 0, stream>>>(
          m.data_ptr<float>(), dp, (float)lr, (int)mode, n.data_ptr<float>(),
          reinterpret_cast<__nv_bfloat16*>(w.data_ptr()), rows, D);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  if (d.scalar_type() == at::kBFloat16) go(reinterpret_cast<const __nv_bfloat16*>(d.data_ptr()));
  else { TORCH_CHECK(d.scalar_type() == at::kFloat); go(d.data_ptr<float>()); }
  count_launch();
  return {n, w};
}

// (gn fp32 or none, gw bf16 or none) -> (g_m fp32, g_d in the dtype of d)
std::vector<at::Tensor> pool_step_bwd(at::Tensor m, at::Tensor d, c10::optional<at::Tensor> gn,
                                      c10::optional<at::Tensor> gw, double lr, int64_t mode) {
  c10::cuda::CUDAGuard guard(m.device());
  const int D = m.size(-1);
  TORCH_CHECK(pool_step_supported(D) && m.is_contiguous() && d.is_contiguous());
  m = dense16(m);
  d = dense16(d);
  const long long rows = m.numel() / D;
  at::Tensor gnc, gwc;
  const float* gnp = nullptr;
  const __nv_bfloat16* gwp = nullptr;
  if (gn.has_value() && gn->defined()) {
    gnc = dense16(gn->to(at::kFloat));
    gnp = gnc.data_ptr<float>();
  }
  if (gw.has_value() && gw->defined()) {
    gwc = dense16(gw->to(at::kBFloat16));
    gwp = reinterpret_cast<const __nv_bfloat16*>(gwc.data_ptr());
  }
  auto gm = at::empty_like(m);
  auto gd = at::empty_like(d);
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int blocks = pool_blocks(rows, D <= 512 ? 8 : 2);
  auto go = [&](auto* dp, auto* gp) {
    using TD = std::remove_cv_t<std::remove_pointer_t<decltype(dp)>>;
    if (D <= 512)
      pool_step_bwd_kernel<TD, 1><<<blocks, 256, 0, stream>>>(m.data_ptr<float>(), dp, gnp, gwp, (float)lr, (int)mode,
                                                              gm.data_ptr<float>(), gp, rows, D);
    else
      pool_step_bwd_kernel<TD, 4><<<blocks, 256, 0, stream>>>(m.data_ptr<float>(), dp, gnp, gwp, (float)lr,
                                                                      (int)mode, gm.data_ptr<float>(), gp, rows, D);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  if (d.scalar_type() == at::kBFloat16)
    go(reinterpret_cast<const __nv_bfloat16*>(d.data_ptr()), reinterpret_cast<__nv_bfloat16*>(gd.data_ptr()));
  else { TORCH_CHECK(d.scalar_type() == at::kFloat); go(d.data_ptr<float>(), gd.data_ptr<float>()); }
  count_launch();
  return {gm, gd};
}

}  // namespace uttt

// ------------------------------------------------------------------------------------ Newton-Schulz input
// X[b] = G[b] / (|G[b]|_F + eps) cast to bf16, per matrix of a batch, in two passes (sum of squares, scale + cast)
// instead of cast / cast back / norm / add / cast / divide; and its VJP
//   dG = dX / (r + eps) - G <dX, G> / (r (r + eps)^2),   r = |G|_F.
namespace uttt {

template <typename T>
__global__ void __launch_bounds__(256) frob_partial_kernel(const T* __restrict__ g, const __nv_bfloat16* __restrict__ dx,
                                                           float* __restrict__ out, long long per_matrix) {
  // grid (chunks, matrices); out[b] += sum g^2 (dx == nullptr) or sum dx * g
  const long long b = blockIdx.y;
  const T* gp = g + b * per_matrix;
  const __nv_bfloat16* dp = dx ? dx + b * per_matrix : nullptr;
  float acc = 0.f;
  const long long nv = per_matrix >> 2;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
    float a[4];
    load4(gp + v * 4, a);
    if (dp) {
      float d[4];
      load4(dp + v * 4, d);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc = fmaf(a[i], d[i], acc);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc = fmaf(a[i], a[i], acc);
    }
  }
  acc = warp_sum(acc);
  __shared__ float red[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < 8; ++i) s += red[i];
    atomicAdd(out + b, s);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) frob_scale_kernel(const T* __restrict__ g, const float* __restrict__ sumsq,
                                                         float eps, __nv_bfloat16* __restrict__ x,
                                                         long long per_matrix) {
  const long long b = blockIdx.y;
  const float inv = 1.f / (sqrtf(sumsq[b]) + eps);
  const long long nv = per_matrix >> 2;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
    float a[4];
    load4(g + b * per_matrix + v * 4, a);
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] *= inv;
    store4(x + b * per_matrix + v * 4, a);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) frob_scale_bwd_kernel(const T* __restrict__ g, const __nv_bfloat16* __restrict__ dx,
                                                             const float* __restrict__ sumsq,
                                                             const float* __restrict__ dot, float eps,
                                                             T* __restrict__ dg, long long per_matrix) {
  const long long b = blockIdx.y;
  const float r = sqrtf(sumsq[b]);
  const float inv = 1.f / (r + eps);
  const float coef = r > 0.f ? dot[b] * inv * inv / r : 0.f;
  const long long nv = per_matrix >> 2;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
    float a[4], d[4], o[4];
    load4(g + b * per_matrix + v * 4, a);
    load4(dx + b * per_matrix + v * 4, d);
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = d[i] * inv - a[i] * coef;
    store4(dg + b * per_matrix + v * 4, o);
  }
}

static dim3 frob_grid(long long per_matrix, int batch) {
  int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  long long want = (per_matrix / 4 + 255) / 256;
  int per = (int)std::max<long long>(1, std::min<long long>(want, std::max(1, sms * 4 / std::max(batch, 1))));
  return dim3(per, batch);
}

// g [B, M, N] (fp32 or bf16) -> (x bf16 [B, M, N], sumsq [B] fp32)
std::vector<at::Tensor> frob_normalize_fwd(at::Tensor g, double eps) {
  c10::cuda::CUDAGuard guard(g.device());
  TORCH_CHECK(g.dim() == 3 && g.is_contiguous() && (g.size(1) * g.size(2)) % 4 == 0);
  g = dense16(g);
  const int batch = g.size(0);
  const long long per = (long long)g.size(1) * g.size(2);
  auto sumsq = at::zeros({batch}, g.options().dtype(at::kFloat));
  auto x = at::empty(g.sizes(), g.options().dtype(at::kBFloat16));
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  dim3 grid = frob_grid(per, batch);
  auto* xp = reinterpret_cast<__nv_bfloat16*>(x.data_ptr());
  if (g.scalar_type() == at::kFloat) {
    frob_partial_kernel<float><<<grid, 256, 0, stream>>>(g.data_ptr<float>(), nullptr, sumsq.data_ptr<float>(), per);
    frob_scale_kernel<float><<<grid, 256, 0, stream>>>(g.data_ptr<float>(), sumsq.data_ptr<float>(), (float)eps, xp, per);
  } else {
    TORCH_CHECK(g.scalar_type() == at::kBFloat16);
    auto* gp = reinterpret_cast<const __nv_bfloat16*>(g.data_ptr());
    frob_partial_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(gp, nullptr, sumsq.data_ptr<float>(), per);
    frob_scale_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(gp, sumsq.data_ptr<float>(), (float)eps, xp, per);
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  return {x, sumsq};
}

at::Tensor frob_normalize_bwd(at::Tensor g, at::Tensor sumsq, at::Tensor dx, double eps) {
  c10::cuda::CUDAGuard guard(g.device());
  TORCH_CHECK(g.dim() == 3 && g.is_contiguous() && sumsq.scalar_type() == at::kFloat);
  g = dense16(g);
  auto dxc = dense16(dx.to(at::kBFloat16));
  const int batch = g.size(0);
  const long long per = (long long)g.size(1) * g.size(2);
  auto dot = at::zeros({batch}, sumsq.options());
  auto dg = at::empty_like(g);
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  dim3 grid = frob_grid(per, batch);
  auto* dp = reinterpret_cast<const __nv_bfloat16*>(dxc.data_ptr());
  if (g.scalar_type() == at::kFloat) {
    frob_partial_kernel<float><<<grid, 256, 0, stream>>>(g.data_ptr<float>(), dp, dot.data_ptr<float>(), per);
    frob_scale_bwd_kernel<float><<<grid, 256, 0, stream>>>(g.data_ptr<float>(), dp, sumsq.data_ptr<float>(),
                                                          dot.data_ptr<float>(), (float)eps, dg.data_ptr<float>(), per);
  } else {
    TORCH_CHECK(g.scalar_type() == at::kBFloat16);
    auto* gp = reinterpret_cast<const __nv_bfloat16*>(g.data_ptr());
    frob_partial_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(gp, dp, dot.data_ptr<float>(), per);
    frob_scale_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(
        gp, dp, sumsq.data_ptr<float>(), dot.data_ptr<float>(), (float)eps,
        reinterpret_cast<__nv_bfloat16*>(dg.data_ptr()), per);
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  return dg;
}

// ------------------------------------------------------------------------------------ momentum + Newton-Schulz input
// z' = a + m[seq] z and X = z' / (|z'|_F + eps) per matrix, and their VJP
//   g  = dz' + dX / (r + eps) - z' <dX, z'> / (r (r + eps)^2),   r = |z'|_F
//   da = g,   dz = m g,   dm[seq] = sum over the matrices of the sequence of <g, z>.
// Bound by memory.  The squares are summed while z' is written, and the VJP forms da, dz and the products for dm from one
// read of its operands: as separate operations the broadcast multiply-add alone ran at 3.9 TB/s, and the backward paid an
// addition, a broadcast product and a product with its reduction on top of the normalisation.  Bank of 113 M values:
// forward 512 -> 333 us, backward 1057 -> 508 us.
__global__ void __launch_bounds__(256) momentum_sumsq_kernel(const float* __restrict__ a, const float* __restrict__ z,
                                                             const float* __restrict__ m, float* __restrict__ z_out,
                                                             float* __restrict__ sumsq, long long per_matrix, int per_seq) {
  const long long b = blockIdx.y;
  const float mc = m[b / per_seq];
  const long long off = b * per_matrix, nv = per_matrix >> 2;
  float acc = 0.f;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
    float x[4], y[4];
    load4(a + off + v * 4, x);
    load4(z + off + v * 4, y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = fmaf(mc, y[i], x[i]);
      acc = fmaf(x[i], x[i], acc);
    }
    store4(z_out + off + v * 4, x);
  }
  acc = warp_sum(acc);
  __shared__ float red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < 8; ++i) s += red[i];
    atomicAdd(sumsq + b, s);
  }
}

// dx, dz_new, dz and dm may be absent; dm[b, chunk] = the block's share of <g, z> of matrix b, so that the sum over the
// blocks has one order
__global__ void __launch_bounds__(256) momentum_bwd_kernel(const float* __restrict__ z_new, const float* __restrict__ z,
                                                           const float* __restrict__ m, const __nv_bfloat16* __restrict__ dx,
                                                           const float* __restrict__ dz_new, const float* __restrict__ sumsq,
                                                           const float* __restrict__ dot, float eps, float* __restrict__ da,
                                                           float* __restrict__ dz, float* __restrict__ dm,
                                                           long long per_matrix, int per_seq) {
  const long long b = blockIdx.y;
  const float mc = m[b / per_seq];
  float inv = 0.f, coef = 0.f;
  if (dx != nullptr) {
    const float r = sqrtf(sumsq[b]);
    inv = 1.f / (r + eps);
    coef = r > 0.f ? dot[b] * inv * inv / r : 0.f;
  }
  const long long off = b * per_matrix, nv = per_matrix >> 2;
  float acc = 0.f;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
    const long long at = off + v * 4;
    float g[4] = {0.f, 0.f, 0.f, 0.f};
    if (dz_new != nullptr) load4(dz_new + at, g);
    if (dx != nullptr) {
      float d[4], x[4];
      load4(dx + at, d);
      load4(z_new + at, x);
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] += d[i] * inv - x[i] * coef;
    }
    store4(da + at, g);
    if (dm != nullptr) {
      float y[4];
      load4(z + at, y);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc = fmaf(g[i], y[i], acc);
    }
    if (dz != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] *= mc;
      store4(dz + at, g);
    }
  }
  if (dm == nullptr) return;
  acc = warp_sum(acc);
  __shared__ float red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < 8; ++i) s += red[i];
    dm[b * gridDim.x + blockIdx.x] = s;
  }
}

static void check_bank(const at::Tensor& t, int64_t matrices) {
  TORCH_CHECK(t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() % (4 * matrices) == 0 &&
              ((uintptr_t)t.data_ptr() & 15) == 0);
}

// a, z fp32 [S, ...] holding `matrices` equal matrices, m fp32 [S] -> (z' like a, X bf16 like a, sumsq [matrices])
std::vector<at::Tensor> momentum_normalize_fwd(at::Tensor a, at::Tensor z, at::Tensor m, int64_t matrices, double eps) {
  c10::cuda::CUDAGuard guard(a.device());
  check_bank(a, matrices);
  check_bank(z, matrices);
  TORCH_CHECK(z.numel() == a.numel() && m.scalar_type() == at::kFloat && m.is_contiguous() && m.numel() > 0 &&
              matrices % m.numel() == 0 && matrices <= 65535);
  const long long per = a.numel() / matrices;
  auto z_new = at::empty_like(a);
  auto x = at::empty(a.sizes(), a.options().dtype(at::kBFloat16));
  auto sumsq = at::zeros({matrices}, a.options());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const dim3 grid = frob_grid(per, (int)matrices);
  momentum_sumsq_kernel<<<grid, 256, 0, stream>>>(a.data_ptr<float>(), z.data_ptr<float>(), m.data_ptr<float>(),
                                                 z_new.data_ptr<float>(), sumsq.data_ptr<float>(), per,
                                                 (int)(matrices / m.numel()));
  frob_scale_kernel<float><<<grid, 256, 0, stream>>>(z_new.data_ptr<float>(), sumsq.data_ptr<float>(), (float)eps,
                                                     reinterpret_cast<__nv_bfloat16*>(x.data_ptr()), per);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  return {z_new, x, sumsq};
}

// -> (da, dz or empty, dm [S] or empty)
std::vector<at::Tensor> momentum_normalize_bwd(at::Tensor z_new, at::Tensor z, at::Tensor m, at::Tensor sumsq,
                                               c10::optional<at::Tensor> dz_new, c10::optional<at::Tensor> dx, double eps,
                                               bool need_dz, bool need_dm) {
  c10::cuda::CUDAGuard guard(z_new.device());
  const int64_t matrices = sumsq.numel();
  TORCH_CHECK(matrices > 0 && sumsq.scalar_type() == at::kFloat && sumsq.is_contiguous());
  z_new = dense16(z_new);
  z = dense16(z);
  check_bank(z_new, matrices);
  check_bank(z, matrices);
  TORCH_CHECK(z.numel() == z_new.numel() && m.scalar_type() == at::kFloat && m.is_contiguous() && m.numel() > 0 &&
              matrices % m.numel() == 0 && matrices <= 65535);
  const long long per = z_new.numel() / matrices;
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const dim3 grid = frob_grid(per, (int)matrices);
  at::Tensor gz, gx, dot;
  if (dz_new.has_value() && dz_new->defined()) {
    gz = dense16(dz_new->to(at::kFloat));
    TORCH_CHECK(gz.numel() == z_new.numel() && gz.device() == z_new.device());
  }
  if (dx.has_value() && dx->defined()) {
    gx = dense16(dx->to(at::kBFloat16));
    TORCH_CHECK(gx.numel() == z_new.numel() && gx.device() == z_new.device());
    dot = at::zeros({matrices}, sumsq.options());
    frob_partial_kernel<float><<<grid, 256, 0, stream>>>(z_new.data_ptr<float>(),
                                                         reinterpret_cast<const __nv_bfloat16*>(gx.data_ptr()),
                                                         dot.data_ptr<float>(), per);
    count_launch();
  }
  auto da = at::empty_like(z_new);
  auto dz = need_dz ? at::empty_like(z) : at::empty({0}, z.options());
  auto dm = at::empty({need_dm ? matrices : 0, (int64_t)grid.x}, m.options());
  momentum_bwd_kernel<<<grid, 256, 0, stream>>>(
      z_new.data_ptr<float>(), z.data_ptr<float>(), m.data_ptr<float>(),
      gx.defined() ? reinterpret_cast<const __nv_bfloat16*>(gx.data_ptr()) : nullptr,
      gz.defined() ? gz.data_ptr<float>() : nullptr, sumsq.data_ptr<float>(), gx.defined() ? dot.data_ptr<float>() : nullptr,
      (float)eps, da.data_ptr<float>(), need_dz ? dz.data_ptr<float>() : nullptr, need_dm ? dm.data_ptr<float>() : nullptr,
      per, (int)(matrices / m.numel()));
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {da, dz, need_dm ? dm.view({m.numel(), -1}).sum(1) : dm};
}

}  // namespace uttt
