// Fused router of the fast-weight expert pool.
//
//   logits = rows . router^T (+ bias)   fp32, rows [R, D] bf16 / fp32, router [E, D] fp32
//   probs  = softmax(logits)                                              mode 0 (softmax)
//            softmax(s * z),  z = logits / max(|logits|_2, eps)           mode 1 (norm_softmax)
//            relu(z) s / sum relu(z) s  (uniform when the sum is 0)       mode 2 (norm_relu)
//   (modes 1 and 2 select on the rescaled scores and keep the raw logits for the backward)
//   idx    = top-k of (logits + selection bias)               (the bias moves selection only, unless it is
//                                                              declared part of the logits)
//   weight = alpha * probs[idx]   or   alpha * probs[idx] / sum_sel probs[idx]
//   probs_sum[b, e] += probs[r, e]                            (load-balance statistics per sequence)
//
// Forward, bf16 rows: tensor cores (router_fwd_tc_kernel).  Other row types and shapes: a block stages 64 rows in shared
// memory, each warp multiplies 8 of them with lane = expert (two experts per lane when E = 64) against the transposed
// router matrix in shared memory, then does the softmax and the top-k with warp shuffles.
// Backward: one kernel turns (d weight, d probs_sum) into d logits and d rows (lane = slice of D), a second one
// reduces d router = d logits^T . rows over row chunks with per-thread register tiles into per-block partials.
// Reference behaviour: flame/custom_models/uttt_moe/moe_routing.py:7-75 (softmax router, selected_prob /
// topk_renorm combine modes).
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "common.cuh"
#include "operand.h"
#include "ptx.cuh"
#include "tc_gemm.cuh"

namespace uttt {

at::Tensor gemm_status(at::Tensor like);
at::Tensor col_sum(at::Tensor partial);

constexpr int kMaxTopK = 4;

template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&f)[8]) { Vec8<T>::load(p, f); }

// ------------------------------------------------------------------------------------ forward
// Block = 8 warps.  Per step the block stages 8 * RPW rows in shared memory with coalesced 16-byte loads (all
// in flight at once), then warp w multiplies its RPW rows: lane = expert, the row values are warp-uniform
// shared-memory reads, the router matrix sits transposed ([D][32 * EPL + 1], padded against bank conflicts).
template <typename T, int EPL, int RPW>
__global__ void __launch_bounds__(256) router_fwd_kernel(const T* __restrict__ rows, const float* __restrict__ router,
                                                         const float* __restrict__ bias, int R, int D, int E, int topk,
                                                         int rows_per_batch, float alpha, int bias_in_logits,
                                                         int renorm, int* __restrict__ idx_out,
                                                         float* __restrict__ w_out, float* __restrict__ probs_out,
                                                         float* __restrict__ probs_sum, int mode, float rscale,
                                                         float norm_eps, float* __restrict__ logits_out) {
  constexpr int EP = 32 * EPL + 1;
  constexpr int VEC = 16 / (int)sizeof(T);           // elements per 16-byte piece
  constexpr int BR = 8 * RPW;                        // rows per block step
  extern __shared__ __align__(16) uint8_t smem_r[];
  float* wt = reinterpret_cast<float*>(smem_r);                        // [D][EP]
  T* xs = reinterpret_cast<T*>(smem_r + (((size_t)D * EP * 4 + 15) & ~(size_t)15));   // [BR][D]
  for (int i = threadIdx.x; i < E * D; i += blockDim.x) {
    int e = i / D, d = i - e * D;
    wt[d * EP + e] = router[i];
  }
  for (int i = threadIdx.x; i < D * (32 * EPL - E); i += blockDim.x) {
    int d = i / (32 * EPL - E), e = E + i % (32 * EPL - E);
    wt[d * EP + e] = 0.f;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float bsel[EPL], blog[EPL];
#pragma unroll
  for (int q = 0; q < EPL; ++q) {
    int e = lane + 32 * q;
    float b = (bias != nullptr && e < E) ? bias[e] : 0.f;
    blog[q] = bias_in_logits ? b : 0.f;
    bsel[q] = bias_in_logits ? 0.f : b;
  }
  float psum[EPL];
#pragma unroll
  for (int q = 0; q < EPL; ++q) psum[q] = 0.f;
  int cur_b = -1;
  auto flush = [&]() {
    if (cur_b >= 0) {
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        int e = lane + 32 * q;
        if (e < E) atomicAdd(probs_sum + (size_t)cur_b * E + e, psum[q]);
        psum[q] = 0.f;
      }
    }
  };
  const int steps = (R + BR - 1) / BR;
  const int vec_per_row = D / VEC;
  // the next step's rows are fetched into registers while this step is being multiplied
  constexpr int MAXP = 16;                           // 16-byte pieces per thread and step (D <= 512)
  uint4 pre[MAXP];
  auto fetch = [&](int step) {
    const int rb = step * BR;
#pragma unroll
    for (int j = 0; j < MAXP; ++j) {
      const int i = threadIdx.x + j * 256;
      if (i < BR * vec_per_row) {
        const int r = i / vec_per_row, v = i - r * vec_per_row;
        const int rr = min(rb + r, R - 1);
        pre[j] = *reinterpret_cast<const uint4*>(rows + (size_t)rr * D + v * VEC);
      }
    }
  };
  if ((int)blockIdx.x < steps) fetch(blockIdx.x);
  for (int step = blockIdx.x; step < steps; step += gridDim.x) {
    const int rb = step * BR;
    __syncthreads();                                 // previous step's readers are done (and wt is written)
#pragma unroll
    for (int j = 0; j < MAXP; ++j) {
      const int i = threadIdx.x + j * 256;
      if (i < BR * vec_per_row) {
        const int r = i / vec_per_row, v = i - r * vec_per_row;
        *reinterpret_cast<uint4*>(xs + (size_t)r * D + v * VEC) = pre[j];
      }
    }
    __syncthreads();
    if (step + (int)gridDim.x < steps) fetch(step + gridDim.x);
    const int r0 = rb + warp * RPW;
    float acc[RPW][EPL];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int q = 0; q < EPL; ++q) acc[r][q] = 0.f;
    const T* xw = xs + (size_t)warp * RPW * D;
#pragma unroll 2
    for (int d0 = 0; d0 < D; d0 += 8) {
      float w[8][EPL];
#pragma unroll
      for (int dd = 0; dd < 8; ++dd)
#pragma unroll
        for (int q = 0; q < EPL; ++q) w[dd][q] = wt[(d0 + dd) * EP + lane + 32 * q];
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        float x[8];
        load8(xw + (size_t)r * D + d0, x);
#pragma unroll
        for (int dd = 0; dd < 8; ++dd)
#pragma unroll
          for (int q = 0; q < EPL; ++q) acc[r][q] = fmaf(x[dd], w[dd][q], acc[r][q]);
      }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const int row = r0 + r;
      if (row >= R) break;                       // warp-uniform
      float lg[EPL], mx = -INFINITY;
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        int e = lane + 32 * q;
        lg[q] = (e < E) ? acc[r][q] + blog[q] : -INFINITY;
        mx = fmaxf(mx, lg[q]);
      }
      if (mode != 0) {
        // normalised variants: keep the raw logits for the backward, continue with the rescaled scores
        float ss = 0.f;
#pragma unroll
        for (int q = 0; q < EPL; ++q)
          if (lane + 32 * q < E) ss += lg[q] * lg[q];
        ss = warp_sum(ss);
        const float inv_n = 1.f / fmaxf(sqrtf(ss), norm_eps);
        mx = -INFINITY;
#pragma unroll
        for (int q = 0; q < EPL; ++q) {
          int e = lane + 32 * q;
          if (e < E) {
            logits_out[(size_t)row * E + e] = lg[q];
            float z = lg[q] * inv_n;
            lg[q] = (mode == 1 ? z : fmaxf(z, 0.f)) * rscale;
            mx = fmaxf(mx, lg[q]);
          }
        }
      }
      mx = warp_max(mx);
      float pr[EPL], sum = 0.f;
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        if (mode == 2) pr[q] = (lane + 32 * q < E) ? lg[q] : 0.f;
        else pr[q] = (lane + 32 * q < E) ? __expf(lg[q] - mx) : 0.f;
        sum += pr[q];
      }
      sum = warp_sum(sum);
      float inv = 1.f / sum, uniform = 0.f;
      if (mode == 2) {
        if (sum > 0.f) inv = 1.f / fmaxf(sum, 1e-9f);
        else { inv = 0.f; uniform = 1.f / (float)E; }
      }
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        int e = lane + 32 * q;
        pr[q] = (e < E) ? pr[q] * inv + uniform : 0.f;
        if (e < E) probs_out[(size_t)row * E + e] = pr[q];
      }
      const int b = row / rows_per_batch;
      if (b != cur_b) {
        flush();
        cur_b = b;
      }
#pragma unroll
      for (int q = 0; q < EPL; ++q) psum[q] += pr[q];
      // top-k by (logit + selection bias); ties go to the lower expert index
      float sc[EPL];
#pragma unroll
      for (int q = 0; q < EPL; ++q) sc[q] = (lane + 32 * q < E) ? lg[q] + bsel[q] : -INFINITY;
      int pick_e[kMaxTopK];
      float pick_p[kMaxTopK], psel = 0.f;
#pragma unroll
      for (int j = 0; j < kMaxTopK; ++j) {
        if (j >= topk) break;
        float bv = sc[0];
        int be = lane;
#pragma unroll
        for (int q = 1; q < EPL; ++q)
          if (sc[q] > bv) { bv = sc[q]; be = lane + 32 * q; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          float ov = __shfl_xor_sync(0xffffffffu, bv, o);
          int oe = __shfl_xor_sync(0xffffffffu, be, o);
          if (ov > bv || (ov == bv && oe < be)) { bv = ov; be = oe; }
        }
        // the owner lane hands out the probability and retires the expert
        float mine = 0.f;
#pragma unroll
        for (int q = 0; q < EPL; ++q)
          if (be == lane + 32 * q) { mine = pr[q]; sc[q] = -INFINITY; }
        pick_e[j] = be;
        pick_p[j] = __shfl_sync(0xffffffffu, mine, be & 31);
        psel += pick_p[j];
      }
      if (lane == 0) {
        const float scale = renorm ? alpha / fmaxf(psel, 1e-9f) : alpha;
#pragma unroll
        for (int j = 0; j < kMaxTopK; ++j) {
          if (j >= topk) break;
          idx_out[(size_t)row * topk + j] = pick_e[j];
          w_out[(size_t)row * topk + j] = pick_p[j] * scale;
        }
      }
    }
  }
  flush();
}

// ------------------------------------------------------------------------------------ forward on tensor cores
// logits[r, e] = <x[r], w[e]> with x in bf16 and w in fp32: w is the sum of three bf16 numbers (8 + 8 + 8 significant
// bits; what is left is below 2^-26 |w|), and products of bf16 numbers are exact in fp32.  The tensor core adds into its
// fp32 accumulator without rounding to nearest, an error that grows with every addition, so each 64-column slab has an
// accumulator of its own and the slabs are added in registers.  A thread owns a whole row of logits: softmax and top-k
// need no shuffles.
//   warp 8 / lane 0 : TMA producer, 64-column slabs of 128 rows -> ring
//   warp 9          : MMA issuer (an elected lane of the converged warp), accumulators of two tiles in flight
//   warps 0-3, 4-7  : softmax, top-k and balance sums of every other tile, thread = row
// One persistent block per SM; the three parts of the router stay in shared memory, swizzled as the B operand.  The
// general kernel is bound by its fp32 multiply-adds and their shared-memory reads.
// 196,608 rows of 64, 64 experts: 233 -> 28 us; 16,384 of 384, 32 experts: 45 -> 11 us; 4 of 192, 16 experts: 16 -> 7 us.
// Relative error of the logits against 64 bits (general kernel): 0.8e-7 (1.4e-7), 0.9e-7 (3.5e-7), 1.0e-7 (2.7e-7); with
// one accumulator for all slabs it was 1.1e-6 at 384 columns.
constexpr int kRtStages = 4;
constexpr int kRtSlab = 128 * 128;               // 128 rows x 64 bf16
constexpr int kRtPad = 4;                        // floats between staged probability rows: conflict-free 16-byte access

struct RouterTcParams {
  const float* router;
  const float* bias;
  int R, D, topk, rows_per_batch;
  float alpha;
  int bias_in_logits, renorm, mode;
  float rscale, norm_eps;
  int* idx;
  float* w;
  float* probs;
  float* probs_sum;
  float* logits;
  int* status;
};

__host__ __device__ constexpr int router_tc_smem(int D, int E) {
  return 3 * D * E * 2 + kRtStages * kRtSlab + 2 * 128 * (E + kRtPad) * 4 + 2 * E * 4 + 256 + 1024;
}

template <int E>
__global__ void __launch_bounds__(320, 1) router_fwd_tc_kernel(const __grid_constant__ CUtensorMap tx, RouterTcParams p) {
  extern __shared__ uint8_t smem_t[];
  const uint32_t base = (ptx::smem_u32(smem_t) + 1023u) & ~1023u;
  uint8_t* gen = smem_t + (base - ptx::smem_u32(smem_t));
  const int slabs = p.D / 64;
  const uint32_t part_bytes = (uint32_t)slabs * E * 128;            // one part of the router: [slab][E rows x 128 bytes]
  const uint32_t ring = base + 3 * part_bytes;
  const uint32_t stage_off = 3 * part_bytes + kRtStages * kRtSlab;
  float* bias_s = reinterpret_cast<float*>(gen + stage_off + 2 * 128 * (E + kRtPad) * 4);      // [2][E]: logits, selection
  const uint32_t bars = base + stage_off + 2 * 128 * (E + kRtPad) * 4 + 2 * E * 4;
  auto full = [&](int s) { return bars + 8 * s; };
  auto empty = [&](int s) { return bars + 32 + 8 * s; };
  auto acc_full = [&](int g) { return bars + 64 + 8 * g; };
  auto acc_empty = [&](int g) { return bars + 80 + 8 * g; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + (bars - base) + 96);
  const int warp = ptx::warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int tiles = (p.R + 127) / 128;
  {
    __shared__ int prior_failure;
    if (threadIdx.x == 0) prior_failure = (p.status != nullptr) ? *(volatile int*)p.status : 0;
    __syncthreads();
    if (prior_failure != 0) return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRtStages; ++s) {
      ptx::mbar_init(full(s), 1);
      ptx::mbar_init(empty(s), 1);
    }
    for (int g = 0; g < 2; ++g) {
      ptx::mbar_init(acc_full(g), 1);
      ptx::mbar_init(acc_empty(g), 128);
    }
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&tx);
  }
  for (int i = threadIdx.x; i < E * (p.D / 8); i += blockDim.x) {
    const int e = i / (p.D / 8), c8 = i % (p.D / 8);
    float v[8];
    Vec8<float>::load(p.router + (size_t)e * p.D + c8 * 8, v);
    const uint32_t off = (uint32_t)(c8 >> 3) * (E * 128) + e * 128 + (((c8 & 7) ^ (e & 7)) << 4);
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      Vec8<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(gen + part * part_bytes + off), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] -= __bfloat162float(__float2bfloat16(v[k]));
    }
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float b = p.bias != nullptr ? p.bias[e] : 0.f;
    bias_s[e] = p.bias_in_logits ? b : 0.f;
    bias_s[E + e] = p.bias_in_logits ? 0.f : b;
  }
  // two tiles in flight, a slab of a tile every kSlabCols columns (a load reads whole powers of two)
  constexpr uint32_t kCols = 512, kAcc = kCols / 2, kSlabCols = E <= 16 ? 16 : E <= 32 ? 32 : 64;
  if (warp == 8) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), kCols);
    ptx::tmem_relinquish();
  }
  ptx::fence_proxy_async();                       // the router parts were written through the generic proxy
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = ptx::warp_uniform(*tmem_slot);
  constexpr uint32_t idesc = ptx::make_instr_desc(128, E, 0, 0);
  bool ok = true;

  if (warp == 8 && lane == 0) {
    int it = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      for (int kb = 0; kb < slabs; ++kb, ++it) {
        const int s = it % kRtStages;
        if (it >= kRtStages) ok = ptx::mbar_wait(empty(s), (it / kRtStages - 1) & 1, p.status, 81);
        if (!ok) break;
        ptx::mbar_expect_tx(full(s), kRtSlab);
        ptx::tma_load_2d(ring + s * kRtSlab, &tx, full(s), kb * 64, t * 128);
      }
    }
  } else if (warp == 9) {
    int it = 0, n = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++n) {
      const int g = n & 1;
      if (n >= 2) ok = ptx::warp_wait(acc_empty(g), ((n >> 1) - 1) & 1, p.status, 82);
      if (!ok) break;
      ptx::tc_fence_after_sync();
      for (int kb = 0; kb < slabs; ++kb, ++it) {
        const int s = it % kRtStages;
        ok = ptx::warp_wait(full(s), (it / kRtStages) & 1, p.status, 83);
        if (!ok) break;
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
#pragma unroll
          for (int part = 2; part >= 0; --part) {   // small terms first
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint64_t da = ptx::make_smem_desc(ring + s * kRtSlab + k * 32, 16, 1024);
              const uint64_t db = ptx::make_smem_desc(base + part * part_bytes + kb * (E * 128) + k * 32, 16, 1024);
              ptx::mma_bf16_ss(tmem + g * kAcc + kb * kSlabCols, da, db, idesc, (part < 2 || k > 0) ? 1u : 0u);
            }
          }
          ptx::mma_commit(empty(s));
        }
      }
      if (ok && ptx::elect_one()) ptx::mma_commit(acc_full(g));
    }
  } else if (warp < 8) {
    const int g = warp >> 2, quarter = warp & 3, r_in = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    float* stage = reinterpret_cast<float*>(gen + stage_off) + g * 128 * (E + kRtPad);
    auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory"); };
    // balance sums: thread = (expert column, strand of rows), carried over the tiles of a sequence
    constexpr int kStrands = 128 / E, kStrandRows = 128 / kStrands;    // E = 48: 2 strands, 32 threads idle
    const int col = r_in % E, strand = r_in / E;
    float psum = 0.f;
    int cur_b = -1;
    int n = g;
    for (int t = blockIdx.x + g * gridDim.x; t < tiles; t += 2 * gridDim.x, n += 2) {
      // a failed wait must not leave part of the group at its barrier: the outcome is shared
      bool got = ptx::mbar_wait(acc_full(g), (n >> 1) & 1, p.status, 84);
      int all;
      asm volatile(
          "{\n\t.reg .pred P, Q;\n\tsetp.ne.b32 P, %1, 0;\n\tbarrier.cta.red.and.pred Q, %2, 128, P;\n\t"
          "selp.b32 %0, 1, 0, Q;\n\t}"
          : "=r"(all)
          : "r"((int)got), "r"(1 + g)
          : "memory");
      if (!all) break;
      ptx::tc_fence_after_sync();
      const int row = t * 128 + r_in;
      const bool live = row < p.R;
      float lg[E];
#pragma unroll
      for (int e = 0; e < E; ++e) lg[e] = bias_s[e];
      for (int kb = 0; kb < slabs; ++kb) {
        uint32_t raw[kSlabCols];
        if constexpr (E <= 16) ptx::tmem_ld_32x16(tmem + g * kAcc + kb * kSlabCols + lane_base, raw);
        else if constexpr (E <= 32) ptx::tmem_ld_32x32(tmem + g * kAcc + kb * kSlabCols + lane_base, raw);
        else ptx::tmem_ld_32x64(tmem + g * kAcc + kb * kSlabCols + lane_base, raw);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < E; ++e) lg[e] += __uint_as_float(raw[e]);
      }
      ptx::tc_fence_before_sync();
      ptx::mbar_arrive(acc_empty(g));
      if (p.mode != 0) {
        // normalised variants: keep the raw logits for the backward, continue with the rescaled scores
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) ss = fmaf(lg[e], lg[e], ss);
        const float inv_n = 1.f / fmaxf(sqrtf(ss), p.norm_eps);
        if (live) {
#pragma unroll
          for (int e = 0; e < E; e += 4)
            *reinterpret_cast<float4*>(p.logits + (size_t)row * E + e) = make_float4(lg[e], lg[e + 1], lg[e + 2], lg[e + 3]);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const float z = lg[e] * inv_n;
          lg[e] = (p.mode == 1 ? z : fmaxf(z, 0.f)) * p.rscale;
        }
      }
      float mx = lg[0];
#pragma unroll
      for (int e = 1; e < E; ++e) mx = fmaxf(mx, lg[e]);
      float pr[E], sum = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        pr[e] = p.mode == 2 ? lg[e] : __expf(lg[e] - mx);
        sum += pr[e];
      }
      float inv = 1.f / sum, uniform = 0.f;
      if (p.mode == 2) {
        if (sum > 0.f) inv = 1.f / fmaxf(sum, 1e-9f);
        else { inv = 0.f; uniform = 1.f / (float)E; }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) pr[e] = fmaf(pr[e], inv, uniform);
      // top-k by (logit + selection bias); ties go to the lower expert index
      int pick_e[kMaxTopK];
      float pick_p[kMaxTopK], psel = 0.f;
      uint64_t taken = 0;
#pragma unroll
      for (int j = 0; j < kMaxTopK; ++j) {
        if (j >= p.topk) break;
        float bv = -INFINITY, bp = pr[0];
        int be = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const float v = lg[e] + bias_s[E + e];
          if (v > bv && !((taken >> e) & 1)) { bv = v; be = e; bp = pr[e]; }
        }
        taken |= 1ull << be;
        pick_e[j] = be;
        pick_p[j] = bp;
        psel += bp;
      }
      if (live) {
        const float scale = p.renorm ? p.alpha / fmaxf(psel, 1e-9f) : p.alpha;
#pragma unroll
        for (int j = 0; j < kMaxTopK; ++j) {
          if (j >= p.topk) break;
          p.idx[(size_t)row * p.topk + j] = pick_e[j];
          p.w[(size_t)row * p.topk + j] = pick_p[j] * scale;
        }
      }
#pragma unroll
      for (int e = 0; e < E; e += 4)
        *reinterpret_cast<float4*>(stage + r_in * (E + kRtPad) + e) = make_float4(pr[e], pr[e + 1], pr[e + 2], pr[e + 3]);
      group_sync();
      const int rows_here = min(128, p.R - t * 128);
      for (int i = r_in; i < rows_here * (E / 4); i += 128) {
        const int r = i / (E / 4), c = i % (E / 4);
        reinterpret_cast<float4*>(p.probs)[(size_t)t * 128 * (E / 4) + i] =
            *reinterpret_cast<const float4*>(stage + r * (E + kRtPad) + c * 4);
      }
      if (strand < kStrands) {
        int r = strand * kStrandRows;
        const int end = min(rows_here, r + kStrandRows);
        while (r < end) {
          const int b = (t * 128 + r) / p.rows_per_batch;
          if (b != cur_b) {
            if (cur_b >= 0) atomicAdd(p.probs_sum + (size_t)cur_b * E + col, psum);
            psum = 0.f;
            cur_b = b;
          }
          const int stop = (int)min((long long)end, (long long)(b + 1) * p.rows_per_batch - (long long)t * 128);
          for (; r < stop; ++r) psum += stage[r * (E + kRtPad) + col];
        }
      }
      group_sync();                               // the stage is free for the next tile
    }
    if (cur_b >= 0) atomicAdd(p.probs_sum + (size_t)cur_b * E + col, psum);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) ptx::tmem_dealloc(tmem, kCols);
}

// ------------------------------------------------------------------------------------ backward: d logits, d rows
template <typename T, int EPL, int DPL, int RPW>
__global__ void __launch_bounds__(256) router_bwd_rows_kernel(
    const float* __restrict__ router, const float* __restrict__ probs, const int* __restrict__ idx,
    const float* __restrict__ dw, const float* __restrict__ dpsum, int R, int D, int E, int topk, int rows_per_batch,
    float alpha, int renorm, float* __restrict__ dlogits, T* __restrict__ drows, int mode, float rscale,
    float norm_eps, const float* __restrict__ logits) {
  extern __shared__ float ws[];                 // [E][D] router matrix
  for (int i = threadIdx.x; i < E * D; i += blockDim.x) ws[i] = router[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int groups = (R + RPW - 1) / RPW;
  for (int g = warp_global; g < groups; g += nwarps) {
    const int r0 = g * RPW;
    float dl[RPW][EPL];
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const int row = min(r0 + r, R - 1);
      const int b = row / rows_per_batch;
      float pr[EPL], dp[EPL];
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        int e = lane + 32 * q;
        pr[q] = (e < E) ? probs[(size_t)row * E + e] : 0.f;
        dp[q] = (e < E && dpsum != nullptr) ? dpsum[(size_t)b * E + e] : 0.f;
      }
      if (dw != nullptr) {
        // weights_j = alpha p_j            -> d p_j = alpha dw_j
        // weights_j = alpha p_j / S        -> d p_j = alpha (dw_j - sum_i dw_i p_i / S) / S,  S = sum_sel p
        float s_sel = 0.f, dot = 0.f;
        int ej[kMaxTopK];
        float gj[kMaxTopK];
#pragma unroll
        for (int j = 0; j < kMaxTopK; ++j) {
          if (j >= topk) break;
          ej[j] = idx[(size_t)row * topk + j];
#ifdef UTTT_BOUNDS_CHECK
          if (ej[j] < 0 || ej[j] >= E) ej[j] = 0;         // reported by the host-side check of the index table
#endif
          gj[j] = dw[(size_t)row * topk + j];
          float pj = __shfl_sync(0xffffffffu, (ej[j] >> 5) == 0 ? pr[0] : pr[EPL - 1], ej[j] & 31);
          s_sel += pj;
          dot += gj[j] * pj;
        }
        const float s_c = fmaxf(s_sel, 1e-9f);
#pragma unroll
        for (int j = 0; j < kMaxTopK; ++j) {
          if (j >= topk) break;
          float contrib = renorm ? alpha * (gj[j] - dot / s_c) / s_c : alpha * gj[j];
#pragma unroll
          for (int q = 0; q < EPL; ++q)
            if (ej[j] == lane + 32 * q) dp[q] += contrib;
        }
      }
      float inner = 0.f;
#pragma unroll
      for (int q = 0; q < EPL; ++q) inner += dp[q] * pr[q];
      inner = warp_sum(inner);
      if (mode == 0) {
#pragma unroll
        for (int q = 0; q < EPL; ++q) dl[r][q] = pr[q] * (dp[q] - inner);
      } else {
        // z = l / max(|l|, eps); scores = z s (mode 1) or relu(z) s (mode 2)
        float lr_[EPL], z[EPL], ss = 0.f;
#pragma unroll
        for (int q = 0; q < EPL; ++q) {
          int e = lane + 32 * q;
          lr_[q] = (e < E) ? logits[(size_t)row * E + e] : 0.f;
          ss += lr_[q] * lr_[q];
        }
        ss = warp_sum(ss);
        const float nr = sqrtf(ss), inv_n = 1.f / fmaxf(nr, norm_eps);
        float ssum = 0.f;
#pragma unroll
        for (int q = 0; q < EPL; ++q) {
          z[q] = lr_[q] * inv_n;
          ssum += fmaxf(z[q], 0.f) * rscale;
        }
        float dz[EPL], zdot = 0.f;
        if (mode == 2) ssum = warp_sum(ssum);
#pragma unroll
        for (int q = 0; q < EPL; ++q) {
          float dsel;
          if (mode == 1) dsel = pr[q] * (dp[q] - inner);
          else if (ssum >= 1e-9f) dsel = (dp[q] - inner) / ssum;
          else dsel = ssum > 0.f ? dp[q] * 1e9f : 0.f;
          dz[q] = (mode == 2 && z[q] <= 0.f) ? 0.f : dsel * rscale;
          if (lane + 32 * q >= E) dz[q] = 0.f;
          zdot += dz[q] * z[q];
        }
        zdot = warp_sum(zdot);
        const bool clamped = nr <= norm_eps;       // the clamp cuts the gradient through the norm
#pragma unroll
        for (int q = 0; q < EPL; ++q) dl[r][q] = (clamped ? dz[q] : dz[q] - z[q] * zdot) * inv_n;
      }
#pragma unroll
      for (int q = 0; q < EPL; ++q) {
        int e = lane + 32 * q;
        if (e < E && r0 + r < R) dlogits[(size_t)row * E + e] = dl[r][q];
      }
    }
    if (drows == nullptr) continue;
    float acc[RPW][DPL];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[r][i] = 0.f;
    for (int e = 0; e < E; ++e) {
      float w[DPL];
#pragma unroll
      for (int i = 0; i < DPL; ++i) {
        int d = lane + 32 * i;
        w[i] = (d < D) ? ws[e * D + d] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        float v = __shfl_sync(0xffffffffu, (e >> 5) == 0 ? dl[r][0] : dl[r][EPL - 1], e & 31);
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[r][i] = fmaf(v, w[i], acc[r][i]);
      }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      if (r0 + r >= R) break;
#pragma unroll
      for (int i = 0; i < DPL; ++i) {
        int d = lane + 32 * i;
        if (d < D) drows[(size_t)(r0 + r) * D + d] = static_cast<T>(acc[r][i]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------ backward: d router
// block = 256 threads = 8 expert groups x 32 lanes; thread tile = EG experts x DPL slices of D.  Every block
// reduces `chunk` rows and writes its [E, D] partial to scratch; the partials are summed afterwards.
template <typename T, int EG, int DPL>
__global__ void __launch_bounds__(256) router_bwd_weight_kernel(const T* __restrict__ rows,
                                                                const float* __restrict__ dlogits, int R, int D,
                                                                int E, int chunk, float* __restrict__ partial) {
  constexpr int SUB = 32;                         // rows staged per step
  constexpr int VEC = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) uint8_t smem_w[];
  float* xs = reinterpret_cast<float*>(smem_w);                   // [SUB][D]
  float* ds = xs + SUB * D;                                       // [SUB][E]
  const int lane = threadIdx.x & 31, eg = threadIdx.x >> 5;
  const int r_begin = blockIdx.x * chunk, r_end = min(R, r_begin + chunk);
  const int vec_per_row = D / VEC;
  float acc[EG][DPL];
#pragma unroll
  for (int a = 0; a < EG; ++a)
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[a][i] = 0.f;
  for (int rs = r_begin; rs < r_end; rs += SUB) {
    const int nr = min(SUB, r_end - rs);
    __syncthreads();
    for (int i = threadIdx.x; i < SUB * vec_per_row; i += blockDim.x) {
      int r = i / vec_per_row, v = i - r * vec_per_row;
      float f[VEC];
      if (r < nr) {
        if (VEC == 8) load8(rows + (size_t)(rs + r) * D + v * VEC, *reinterpret_cast<float (*)[8]>(&f[0]));
        else {
          float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(rows) + (size_t)(rs + r) * D + v * 4);
          f[0] = t.x; f[1] = t.y; f[2] = t.z; f[3] = t.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) f[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < VEC; j += 4)
        *reinterpret_cast<float4*>(xs + r * D + v * VEC + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
    }
    for (int i = threadIdx.x; i < SUB * E; i += blockDim.x) {
      int r = i / E;
      ds[i] = (r < nr) ? dlogits[(size_t)rs * E + i] : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < SUB; ++r) {
      float x[DPL], g[EG];
#pragma unroll
      for (int i = 0; i < DPL; ++i) {
        int d = lane + 32 * i;
        x[i] = (d < D) ? xs[r * D + d] : 0.f;
      }
#pragma unroll
      for (int a = 0; a < EG; ++a) g[a] = ds[r * E + eg * EG + a];
#pragma unroll
      for (int a = 0; a < EG; ++a)
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[a][i] = fmaf(g[a], x[i], acc[a][i]);
    }
  }
  float* out = partial + (size_t)blockIdx.x * E * D;
#pragma unroll
  for (int a = 0; a < EG; ++a)
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      int d = lane + 32 * i;
      if (d < D) out[(size_t)(eg * EG + a) * D + d] = acc[a][i];
    }
}

// ------------------------------------------------------------------------------------ host
static int sm_count() { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }

// Supported shapes of the fused path (anything else takes the unfused route in Python).
bool router_supported(int64_t D, int64_t E, int64_t topk) {
  return D % 8 == 0 && D <= 512 && E % 8 == 0 && E <= 64 && topk >= 1 && topk <= kMaxTopK && topk <= E;
}

// returns (idx [R, k] int32, weights [R, k] fp32, probs [R, E] fp32, probs_sum [B, E] fp32,
//          raw logits [R, E] fp32 for modes 1 and 2, empty for mode 0)
std::vector<at::Tensor> router_fwd(at::Tensor rows, at::Tensor router, c10::optional<at::Tensor> bias, int64_t topk,
                                   int64_t rows_per_batch, double alpha, bool bias_in_logits, bool renorm,
                                   int64_t mode, double rscale, double norm_eps) {
  c10::cuda::CUDAGuard guard(rows.device());
  TORCH_CHECK(rows.dim() == 2 && rows.is_contiguous() && router.is_contiguous() && router.scalar_type() == at::kFloat);
  const int R = rows.size(0), D = rows.size(1), E = router.size(0);
  TORCH_CHECK(router.size(1) == D && router_supported(D, E, topk) && R % rows_per_batch == 0);
  rows = dense16(rows);                           // both variants fetch rows 16 bytes at a time
  const float* bp = nullptr;
  at::Tensor bc;
  if (bias.has_value() && bias->defined()) {
    bc = bias->to(at::kFloat).contiguous();
    TORCH_CHECK(bc.numel() == E);
    bp = bc.data_ptr<float>();
  }
  auto opts = rows.options();
  auto idx = at::empty({R, topk}, opts.dtype(at::kInt));
  auto w = at::empty({R, topk}, opts.dtype(at::kFloat));
  auto probs = at::empty({R, E}, opts.dtype(at::kFloat));
  auto psum = at::zeros({R / rows_per_batch, E}, opts.dtype(at::kFloat));
  TORCH_CHECK(mode >= 0 && mode <= 2, "router mode: 0 softmax, 1 norm_softmax, 2 norm_relu");
  auto logits = mode != 0 ? at::empty({R, E}, opts.dtype(at::kFloat)) : at::empty({0}, opts.dtype(at::kFloat));
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  // Tensor cores need whole 64-column slabs, an expert count that is an MMA width, room for the three router parts, and an
  // accumulator per slab and tile; the general kernel reads the router one value at a time, from any address.
  const int tc_smem = router_tc_smem(D, E);
  const int slab_cols = E <= 16 ? 16 : E <= 32 ? 32 : 64;
  if (rows.scalar_type() == at::kBFloat16 && D % 64 == 0 && E % 16 == 0 && tc_smem <= 227 * 1024 - 64 && D / 64 * slab_cols <= 256 && R > 0 &&
      ((uintptr_t)router.data_ptr() & 15) == 0) {
    RouterTcParams tp{router.data_ptr<float>(), bp, R, D, (int)topk, (int)rows_per_batch, (float)alpha,
                      bias_in_logits ? 1 : 0, renorm ? 1 : 0, (int)mode, (float)rscale, (float)norm_eps,
                      idx.data_ptr<int>(), w.data_ptr<float>(), probs.data_ptr<float>(), psum.data_ptr<float>(),
                      logits.data_ptr<float>(), gemm_status(rows).data_ptr<int>()};
    auto tx = make_tmap_2d_bf16(rows.data_ptr(), R, D, 128, 64);
    const int blocks = std::min((R + 127) / 128, sm_count());
    auto launch = [&](auto kernel) {
      C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem));
      kernel<<<blocks, 320, tc_smem, stream>>>(tx, tp);
      C10_CUDA_KERNEL_LAUNCH_CHECK();
    };
    if (E == 16) launch(router_fwd_tc_kernel<16>);
    else if (E == 32) launch(router_fwd_tc_kernel<32>);
    else if (E == 48) launch(router_fwd_tc_kernel<48>);
    else launch(router_fwd_tc_kernel<64>);
    count_launch();
    return {idx, w, probs, psum, logits};
  }
  const int epl = E > 32 ? 2 : 1;
  const bool bf = rows.scalar_type() == at::kBFloat16;
  const int rpw = bf ? 8 : 4;
  const size_t smem = (((size_t)D * (32 * epl + 1) * 4 + 15) & ~(size_t)15) + (size_t)8 * rpw * D * (bf ? 2 : 4);
  const int steps = (R + 8 * rpw - 1) / (8 * rpw);
  const int blocks = std::max(1, std::min(steps, 2 * sm_count()));
  auto launch = [&](auto kernel, auto* rp) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<blocks, 256, smem, stream>>>(rp, router.data_ptr<float>(), bp, R, D, E, (int)topk, (int)rows_per_batch,
                                          (float)alpha, bias_in_logits ? 1 : 0, renorm ? 1 : 0, idx.data_ptr<int>(),
                                          w.data_ptr<float>(), probs.data_ptr<float>(), psum.data_ptr<float>(),
                                          (int)mode, (float)rscale, (float)norm_eps, logits.data_ptr<float>());
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  if (rows.scalar_type() == at::kBFloat16) {
    auto* rp = reinterpret_cast<const __nv_bfloat16*>(rows.data_ptr());
    if (epl == 1) launch(router_fwd_kernel<__nv_bfloat16, 1, 8>, rp);
    else launch(router_fwd_kernel<__nv_bfloat16, 2, 8>, rp);
  } else {
    TORCH_CHECK(rows.scalar_type() == at::kFloat);
    auto* rp = rows.data_ptr<float>();
    if (epl == 1) launch(router_fwd_kernel<float, 1, 4>, rp);
    else launch(router_fwd_kernel<float, 2, 4>, rp);
  }
  count_launch();
  return {idx, w, probs, psum, logits};
}

template <typename T, int EPL>
static void launch_bwd_rows(int dpl, const float* router, const float* probs, const int* idx, const float* dw,
                            const float* dpsum, int R, int D, int E, int topk, int rpb, float alpha, int renorm,
                            float* dlogits, T* drows, cudaStream_t stream, int mode, float rscale, float norm_eps,
                            const float* logits) {
  const size_t smem = (size_t)E * D * sizeof(float);
  auto go = [&](auto kernel, int rpw) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int groups = (R + rpw - 1) / rpw;
    const int blocks = std::max(1, std::min((groups + 7) / 8, 2 * sm_count()));
    kernel<<<blocks, 256, smem, stream>>>(router, probs, idx, dw, dpsum, R, D, E, topk, rpb, alpha, renorm, dlogits,
                                          drows, mode, rscale, norm_eps, logits);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  // slices of 32 columns per lane: with four of them for a head of 64 half of the multiply-adds were by zero (196,608
  // rows, 64 experts: 194 -> 161 us)
  if (dpl <= 2) go(router_bwd_rows_kernel<T, EPL, 2, 8>, 8);
  else if (dpl <= 4) go(router_bwd_rows_kernel<T, EPL, 4, 8>, 8);
  else if (dpl <= 8) go(router_bwd_rows_kernel<T, EPL, 8, 8>, 8);
  else if (dpl <= 12) go(router_bwd_rows_kernel<T, EPL, 12, 8>, 8);
  else go(router_bwd_rows_kernel<T, EPL, 16, 4>, 4);
}

template <typename T, int EG>
static void launch_bwd_weight(int dpl, const T* rows, const float* dlogits, int R, int D, int E, float* partial,
                              int chunk, cudaStream_t stream) {
  const int blocks = (R + chunk - 1) / chunk;
  const size_t smem = (size_t)32 * (D + E) * sizeof(float);
  auto go = [&](auto kernel) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<blocks, 256, smem, stream>>>(rows, dlogits, R, D, E, chunk, partial);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  if (dpl <= 4) go(router_bwd_weight_kernel<T, EG, 4>);
  else if (dpl <= 8) go(router_bwd_weight_kernel<T, EG, 8>);
  else if (dpl <= 12) go(router_bwd_weight_kernel<T, EG, 12>);
  else go(router_bwd_weight_kernel<T, EG, 16>);
}

// returns (d rows [R, D] in the dtype of rows, d router [E, D] fp32)
std::vector<at::Tensor> router_bwd(at::Tensor rows, at::Tensor router, at::Tensor probs, at::Tensor idx,
                                   c10::optional<at::Tensor> dweights, c10::optional<at::Tensor> dprobs_sum,
                                   int64_t rows_per_batch, double alpha, bool renorm, bool need_drows, int64_t mode,
                                   double rscale, double norm_eps, c10::optional<at::Tensor> logits) {
  c10::cuda::CUDAGuard guard(rows.device());
  const int R = rows.size(0), D = rows.size(1), E = router.size(0), topk = idx.size(1);
  TORCH_CHECK(router_supported(D, E, topk) && probs.is_contiguous() && idx.is_contiguous() && rows.is_contiguous());
  rows = dense16(rows);
  at::Tensor dwc, dpc;
  const float *dwp = nullptr, *dpp = nullptr;
  if (dweights.has_value() && dweights->defined()) {
    dwc = dweights->to(at::kFloat).contiguous();
    dwp = dwc.data_ptr<float>();
  }
  if (dprobs_sum.has_value() && dprobs_sum->defined()) {
    dpc = dprobs_sum->to(at::kFloat).contiguous();
    dpp = dpc.data_ptr<float>();
  }
  const float* lgp = nullptr;
  if (mode != 0) {
    TORCH_CHECK(logits.has_value() && logits->defined() && logits->is_contiguous() && logits->numel() == (int64_t)R * E,
                "the normalised router modes need the raw logits of the forward");
    lgp = logits->data_ptr<float>();
  }
  auto dlogits = at::empty({R, E}, probs.options());
  auto drows = need_drows ? at::empty_like(rows) : at::Tensor();
  // rows per block of the weight reduction; two long blocks per SM took 177 us at 196,608 rows of 64 where these take 137
  const int wchunk = 128;
  auto partial = at::empty({(R + wchunk - 1) / wchunk, E, D}, router.options());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const int dpl = (D + 31) / 32;
  const bool bf = rows.scalar_type() == at::kBFloat16;
  TORCH_CHECK(bf || rows.scalar_type() == at::kFloat);
  const float* rt = router.data_ptr<float>();
  const float* pp = probs.data_ptr<float>();
  const int* ip = idx.data_ptr<int>();
  float* dl = dlogits.data_ptr<float>();
#define UTTT_ROUTER_BWD(T_, EPL_)                                                                              \
  launch_bwd_rows<T_, EPL_>(dpl, rt, pp, ip, dwp, dpp, R, D, E, topk, (int)rows_per_batch, (float)alpha,       \
                            renorm ? 1 : 0, dl, need_drows ? reinterpret_cast<T_*>(drows.data_ptr()) : nullptr, \
                            stream, (int)mode, (float)rscale, (float)norm_eps, lgp)
  if (bf) {
    if (E > 32) UTTT_ROUTER_BWD(__nv_bfloat16, 2); else UTTT_ROUTER_BWD(__nv_bfloat16, 1);
  } else {
    if (E > 32) UTTT_ROUTER_BWD(float, 2); else UTTT_ROUTER_BWD(float, 1);
  }
#undef UTTT_ROUTER_BWD
#define UTTT_ROUTER_BWD_W(T_)                                                                                  \
  do {                                                                                                         \
    auto* rp = reinterpret_cast<const T_*>(rows.data_ptr());                                                   \
    float* dr = partial.data_ptr<float>();                                                                     \
    switch (E / 8) {                                                                                           \
      case 1: launch_bwd_weight<T_, 1>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 2: launch_bwd_weight<T_, 2>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 3: launch_bwd_weight<T_, 3>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 4: launch_bwd_weight<T_, 4>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 5: launch_bwd_weight<T_, 5>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 6: launch_bwd_weight<T_, 6>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      case 7: launch_bwd_weight<T_, 7>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                               \
      default: launch_bwd_weight<T_, 8>(dpl, rp, dl, R, D, E, dr, wchunk, stream); break;                              \
    }                                                                                                          \
  } while (0)
  if (bf) UTTT_ROUTER_BWD_W(__nv_bfloat16); else UTTT_ROUTER_BWD_W(float);
#undef UTTT_ROUTER_BWD_W
  count_launch();
  count_launch();
  auto drouter = col_sum(partial);
  if (!need_drows) drows = at::empty({0}, rows.options());
  return {drows, drouter};
}

}  // namespace uttt
