// Sliding-window causal attention, backward, on tcgen05 tensor cores with TMEM accumulators.
//
// Same problem statement as the forward kernel: q [b, lq, h, hd], k/v [b, lk, h, hd] (bf16), the queries are
// aligned to the last lq keys, key j is visible to query i (absolute position p = lk - lq + i) iff j <= p and
// j > p - window (causal), or every key is visible (non-causal).  With P = exp(scale * S - lse) and
// D_i = sum_d dO_id O_id:
//     dV = P^T dO          dP = dO V^T          dS = P o (dP - D) * scale
//     dK = dS^T Q          dQ = dS K
//
// Three launches (and one memset of the dQ sums):
//   swa_bwd_prep_kernel    -D and -lse * log2(e), padded along the query axis so that the tiles below can fetch
//                          them with 16-byte aligned bulk copies
//   swa_bwd_kernel         one CTA per (batch, head, 128-key tile), keys on the TMEM lanes: walks the 128-query
//                          tiles of its band.  S^T = K Q^T and dP^T = V dO^T in TMEM; P^T goes back to TMEM as the A
//                          operand of dV += P^T dO, dS^T to shared memory, where it is the A operand of both
//                          dK += dS^T Q (as stored) and dQ = dS K (read transposed).  dK and dV stay in TMEM for the
//                          whole band; the dQ tile takes the columns of dP^T, and four warps add it to fp32 sums in
//                          global memory with vector reductions
//   swa_bwd_dq_out_kernel  fp32 dQ sums -> bf16, scaled
// S, P and dS are formed once for all three gradients: five products and one exponential per element, where separate
// dK/dV and dQ kernels needed seven and two.  The price is the addition of dQ in L2 (48 KB per tile at 96), in no fixed
// order unless deterministic algorithms are asked for (see launch_bwd), to fp32 sums of b * h * ceil(lq, 128) * hd that
// are allocated and cleared on every call: 50 MB at 4 x 16 heads x 96 with 2048 queries.
// Bound by the hand-overs between the products and the warps.  Measured with its preparation and conversion:
// 785 -> 459 us at that size on 4096 keys, window 2048.
// Warps: 0-7 P and dS (two per TMEM lane quarter, each owning half of the 128 columns of a tile), 8-11 dQ,
// 12 TMA producer (one lane), 13 MMA issuer (an elected lane of the converged warp).
// Every wait is bounded (ptx::mbar_wait).
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cudaTypedefs.h>
#include <torch/extension.h>

#include "common.cuh"
#include "ptx.cuh"

namespace uttt {

CUtensorMap make_tmap_3d_bf16(const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1_bytes,
                              uint64_t stride2_bytes, uint32_t box0, uint32_t box1);
at::Tensor gemm_status(at::Tensor like);

struct SwaBwdParams {
  int lq, lk, heads, lq_pad;
  int window;          // 0 = unlimited
  int causal;
  int kt_first, kt_step;   // the launch's key tiles: kt_first + blockIdx.x * kt_step
  float scale, scale_log2;
  const float* nlse2;  // [b, h, lq_pad]  -lse * log2(e); -inf on padding rows
  const float* ndsum;  // [b, h, lq_pad]  -D; 0 on padding rows
  float* dq_sum;       // [b, h, lq_pad / 128][hd / 4][128 rows][4]: a warp's vector reductions are contiguous
  __nv_bfloat16* dk;   // [b, lk, h, hd]
  __nv_bfloat16* dv;
  int* status;
};

// ------------------------------------------------------------------------------------ D and scaled lse
template <int HD>
__global__ void swa_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                    const float* __restrict__ lse, float* __restrict__ nlse2,
                                    float* __restrict__ ndsum, int lq, int lq_pad, int heads, int total) {
  // one 8-lane group per (batch, head, padded query) row; each lane takes 16-byte pieces of the head vector
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  if (gid >= total) return;
  const int i = gid % lq_pad;
  const int bh = gid / lq_pad;
  const int head = bh % heads, batch = bh / heads;
  float acc = 0.f;
  if (i < lq) {
    const size_t off = (((size_t)batch * lq + i) * heads + head) * HD;
    for (int c = sub * 8; c < HD; c += 64) {
      float a[8], g[8];
      Vec8<__nv_bfloat16>::load(o + off + c, a);
      Vec8<__nv_bfloat16>::load(dout + off + c, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += a[j] * g[j];
    }
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  if (sub == 0) {
    ndsum[gid] = (i < lq) ? -acc : 0.f;
    float l = (i < lq) ? lse[(size_t)bh * lq + i] : INFINITY;
    // a row that saw no key (lse = -inf) gets P = 0, like a padding row
    nlse2[gid] = (l == -INFINITY) ? -INFINITY : l * -1.4426950408889634f;
  }
}

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void red_add_v4(float* dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(__uint_as_float(a)),
               "f"(__uint_as_float(b)), "f"(__uint_as_float(c)), "f"(__uint_as_float(d))
               : "memory");
}

// ------------------------------------------------------------------------------------ dQ, dK, dV
constexpr int kT = 128;                      // keys per CTA and queries per tile
constexpr int kSlab = 128 * 128;             // 128 rows x 64 bf16, one 128-byte swizzle row each

// Four warpgroups at 128 registers each; P and dS take 152, dQ keeps 128, the issuing warps give their share up:
// 2 x 152 + 128 + 72 <= 4 x 128.
constexpr int kThreads = 512;
constexpr int kComputeRegs = 152, kIssueRegs = 72;
static_assert(2 * kComputeRegs + 128 + kIssueRegs <= 4 * 128, "more registers than the block is launched with");

template <int HD>
struct BwdCfg {
  static constexpr int KB = (HD + 63) / 64;  // 64-wide slabs along the head dimension
  static constexpr int kTile = KB * kSlab;
  // K | V | 2 x Q | dO | dS^T | 2 x (-lse2 512, -D 512) | barriers | tmem slot
  static constexpr int kV = kTile, kQ = 2 * kTile, kDO = 4 * kTile, kDS = 5 * kTile, kVec = kDS + 2 * kSlab;
  static constexpr int kBars = kVec + 2048;
  static constexpr int kSmem = kBars + 256 + 1024;
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 1) swa_bwd_kernel(const __grid_constant__ CUtensorMap tq,
                                                         const __grid_constant__ CUtensorMap tdo,
                                                         const __grid_constant__ CUtensorMap tk,
                                                         const __grid_constant__ CUtensorMap tv, SwaBwdParams p) {
  using C = BwdCfg<HD>;
  constexpr int KB = C::KB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - ptx::smem_u32(smem_raw));
  const uint32_t k_smem = base, v_smem = base + C::kV, do_smem = base + C::kDO, ds_smem = base + C::kDS;
  auto q_smem = [&](int s) { return base + C::kQ + s * C::kTile; };
  const uint32_t bars = base + C::kBars;
  const uint32_t kv_full = bars, do_full = bars + 8, do_empty = bars + 16, s_done = bars + 24, p_ready = bars + 32,
                 dp_done = bars + 40, ds_ready = bars + 48, dq_done = bars + 56, dq_free = bars + 64, acc_done = bars + 72;
  auto q_full = [&](int s) { return bars + 80 + 8 * s; };
  auto q_empty = [&](int s) { return bars + 96 + 8 * s; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + C::kBars + 128);

  const int warp = ptx::warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int head = blockIdx.y, batch = blockIdx.z;
  const int k0 = (p.kt_first + (int)blockIdx.x * p.kt_step) * kT;
  const int shift = p.lk - p.lq;
  // queries that can see any key of [k0, k0 + 127]
  int first_q = 0, last_q = p.lq - 1;
  if (p.causal) {
    first_q = max(0, k0 - shift);
    if (p.window > 0) last_q = min(p.lq - 1, k0 + kT - 2 + p.window - shift);
  }
  const int t0 = first_q / kT;
  const int nq = (last_q >= first_q) ? (last_q / kT - t0 + 1) : 0;

  {
    __shared__ int prior_failure;
    if (threadIdx.x == 0) prior_failure = (p.status != nullptr) ? *(volatile int*)p.status : 0;
    __syncthreads();
    if (prior_failure != 0) return;
  }
  if (nq == 0) {
    // no query sees these keys: their gradients are zero
    for (int idx = threadIdx.x; idx < kT * (HD / 8); idx += blockDim.x) {
      int r = idx / (HD / 8), c = (idx % (HD / 8)) * 8;
      if (k0 + r < p.lk) {
        size_t off = (((size_t)batch * p.lk + k0 + r) * p.heads + head) * HD + c;
        *reinterpret_cast<uint4*>(p.dk + off) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(p.dv + off) = make_uint4(0, 0, 0, 0);
      }
    }
    return;
  }
  if (threadIdx.x == 0) {
    for (uint32_t bar : {kv_full, do_full, do_empty, s_done, dp_done, dq_done, acc_done, q_full(0), q_full(1),
                         q_empty(0), q_empty(1)})
      ptx::mbar_init(bar, 1);
    ptx::mbar_init(p_ready, 256);
    ptx::mbar_init(ds_ready, 256);
    ptx::mbar_init(dq_free, 128);
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&tq);
    ptx::tma_prefetch_desc(&tdo);
    ptx::tma_prefetch_desc(&tk);
    ptx::tma_prefetch_desc(&tv);
  }
  if (warp == 12) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = ptx::warp_uniform(*tmem_slot);
  const uint32_t tmem_dk = tmem, tmem_dv = tmem + 128;
  const uint32_t tmem_s = tmem + 256;         // S^T; each column half's P^T (bf16, 32 columns) replaces its first half
  const uint32_t tmem_dp = tmem + 384;        // dP^T, then the dQ tile
  const size_t bh = (size_t)batch * p.heads + head;

  constexpr uint32_t idesc_s = ptx::make_instr_desc(kT, kT, 0, 0);
  constexpr uint32_t idesc_acc = ptx::make_instr_desc(kT, HD, 0, 1);
  constexpr uint32_t idesc_dq = ptx::make_instr_desc(kT, HD, 1, 1);
  bool ok = true;

  // each role's code stays inside the branch that sets its register share
  if (warp >= 12) {
    ptx::reg_dec<kIssueRegs>();
    if (warp == 12 && lane == 0) {
      // ================= producer =================
      auto load = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int row) {
        for (int kb = 0; kb < KB; ++kb) ptx::tma_load_3d(dst + kb * kSlab, map, bar, head * HD + kb * 64, row, batch);
      };
      for (int j = 0; j < nq && ok; ++j) {
        const int s = j & 1, q0 = (t0 + j) * kT;
        if (j == 0) {
          ptx::mbar_expect_tx(kv_full, 2 * C::kTile);
          load(k_smem, &tk, kv_full, k0);
        }
        if (j >= 2) ok = ptx::mbar_wait(q_empty(s), ((j >> 1) - 1) & 1, p.status, 31);
        if (!ok) break;
        ptx::mbar_expect_tx(q_full(s), C::kTile + 2 * kT * 4);
        load(q_smem(s), &tq, q_full(s), q0);
        const size_t vec = bh * p.lq_pad + q0;
        bulk_load_1d(base + C::kVec + s * 1024, p.nlse2 + vec, kT * 4, q_full(s));
        bulk_load_1d(base + C::kVec + s * 1024 + 512, p.ndsum + vec, kT * 4, q_full(s));
        if (j == 0) load(v_smem, &tv, kv_full, k0);
        if (j >= 1) ok = ptx::mbar_wait(do_empty, (j - 1) & 1, p.status, 32);
        if (!ok) break;
        ptx::mbar_expect_tx(do_full, C::kTile);
        load(do_smem, &tdo, do_full, q0);
      }
    } else if (warp == 13) {
      // ================= MMA issuer =================
      // One thread issues every product, and the tensor core runs them in order.  So S(j+1) may take the columns of
      // P(j) after dV has read them, and dp_done(j+1) also says that dQ(j) and dK(j) have read dS(j).
      const bool leader = ptx::elect_one();
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1;
        if (!ptx::warp_wait(q_full(s), (j >> 1) & 1, p.status, 33)) return false;
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint64_t da = ptx::make_smem_desc(k_smem + (k >> 2) * kSlab + (k & 3) * 32, 16, 1024);
          const uint64_t db = ptx::make_smem_desc(q_smem(s) + (k >> 2) * kSlab + (k & 3) * 32, 16, 1024);
          if (leader) ptx::mma_bf16_ss(tmem_s, da, db, idesc_s, k > 0 ? 1u : 0u);
        }
        if (leader) ptx::mma_commit(s_done);
        return true;
      };
      auto issue_dp = [&](int j) -> bool {
        if (!ptx::warp_wait(do_full, j & 1, p.status, 34)) return false;
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint64_t da = ptx::make_smem_desc(v_smem + (k >> 2) * kSlab + (k & 3) * 32, 16, 1024);
          const uint64_t db = ptx::make_smem_desc(do_smem + (k >> 2) * kSlab + (k & 3) * 32, 16, 1024);
          if (leader) ptx::mma_bf16_ss(tmem_dp, da, db, idesc_s, k > 0 ? 1u : 0u);
        }
        if (leader) ptx::mma_commit(dp_done);
        return true;
      };
      ok = ptx::warp_wait(kv_full, 0, p.status, 35) && issue_s(0) && issue_dp(0);
      // P and dS are zero where they are masked (dS is NaN there when dP is), but zero times a NaN or an infinity is not:
      // the sums over queries leave out the groups of 16 that see no key of this block, the sum over keys the groups that
      // no query of the tile sees.
      for (int j = 0; j < nq && ok; ++j) {
        const int s = j & 1, q0 = (t0 + j) * kT;
        const int qlo = max(0, first_q - q0) >> 4, qhi = min(kT - 1, last_q - q0) >> 4;
        const int key_lo = p.causal && p.window > 0 ? shift + q0 - p.window + 1 : 0;
        const int key_hi = p.causal ? min(p.lk - 1, shift + q0 + kT - 1) : p.lk - 1;
        const int klo = max(0, key_lo - k0) >> 4, khi = min(kT - 1, key_hi - k0) >> 4;
        ok = ptx::warp_wait(p_ready, j & 1, p.status, 36);
        if (!ok) break;
        ptx::tc_fence_after_sync();
        ptx::mma_groups<kT / 16>(qlo, qhi, [&](int k, bool start) {
          const uint64_t db = ptx::make_smem_desc(do_smem + k * 2048, kSlab, 1024);         // dO (N-major slabs)
          if (leader) ptx::mma_bf16_ts(tmem_dv, tmem_s + (k >> 2) * 64 + (k & 3) * 8, db, idesc_acc, (j > 0 || !start) ? 1u : 0u);
        });
        if (leader) ptx::mma_commit(do_empty);
        if (j + 1 < nq) ok = issue_s(j + 1);
        ok = ok && ptx::warp_wait(ds_ready, j & 1, p.status, 37);
        if (!ok) break;
        ptx::tc_fence_after_sync();
        ptx::mma_groups<kT / 16>(klo, khi, [&](int k, bool start) {
          const uint64_t da = ptx::make_smem_desc(ds_smem + k * 2048, kSlab, 1024);          // dS (M-major: queries)
          const uint64_t db = ptx::make_smem_desc(k_smem + k * 2048, kSlab, 1024);           // K (N-major slabs)
          if (leader) ptx::mma_bf16_ss(tmem_dp, da, db, idesc_dq, start ? 0u : 1u);
        });
        if (leader) ptx::mma_commit(dq_done);
        ptx::mma_groups<kT / 16>(qlo, qhi, [&](int k, bool start) {
          const uint64_t da = ptx::make_smem_desc(ds_smem + (k >> 2) * kSlab + (k & 3) * 32, 16, 1024);   // dS^T
          const uint64_t db = ptx::make_smem_desc(q_smem(s) + k * 2048, kSlab, 1024);        // Q (N-major slabs)
          if (leader) ptx::mma_bf16_ss(tmem_dk, da, db, idesc_acc, (j > 0 || !start) ? 1u : 0u);
        });
        if (leader) ptx::mma_commit(q_empty(s));
        if (j + 1 < nq) ok = ptx::warp_wait(dq_free, j & 1, p.status, 38) && issue_dp(j + 1);
      }
      if (ok && leader) ptx::mma_commit(acc_done);
    }
  } else if (warp < 8) {
    ptx::reg_inc<kComputeRegs>();
    // ================= P and dS: thread = (key row, half of the 128 query columns) =================
    const int half = warp >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int kp = k0 + r;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t col0 = lane_base + half * 64;
    uint8_t* drow = gen + C::kDS + half * kSlab + r * 128;
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    for (int j = 0; j < nq; ++j) {
      const int s = j & 1, q0 = (t0 + j) * kT;
      if (!ptx::mbar_wait(q_full(s), (j >> 1) & 1, p.status, 39) || !ptx::mbar_wait(s_done, j & 1, p.status, 40)) {
        ok = false;
        break;
      }
      ptx::tc_fence_after_sync();
      uint32_t pr[2][32];
      ptx::tmem_ld_32x32(tmem_s + col0, pr[0]);
      ptx::tmem_ld_32x32(tmem_s + col0 + 32, pr[1]);
      ptx::tmem_ld_wait();
      const float4* nl = reinterpret_cast<const float4*>(gen + C::kVec + s * 1024 + half * 256);
      const float4* nd = reinterpret_cast<const float4*>(gen + C::kVec + s * 1024 + 512 + half * 256);
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float4 l4 = nl[i >> 2];
        uint32_t* x = &pr[i >> 5][i & 31];
        const float2 a = __ffma2_rn(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), scale2, make_float2(l4.x, l4.y));
        const float2 b = __ffma2_rn(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), scale2, make_float2(l4.z, l4.w));
        x[0] = __float_as_uint(exp2f(a.x));
        x[1] = __float_as_uint(exp2f(a.y));
        x[2] = __float_as_uint(exp2f(b.x));
        x[3] = __float_as_uint(exp2f(b.y));
      }
      bool need_mask = k0 + kT > p.lk;
      if (p.causal) {
        need_mask = need_mask || (k0 + kT - 1 > shift + q0);
        if (p.window > 0) need_mask = need_mask || (k0 <= shift + q0 + kT - 1 - p.window);
      }
      if (need_mask) {
        // query columns that see this key: [lo, lo + span]; none when the key lies past the end of the sequence
        int lo = 0;
        uint32_t span = 1u << 30;
        if (p.causal) {
          lo = kp - shift - q0 - half * 64;
          if (p.window > 0) span = (uint32_t)(p.window - 1);
        }
        if (kp >= p.lk) { lo = 1 << 20; span = 0; }
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if ((uint32_t)(i - lo) > span) pr[i >> 5][i & 31] = 0u;
      }
      {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t* x = &pr[i >> 4][(2 * i) & 31];
          w[i] = ptx::pack_bf16x2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])));
        }
        ptx::tmem_st_32x32(tmem_s + col0, w);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      ptx::mbar_arrive(p_ready);
      if (!ptx::mbar_wait(dp_done, j & 1, p.status, 41)) { ok = false; break; }
      ptx::tc_fence_after_sync();
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t d[32];
        ptx::tmem_ld_32x32(tmem_dp + col0 + hc * 32, d);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint32_t w[4];
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float4 d4 = nd[hc * 8 + ch * 2 + hh];
            const uint32_t* x = &d[ch * 8 + hh * 4];
            const uint32_t* e = &pr[hc][ch * 8 + hh * 4];
            const float2 a = __fadd2_rn(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), make_float2(d4.x, d4.y));
            const float2 b = __fadd2_rn(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), make_float2(d4.z, d4.w));
            w[hh * 2] = ptx::pack_bf16x2(__fmul2_rn(a, make_float2(__uint_as_float(e[0]), __uint_as_float(e[1]))));
            w[hh * 2 + 1] = ptx::pack_bf16x2(__fmul2_rn(b, make_float2(__uint_as_float(e[2]), __uint_as_float(e[3]))));
          }
          const int chunk = hc * 4 + ch;
          *reinterpret_cast<uint4*>(drow + ((chunk ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      ptx::fence_proxy_async();          // make the generic-proxy writes of dS visible to the tensor core
      ptx::tc_fence_before_sync();
      ptx::mbar_arrive(ds_ready);
    }
    if (ok) ok = ptx::mbar_wait(acc_done, 0, p.status, 42);
    if (ok) {
      ptx::tc_fence_after_sync();
      // the TMEM loads are warp-collective: rows past the end of the sequence take part and skip the stores
      const bool live = kp < p.lk;
      const size_t off = (((size_t)batch * p.lk + (live ? kp : 0)) * p.heads + head) * HD;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        if ((c & 1) != half) continue;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          uint32_t raw[32];
          ptx::tmem_ld_32x32((which ? tmem_dv : tmem_dk) + lane_base + c * 32, raw);
          ptx::tmem_ld_wait();
          const float f = which ? 1.f : p.scale;
          __nv_bfloat16* dst = (which ? p.dv : p.dk) + off + c * 32;
          if (live) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint32_t w[4];
#pragma unroll
              for (int t = 0; t < 4; ++t)
                w[t] = pack_bf16(__uint_as_float(raw[i + 2 * t]) * f, __uint_as_float(raw[i + 2 * t + 1]) * f);
              *reinterpret_cast<uint4*>(dst + i) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
    }
  } else {
    // ================= dQ tile -> fp32 sums: thread = query row =================
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    for (int j = 0; j < nq; ++j) {
      if (!ptx::mbar_wait(dq_done, j & 1, p.status, 43)) break;
      ptx::tc_fence_after_sync();
      float* dst = p.dq_sum + ((bh * (p.lq_pad / kT) + t0 + j) * kT * HD + r * 4);
#pragma unroll
      for (int c0 = 0; c0 < HD / 32; c0 += 2) {
        constexpr int kChunks = HD / 32;
        uint32_t o[2][32];
        ptx::tmem_ld_32x32(tmem_dp + lane_base + c0 * 32, o[0]);
        if (c0 + 1 < kChunks) ptx::tmem_ld_32x32(tmem_dp + lane_base + c0 * 32 + 32, o[1]);
        ptx::tmem_ld_wait();
        if (c0 + 2 >= kChunks) {
          ptx::tc_fence_before_sync();
          ptx::mbar_arrive(dq_free);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (c0 + c >= kChunks) continue;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            red_add_v4(dst + (size_t)((c0 + c) * 8 + i / 4) * (kT * 4), o[c][i], o[c][i + 1], o[c][i + 2], o[c][i + 3]);
        }
      }
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 12) ptx::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------ dQ sums -> bf16
// One block = 64 rows of one (batch, head): the sums are read four columns at a time along the rows, turned in shared
// memory and written as whole head vectors.
template <int HD>
__global__ void __launch_bounds__(256) swa_bwd_dq_out_kernel(const float* __restrict__ sum, __nv_bfloat16* __restrict__ dq,
                                                             float scale, int lq, int lq_pad, int heads) {
  __shared__ float4 tile[64][HD / 4 + 1];
  const int blocks_q = lq_pad / 64;
  const int row0 = (blockIdx.x % blocks_q) * 64;
  const size_t bh = blockIdx.x / blocks_q;
  const float4* src = reinterpret_cast<const float4*>(sum) + (bh * (lq_pad / kT) + row0 / kT) * (kT * HD / 4) + row0 % kT;
  for (int i = threadIdx.x; i < 64 * (HD / 4); i += 256) tile[i & 63][i >> 6] = src[(size_t)(i >> 6) * kT + (i & 63)];
  __syncthreads();
  const size_t batch = bh / heads, head = bh % heads;
  for (int i = threadIdx.x; i < 64 * (HD / 8); i += 256) {
    const int r = i / (HD / 8), c = i % (HD / 8);
    if (row0 + r >= lq) continue;
    const float4 a = tile[r][2 * c], b = tile[r][2 * c + 1];
    const float f[8] = {a.x * scale, a.y * scale, a.z * scale, a.w * scale, b.x * scale, b.y * scale, b.z * scale, b.w * scale};
    Vec8<__nv_bfloat16>::store(dq + ((batch * lq + row0 + r) * heads + head) * HD + c * 8, f);
  }
}

// ------------------------------------------------------------------------------------ host
template <int HD>
static void launch_bwd(const at::Tensor& o, const at::Tensor& dout, const at::Tensor& lse, const CUtensorMap& tq,
                       const CUtensorMap& tdo, const CUtensorMap& tk, const CUtensorMap& tv, SwaBwdParams p,
                       float* nlse2, float* ndsum, __nv_bfloat16* dq, int b, cudaStream_t stream) {
  const int total = b * p.heads * p.lq_pad;
  swa_bwd_prep_kernel<HD><<<(total + 31) / 32, 256, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(o.data_ptr()), reinterpret_cast<const __nv_bfloat16*>(dout.data_ptr()),
      lse.data_ptr<float>(), nlse2, ndsum, p.lq, p.lq_pad, p.heads, total);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  auto kernel = swa_bwd_kernel<HD>;
  C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdCfg<HD>::kSmem));
  // Under torch.use_deterministic_algorithms a launch takes only key tiles whose bands share no query tile, every
  // kt_step-th one: it adds at most once to any sum of dQ, and the launches follow one another.  A band of 128 keys and a
  // window covers fewer than (window + 253) / 128 + 1 query tiles.  4 x 16 heads x 96, 2048 queries on 4096 keys,
  // window 2048: 968 us for the whole backward, against 528 with all key tiles in one launch (the two kernels that this one
  // replaced, which needed no such order, 785).
  const int tiles = (p.lk + kT - 1) / kT;
  p.kt_step = 1;
  if (at::globalContext().deterministicAlgorithms())
    p.kt_step = p.causal && p.window > 0 ? (int)std::min<long long>(tiles, ((long long)p.window + 253) / kT + 1) : tiles;
  for (p.kt_first = 0; p.kt_first < p.kt_step; ++p.kt_first) {
    const int blocks = (tiles - p.kt_first + p.kt_step - 1) / p.kt_step;
    kernel<<<dim3(blocks, p.heads, b), kThreads, BwdCfg<HD>::kSmem, stream>>>(tq, tdo, tk, tv, p);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
    count_launch();
  }
  swa_bwd_dq_out_kernel<HD><<<p.lq_pad / 64 * p.heads * b, 256, 0, stream>>>(p.dq_sum, dq, p.scale, p.lq, p.lq_pad,
                                                                                  p.heads);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

std::vector<at::Tensor> swa_bwd(at::Tensor dout, at::Tensor q, at::Tensor k, at::Tensor v, at::Tensor o, at::Tensor lse,
                                int64_t window, bool causal, double scale) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 &&
              v.scalar_type() == at::kBFloat16 && o.scalar_type() == at::kBFloat16 &&
              dout.scalar_type() == at::kBFloat16 && lse.scalar_type() == at::kFloat);
  TORCH_CHECK(q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && o.is_contiguous() &&
              dout.is_contiguous() && lse.is_contiguous());
  int b = q.size(0), lq = q.size(1), h = q.size(2), hd = q.size(3), lk = k.size(1);
  TORCH_CHECK(k.size(2) == h && k.size(3) == hd && v.sizes() == k.sizes() && lk >= lq && dout.sizes() == q.sizes() &&
              o.sizes() == q.sizes() && lse.numel() == (int64_t)b * h * lq);
  TORCH_CHECK(hd == 64 || hd == 96 || hd == 128, "swa_bwd: head dim must be 64, 96 or 128");
  auto dq = at::empty_like(q);
  auto dk = at::empty_like(k);
  auto dv = at::empty_like(v);
  const int lq_pad = (lq + 127) / 128 * 128;
  auto aux = at::empty({2, b, h, lq_pad}, q.options().dtype(at::kFloat));
  auto dq_sum = at::zeros({b, h, lq_pad, hd}, q.options().dtype(at::kFloat));
  float* nlse2 = aux.data_ptr<float>();
  float* ndsum = nlse2 + (size_t)b * h * lq_pad;
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  uint64_t row = (uint64_t)h * hd * 2;
  auto tq = make_tmap_3d_bf16(q.data_ptr(), (uint64_t)h * hd, lq, b, row, row * lq, 64, kT);
  auto tdo = make_tmap_3d_bf16(dout.data_ptr(), (uint64_t)h * hd, lq, b, row, row * lq, 64, kT);
  auto tk = make_tmap_3d_bf16(k.data_ptr(), (uint64_t)h * hd, lk, b, row, row * lk, 64, kT);
  auto tv = make_tmap_3d_bf16(v.data_ptr(), (uint64_t)h * hd, lk, b, row, row * lk, 64, kT);
  SwaBwdParams p{};
  p.lq = lq; p.lk = lk; p.heads = h; p.lq_pad = lq_pad;
  p.window = causal ? (int)window : 0;
  p.causal = causal ? 1 : 0;
  p.scale = (float)scale;
  p.scale_log2 = (float)(scale * 1.4426950408889634);
  p.nlse2 = nlse2; p.ndsum = ndsum;
  p.dq_sum = dq_sum.data_ptr<float>();
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk.data_ptr());
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv.data_ptr());
  p.status = gemm_status(q).data_ptr<int>();
  auto* dqp = reinterpret_cast<__nv_bfloat16*>(dq.data_ptr());
  if (hd == 64) launch_bwd<64>(o, dout, lse, tq, tdo, tk, tv, p, nlse2, ndsum, dqp, b, stream);
  else if (hd == 96) launch_bwd<96>(o, dout, lse, tq, tdo, tk, tv, p, nlse2, ndsum, dqp, b, stream);
  else launch_bwd<128>(o, dout, lse, tq, tdo, tk, tv, p, nlse2, ndsum, dqp, b, stream);
  count_launch(2);
  return {dq, dk, dv};
}

}  // namespace uttt
