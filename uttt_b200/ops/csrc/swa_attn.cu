// Sliding-window causal attention, forward, on tcgen05 tensor cores with TMEM accumulators.
//
//   q [b, lq, h, hd], k/v [b, lk, h, hd] (bf16); the queries are aligned to the last lq keys.
//   causal: key j visible to query i (absolute position p = lk - lq + i) iff j <= p and j > p - window.
//   non-causal (window ignored): every key visible (full attention inside one view).
//
// One CTA = one (batch, head) and one or two 128-query tiles.  It walks the 128-key tiles of the union of their bands:
//   warps 0-3, 4-7  : softmax of query tile 0 / 1, one thread per query row (= TMEM lane): the whole row of S_j is read
//                     into registers, P_j = 2^(S_j - ref) goes back to tensor memory as bf16 over S_j and is the A
//                     operand of the second product.  O is accumulated in TMEM relative to a per-row reference
//                     maximum that moves only when the running maximum exceeds it by 8 (log2 units); only then O is
//                     rescaled in TMEM.
//   warp 8 / lane 0 : TMA producer   K_j, V_j -> 128B-swizzled rings
//   warp 9          : MMA issuer     (an elected lane of the converged warp) per step and query tile:
//                                    O += P_{j-1} V_{j-1}, then S_j = Q K_j^T
// The two query tiles alternate: while the tensor core works for one, the other's softmax warps run, and each K/V tile
// is fetched once for 256 queries.  Bound by the chain S -> softmax -> P -> MMA of a tile (tensor pipe a third busy,
// exponential unit under half); a step of 128 keys pays its hand-overs once where a step of 64 paid them twice.
// Measured against two 128-query CTAs per SM with steps of 64 keys and two threads to a row: 275 -> 152 us at 4 x 16
// heads x 96, 2048 queries on 4096 keys, window 2048; 109 -> 72 us at 12 x 12 heads x 64, 1024 tokens unmasked.  Steps of
// 64 keys with two S buffers per query tile in this layout: 180 and 83 us.
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

struct SwaParams {
  int lq, lk, heads, hd;
  int window;       // 0 = unlimited
  int causal;
  int tiles;        // 128-query tiles per CTA: 1 or 2
  int flip;         // the softmax scale is negative: S is negated and scale_log2 holds |scale| * log2(e)
  float scale_log2; // |softmax scale| * log2(e), > 0
  __nv_bfloat16* out;
  float* lse;       // [b, h, lq], natural log of the row sums of exp(scale * s)
  int* status;
};

constexpr int kQ = 128;   // queries per tile
constexpr int kKV = 128;  // keys per tile
constexpr int kSlabBytes = 128 * 128;        // 128 rows x 64 bf16, one 128-byte swizzle row each
// Three warpgroups at 168 registers each; the softmax ones take 208 (a row of S lives in registers), the third gives
// its share up: 2 x 208 + 80 <= 3 x 168.
constexpr int kThreads = 384;
constexpr int kSoftmaxRegs = 208, kOtherRegs = 80;
static_assert(2 * kSoftmaxRegs + kOtherRegs <= 3 * 168, "more registers than the block is launched with");
constexpr float kRescaleThreshold = 8.f;     // log2 units: P stays below 2^8 between rescales

template <int HD>
struct SwaCfg {
  static constexpr int KB = (HD + 63) / 64;                // 64-wide slabs along the head dimension
  static constexpr int kTile = KB * kSlabBytes;
  static constexpr int kStages = HD == 64 ? 4 : 2;         // K and V ring depth
  static constexpr int kBars = 2 * kTile + 2 * kStages * kTile;
  static constexpr int kSmem = kBars + 256 + 1024;
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 1) swa_fwd_kernel(const __grid_constant__ CUtensorMap tq,
                                                         const __grid_constant__ CUtensorMap tk,
                                                         const __grid_constant__ CUtensorMap tv, SwaParams p) {
  using C = SwaCfg<HD>;
  constexpr int KB = C::KB, ST = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - ptx::smem_u32(smem_raw));
  auto q_smem = [&](int s) { return base + s * C::kTile; };
  auto k_smem = [&](int st) { return base + (2 + st) * C::kTile; };
  auto v_smem = [&](int st) { return base + (2 + ST + st) * C::kTile; };
  const uint32_t bars = base + C::kBars;
  auto q_full = [&](int s) { return bars + 8 * s; };
  auto s_done = [&](int s) { return bars + 16 + 8 * s; };
  auto p_ready = [&](int s) { return bars + 32 + 8 * s; };
  auto o_done = [&](int s) { return bars + 48 + 8 * s; };
  auto k_full = [&](int st) { return bars + 64 + 8 * st; };
  auto v_full = [&](int st) { return bars + 96 + 8 * st; };
  auto k_empty = [&](int st) { return bars + 128 + 8 * st; };
  auto v_empty = [&](int st) { return bars + 160 + 8 * st; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + C::kBars + 192);

  const int warp = ptx::warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  // the last query tiles see the most keys when the history is short: they are issued first
  const int blocks_q = (p.lq + kQ * p.tiles - 1) / (kQ * p.tiles);
  const int head = blockIdx.x % p.heads, batch = blockIdx.y;
  const int q00 = (blocks_q - 1 - blockIdx.x / p.heads) * kQ * p.tiles;
  const int shift = p.lk - p.lq;          // absolute position of query 0
  // key tile range of each query tile
  int lo_t[2] = {0, 0}, hi_t[2] = {0, 0};
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int q0 = q00 + s * kQ;
    if (s < p.tiles && q0 < p.lq) {
      int first_key = 0, last_key = p.lk - 1;
      if (p.causal) {
        last_key = min(p.lk - 1, shift + q0 + kQ - 1);
        if (p.window > 0) first_key = max(0, shift + q0 - p.window + 1);
      }
      lo_t[s] = first_key / kKV;
      hi_t[s] = last_key / kKV + 1;
    }
  }
  const bool two = hi_t[1] > lo_t[1];
  const int t0 = lo_t[0];                                   // the first query tile's band starts first
  const int nt = (two ? hi_t[1] : hi_t[0]) - t0;            // and the second one's ends last

  {
    __shared__ int prior_failure;
    if (threadIdx.x == 0) prior_failure = (p.status != nullptr) ? *(volatile int*)p.status : 0;
    __syncthreads();
    if (prior_failure != 0) return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(q_full(s), 1);
      ptx::mbar_init(s_done(s), 1);
      ptx::mbar_init(p_ready(s), 128);
      ptx::mbar_init(o_done(s), 1);
    }
    for (int st = 0; st < ST; ++st) {
      ptx::mbar_init(k_full(st), 1);
      ptx::mbar_init(v_full(st), 1);
      ptx::mbar_init(k_empty(st), 1);
      ptx::mbar_init(v_empty(st), 1);
    }
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&tq);
    ptx::tma_prefetch_desc(&tk);
    ptx::tma_prefetch_desc(&tv);
  }
  if (warp == 8) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = ptx::warp_uniform(*tmem_slot);
  auto tmem_s = [&](int s) { return tmem + s * 128; };           // S_j (fp32), overwritten by P_j (bf16, 64 columns)
  auto tmem_o = [&](int s) { return tmem + 256 + s * 128; };

  constexpr uint32_t idesc_s = ptx::make_instr_desc(kQ, kKV, 0, 0);
  constexpr uint32_t idesc_o = ptx::make_instr_desc(kQ, HD, 0, 1);
  bool ok = true;

  // each role's code stays inside the branch that sets its register share
  if (warp >= 8) {
    ptx::reg_dec<kOtherRegs>();
    if (warp == 8 && lane == 0) {
      // ================= producer =================
      auto load = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int row) {
        ptx::mbar_expect_tx(bar, C::kTile);
        for (int kb = 0; kb < KB; ++kb)
          ptx::tma_load_3d(dst + kb * kSlabBytes, map, bar, head * HD + kb * 64, row, batch);
      };
      load(q_smem(0), &tq, q_full(0), q00);
      for (int j = 0; j < nt && ok; ++j) {
        const int st = j % ST;
        if (j >= ST) ok = ptx::mbar_wait(k_empty(st), (j / ST - 1) & 1, p.status, 11);
        if (!ok) break;
        load(k_smem(st), &tk, k_full(st), (t0 + j) * kKV);
        if (j == 0 && two) load(q_smem(1), &tq, q_full(1), q00 + kQ);
        if (j >= ST) ok = ptx::mbar_wait(v_empty(st), (j / ST - 1) & 1, p.status, 12);
        if (!ok) break;
        load(v_smem(st), &tv, v_full(st), (t0 + j) * kKV);
      }
    } else if (warp == 9) {
      // ================= MMA issuer =================
      // S_j overwrites P_{j-1}: the product that reads P_{j-1} was issued before it by this thread, and the tensor core
      // runs them in order.  For the same reason "S_j is complete" says that O has received P_{j-1} V_{j-1}.
      const bool leader = ptx::elect_one();
      // P is zero where it is masked, but zero times a NaN or an infinity in V is not: the product leaves out the groups
      // of 16 keys that no query of the tile sees.
      int key_lo[2], key_hi[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q0 = q00 + s * kQ;
        key_lo[s] = p.causal && p.window > 0 ? max(0, shift + q0 - p.window + 1) : 0;
        key_hi[s] = p.causal ? min(p.lk - 1, shift + q0 + kQ - 1) : p.lk - 1;
      }
      for (int j = 0; j <= nt && ok; ++j) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int first = lo_t[s] - t0, last = hi_t[s] - t0 - 1;       // this query tile's steps
          if (s == 1 && !two) continue;
          if (j - 1 >= first && j - 1 <= last) {
            const int st = (j - 1) % ST;
            ok = ptx::warp_wait(p_ready(s), (j - 1 - first) & 1, p.status, 13) &&
                 ptx::warp_wait(v_full(st), ((j - 1) / ST) & 1, p.status, 14);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const int key0 = (t0 + j - 1) * kKV;
            const int klo = max(0, key_lo[s] - key0) >> 4, khi = min(kKV - 1, key_hi[s] - key0) >> 4;
            ptx::mma_groups<kKV / 16>(klo, khi, [&](int k, bool start) {
              const uint64_t db = ptx::make_smem_desc(v_smem(st) + k * 2048, kSlabBytes, 1024);   // V_j (N-major slabs)
              if (leader) ptx::mma_bf16_ts(tmem_o(s), tmem_s(s) + k * 8, db, idesc_o, (j - 1 > first || !start) ? 1u : 0u);
            });
            if (leader && j - 1 == last) ptx::mma_commit(o_done(s));
          }
          if (j >= first && j <= last) {
            const int st = j % ST;
            if (j == first) ok = ptx::warp_wait(q_full(s), 0, p.status, 15);
            ok = ok && ptx::warp_wait(k_full(st), (j / ST) & 1, p.status, 16);
            if (!ok) break;
            ptx::tc_fence_after_sync();
#pragma unroll
            for (int k = 0; k < HD / 16; ++k) {
              const uint64_t da = ptx::make_smem_desc(q_smem(s) + (k >> 2) * kSlabBytes + (k & 3) * 32, 16, 1024);
              const uint64_t db = ptx::make_smem_desc(k_smem(st) + (k >> 2) * kSlabBytes + (k & 3) * 32, 16, 1024);
              if (leader) ptx::mma_bf16_ss(tmem_s(s), da, db, idesc_s, k > 0 ? 1u : 0u);
            }
            if (leader) ptx::mma_commit(s_done(s));
          }
        }
        if (!ok) break;
        if (leader && j < nt) ptx::mma_commit(k_empty(j % ST));
        if (leader && j > 0) ptx::mma_commit(v_empty((j - 1) % ST));
      }
    }
  } else {
    ptx::reg_inc<kSoftmaxRegs>();
    // ================= softmax (warps 0-7): thread = query row =================
    const int s = warp >> 2;
    const int quarter = warp & 3;
    const int q0 = q00 + s * kQ;
    const int r = quarter * 32 + lane;            // query row inside the tile == TMEM lane
    const int qpos = shift + q0 + r;              // absolute position
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int first = s ? lo_t[1] : lo_t[0], n = s ? hi_t[1] - lo_t[1] : hi_t[0] - lo_t[0];
    float m_ref = -INFINITY, l_run = 0.f;

    for (int j = 0; j < n; ++j) {
      if (!ptx::mbar_wait(s_done(s), j & 1, p.status, 17)) { ok = false; break; }
      ptx::tc_fence_after_sync();
      uint32_t raw[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) ptx::tmem_ld_32x32(tmem_s(s) + lane_base + c * 32, raw[c]);
      ptx::tmem_ld_wait();
      if (p.flip) {
#pragma unroll
        for (int i = 0; i < 128; ++i) raw[i >> 5][i & 31] ^= 0x80000000u;
      }
      const int key0 = (first + j) * kKV;
      bool need_mask = (key0 + kKV > p.lk);
      if (p.causal) {
        need_mask = need_mask || (key0 + kKV - 1 > shift + q0);
        if (p.window > 0) need_mask = need_mask || (key0 <= shift + q0 + kQ - 1 - p.window);
      }
      if (need_mask) {
        // visible columns of this row: [lo, lo + span]
        int hi = p.lk - 1 - key0, lo = 0;
        if (p.causal) {
          hi = min(hi, qpos - key0);
          if (p.window > 0) lo = max(0, qpos - key0 - p.window + 1);
        }
        if (hi < lo) { lo = 1 << 20; hi = lo; }
        const uint32_t span = (uint32_t)(hi - lo);
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if ((uint32_t)(i - lo) > span) raw[i >> 5][i & 31] = 0xff800000u;
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i) {
#pragma unroll
        for (int c = 0; c < 4; ++c) m4[c] = fmaxf(m4[c], __uint_as_float(raw[c][i]));
      }
      const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;
      const bool move_ref = mx > m_ref + kRescaleThreshold;     // also true for the first visible key (m_ref = -inf)
      const float new_ref = move_ref ? mx : m_ref;
      if (j > 0 && __any_sync(0xffffffffu, move_ref)) {
        const float factor = move_ref ? exp2f(m_ref - new_ref) : 1.f;    // m_ref = -inf -> 0
        l_run *= factor;
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          ptx::tmem_ld_32x32(tmem_o(s) + lane_base + c * 32, o);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
          ptx::tmem_st_32x32(tmem_o(s) + lane_base + c * 32, o);
        }
      }
      m_ref = new_ref;
      const float neg = (new_ref == -INFINITY) ? 0.f : -new_ref;
      const float2 neg2 = make_float2(neg, neg), scale2 = make_float2(p.scale_log2, p.scale_log2);
      float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int col = c * 64 + 2 * i;
          float2 x = make_float2(__uint_as_float(raw[col >> 5][col & 31]), __uint_as_float(raw[col >> 5][(col & 31) + 1]));
          x = __ffma2_rn(x, scale2, neg2);
          x.x = exp2f(x.x);
          x.y = exp2f(x.y);
          rs[i & 1] = __fadd2_rn(rs[i & 1], x);
          w[i] = ptx::pack_bf16x2(x);
        }
        ptx::tmem_st_32x32(tmem_s(s) + lane_base + c * 32, w);
      }
      l_run += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      ptx::mbar_arrive(p_ready(s));
    }

    if (ok && n > 0) ok = ptx::mbar_wait(o_done(s), 0, p.status, 18);
    if (ok && n > 0) {
      ptx::tc_fence_after_sync();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const bool live = q0 + r < p.lq;
      __nv_bfloat16* orow = p.out + (((size_t)batch * p.lq + (live ? q0 + r : 0)) * p.heads + head) * HD;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        ptx::tmem_ld_32x32(tmem_o(s) + lane_base + c * 32, o);
        ptx::tmem_ld_wait();
        if (live) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float f[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) f[t] = __uint_as_float(o[i + t]) * inv;
            Vec8<__nv_bfloat16>::store(orow + c * 32 + i, f);
          }
        }
      }
      if (live)
        p.lse[((size_t)batch * p.heads + head) * p.lq + q0 + r] =
            l_run > 0.f ? (m_ref * 0.6931471805599453f + __logf(l_run)) : -INFINITY;
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) ptx::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------ host
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    auto err = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q);
    TORCH_CHECK(err == cudaSuccess && q == cudaDriverEntryPointSuccess && ptr != nullptr,
                "cuTensorMapEncodeTiled is not available from the driver");
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}

// bf16 tensor [d2, d1, d0] with d0 contiguous; box = [1, box1, box0]; 128-byte swizzle; out-of-range reads give 0.
CUtensorMap make_tmap_3d_bf16(const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1_bytes,
                              uint64_t stride2_bytes, uint32_t box0, uint32_t box1) {
  CUtensorMap m;
  TORCH_CHECK(ensure_context_current(), "no CUDA context on this thread");
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {box0, box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  TORCH_CHECK(((uintptr_t)base & 15) == 0 && stride1_bytes % 16 == 0 && stride2_bytes % 16 == 0);
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (3d) failed with code ", (int)r);
  return m;
}

at::Tensor gemm_status(at::Tensor like);

std::vector<at::Tensor> swa_fwd(at::Tensor q, at::Tensor k, at::Tensor v, int64_t window, bool causal, double scale) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 &&
              v.scalar_type() == at::kBFloat16 && q.is_contiguous() && k.is_contiguous() && v.is_contiguous());
  int b = q.size(0), lq = q.size(1), h = q.size(2), hd = q.size(3), lk = k.size(1);
  TORCH_CHECK(k.size(2) == h && k.size(3) == hd && v.sizes() == k.sizes() && lk >= lq);
  TORCH_CHECK(hd == 64 || hd == 96 || hd == 128, "swa_fwd: head dim must be 64, 96 or 128");
  auto out = at::empty_like(q);
  auto lse = at::empty({b, h, lq}, q.options().dtype(at::kFloat));
  uint64_t row = (uint64_t)h * hd * 2;
  auto tq = make_tmap_3d_bf16(q.data_ptr(), (uint64_t)h * hd, lq, b, row, row * lq, 64, kQ);
  auto tk = make_tmap_3d_bf16(k.data_ptr(), (uint64_t)h * hd, lk, b, row, row * lk, 64, kKV);
  auto tv = make_tmap_3d_bf16(v.data_ptr(), (uint64_t)h * hd, lk, b, row, row * lk, 64, kKV);
  SwaParams p{};
  p.lq = lq; p.lk = lk; p.heads = h; p.hd = hd;
  p.window = causal ? (int)window : 0;
  p.causal = causal ? 1 : 0;
  // the kernel takes row maxima before it scales, which needs a positive factor: the sign goes to S, and a scale of
  // zero becomes one that no product of finite values notices (0 * -inf of a masked key would be NaN)
  const float scale_log2 = (float)(scale * 1.4426950408889634);
  p.flip = scale_log2 < 0.f ? 1 : 0;
  p.scale_log2 = scale_log2 == 0.f ? 1e-37f : fabsf(scale_log2);
  p.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  p.lse = lse.data_ptr<float>();
  p.status = gemm_status(q).data_ptr<int>();
  // One 128-query tile per CTA as long as every tile has an SM of its own; beyond that two, which cost one and a half
  // times a single one and fetch K and V once.
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  p.tiles = (int64_t)((lq + kQ - 1) / kQ) * h * b <= sms ? 1 : 2;
  dim3 grid((lq + kQ * p.tiles - 1) / (kQ * p.tiles) * h, b);
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  auto launch = [&](auto kernel, int smem) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<grid, kThreads, smem, stream>>>(tq, tk, tv, p);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
  };
  if (hd == 64) launch(swa_fwd_kernel<64>, SwaCfg<64>::kSmem);
  else if (hd == 96) launch(swa_fwd_kernel<96>, SwaCfg<96>::kSmem);
  else launch(swa_fwd_kernel<128>, SwaCfg<128>::kSmem);
  count_launch();
  return {out, lse};
}

}  // namespace uttt
