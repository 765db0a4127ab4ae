// tcgen05 backward kernels of attention() (sm_100a): dQ, dK, dV from q, k, v, out, dout and the
// saved log-normaliser L.
//
// Same split as the reference (flash.py:172-261): a pre-pass (delta_i = sum_d out_id dout_id,
// flash.py:532-577), a key-major kernel for dK and dV (flash.py:581-754) and a query-major kernel
// for dQ (flash.py:758-918).  Both kernels are one template, tc_bwd_kernel<T, D, KEY_MAJOR>:
//
//   the CTA owns 128 rows of two *stationary* tiles X, Y and streams tile pairs (A_u, B_u):
//                       X   Y      A_u         B_u           accumulators
//     key-major         K   V      Q tile u    dout tile u   dV += P^T.dout,  dK += dS^T.Q
//     query-major       Q   dout   K tile u    V tile u      dQ += dS.K
//   per streamed pair:  S' = X.A^T and dP' = Y.B^T (fp32, TMEM; rows = the owned index), then
//   P' = exp(S'*scale - L), dS' = P' * (dP' - delta) in registers, written back to TMEM as 16-bit
//   operands over S' and dP', then the accumulating MMAs (A operand from TMEM).
//
// The tensor pipe is kept busy by the order of a step's MMAs, each group of 128 x 128 x D:
//   key-major     dV += P_u^T.dout_u | S'_u+1 | dK += dS_u^T.Q_u | dP'_u+1     (S' and P share columns, dP' and dS too)
//   query-major   S'_u+1 | dP'_u+1 | dQ += dS_u.K_u                            (two dP' buffers; S' is free once read)
// so that P is computed while dK and dP' run, and dS while dV and the next S' do.  S' and dP' are whole 128-column MMAs:
// with 64 columns an MMA reads 6 KB of shared memory per 32 cycles (51 cycles measured), with 128 8 KB per 64 (65
// measured).  One thread issues them: the pipe's queue holds about six, and a whole warp that elects a lane for each
// group spends another 100 cycles between groups (4 340 against 3 390 cycles a step, key-major D128, all else alike).
// The 128 streamed rows are shared out to two consumer warpgroups, 64 rows each.
// Warp roles (12 warps): warp 0 TMA producer (X, Y once, then rings of A and B tiles), warp 1 TMEM allocation and
// the MMA-issuing thread, warp 2 (key-major) the L / delta vectors of the streamed query tiles, warps 4-7 / 8-11
// consumers of half 0 / 1 (thread = owned row = TMEM lane).
// Modes.  kPlain rounds dS to the 16-bit type for its MMAs.  kFine keeps it as the sum of two 16-bit values
// (dS = hi + lo, one more MMA per accumulator and K-step; 16 significant bits in bf16, 22 in fp16) and adds the G
// heads' dK / dV from fp32 partials: problems that the CUDA-core kernels, which hold dS in fp32, would otherwise take
// (head dims 16 and 32) keep their precision this way.  In fp16 the 22 bits hold between 2^-3 and 2^16 only, so dS is
// moved there by a power of two per head, from the largest |dout|, |v| and |delta| that the pre-pass meets
// (GradScale), and moved back in the epilogue: exact, and gradients of any size come out as from fp32 dS.
// kDrop is kFine with the dropout mask, which the pre-pass draws (draw_mask).  In fine modes hi and lo of 16 streamed
// rows, the K-step of the accumulating MMAs, take the 16 columns that their dP' leaves.  fp16 B4 H16 S1024 D64 causal,
// p = 0.1, forward and backward: 194 us, 3 717 us with the CUDA-core kernels; errors of the gradients against fp64 as
// there (2.32e-4, 2.28e-4, 2.92e-4 for dq, dk, dv, fp16; dout of 1e-4, where the results are fp16 subnormals: 1.6e-3,
// 6.6e-3 with an unmoved dS).
// Deterministic: every output element is written once, by one CTA, in a fixed order; with GQA the
// key-major kernel writes per-query-head dK / dV and a second kernel adds the G heads in order.
// Out-of-range query rows need no predicates without dropout: TMA zero-fills the loads (with L = delta = 0 their P
// is 1 and their dS is 0, and the zero Q / dout row contributes nothing); stores are clipped.  Every mbarrier wait is bounded.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "faws_internal.cuh"
#include "faws_tc_host.cuh"
#include "faws_tc_ptx.cuh"

namespace faws {
namespace {
using namespace ptx;

constexpr int BT = 128;        // tile edge (owned rows and streamed rows)
constexpr int HALF = 64;       // streamed rows per consumer warpgroup
constexpr int NTHREADS = 384;
constexpr int TMEM_COLS = 512;
constexpr int REGS_LAUNCH = 168;
constexpr int REGS_AUX = 88;
constexpr int REGS_CONSUMER = ((REGS_LAUNCH * NTHREADS - 128 * REGS_AUX) / 256) & ~7;
static_assert(128 * REGS_AUX + 256 * REGS_CONSUMER <= REGS_LAUNCH * NTHREADS, "setmaxnreg would block");
constexpr float kLog2e = 1.4426950408889634f;

enum BwMode : int { kPlain = 0, kFine = 1, kDrop = 2 };

template <int D, bool KM>
struct BwSmem {
  static constexpr int kTile = 128 * D * 2;
  static constexpr int kSub = 128 * 128;  // one 64-element-wide sub-tile: 128 rows x 128 B
  // A tiles are held from S' to the last accumulating MMA of their step, B tiles for a shorter time
  static constexpr int kStagesA = D == 128 ? 3 : 4, kStagesB = D == 128 ? 2 : 4;
  // TMEM: S' buffers, dP' buffers (128 fp32 columns each), then the accumulators
  static constexpr int kSBufs = KM && D == 64 ? 2 : 1, kDpBufs = KM ? 1 : 2;
  static_assert((kSBufs + kDpBufs) * 128 + (KM ? 2 : 1) * D <= TMEM_COLS, "TMEM");
  static constexpr int x_off = 0;
  static constexpr int y_off = kTile;
  static constexpr int a_off = 2 * kTile;
  static constexpr int b_off = a_off + kStagesA * kTile;
  static constexpr int vec_off = b_off + kStagesB * kTile;  // 2 x (128 -L*log2e, 128 -delta) floats
  static constexpr int bar_off = vec_off + (KM ? 2 * 1024 : 0);
  static constexpr int total = bar_off + 384;
};

struct BwBars {
  uint64_t x_full, y_full;
  uint64_t a_full[4], a_empty[4], b_full[4], b_empty[4];
  uint64_t s_full[2], dp_full[2];  // per buffer: written by the tensor pipe
  uint64_t s_free;                 // query-major: S' is in the consumers' registers
  uint64_t p_ready[2][2];          // key-major, per S' buffer: P' of the first, last 32 rows of each warpgroup written
  uint64_t ds_ready[2];            // per dP' buffer: dS' written
  uint64_t vec_full[2], vec_empty[2];
  uint64_t acc_done;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(BwBars) <= 384, "room for the barriers");

struct BwMaps {
  CUtensorMap x, y, a, b;  // loads, 128-row boxes
  CUtensorMap o0, o1;      // stores, 32-row boxes: key-major dV, dK; query-major dQ (o1 unused)
};

struct BwTcParams {
  int Hq, G, M, N, p_seq, causal, Mpad;
  float sm_scale;
  const float* negl2;  // (B,Hq,Mpad): -L_i * log2(e), 0 for padded rows and rows without a visible key
  const float* neg_delta;  // (B,Hq,Mpad): -sum_d out_id * dout_id, 0 for padded rows
  float* part0;        // fine modes with grouped queries: fp32 (B,Hq,N,D) per-head dV and dK instead of the
  float* part1;        // store maps; null otherwise
  int D;               // the head dim (the instance's D is 64 for 16 and 32)
  DropoutParams drop;
  float keep_scale;    // 1 / (1 - p)
  const float2* g_stat;  // kScaledDs: (B,Hq,g_blocks) bounds of |dout_i|^2 and |delta_i| over a pre-pass block's rows,
  const float* v_stat;   // (B,Hk,v_blocks) of |v_j|^2
  int g_blocks, v_blocks;
  const uint32_t* mask;  // dropout: the mask as the pre-pass has drawn it (see draw_mask), or null
  int bh0;               // dropout: the launch's first (batch, head)
};

// The dropout mask (mask_word) in scratch, where the forward pass kept none.  Both kernels need it, and a kernel with nothing else to
// do draws it at twice the rate of the two consumer warps that a scheduler of the main kernels has: fp16 B4 H16 S1024 D64
// causal, p = 0.1, forward and backward: 247 us, 282 with the mask drawn in both.  One bit per entry grows with M * N:
// beyond kMaskBytes the heads take turns, pre-pass and both kernels for as many at a time as fit, or as keep the SMs
// busy (kMaskCtas) if those are more: backward passes of fp16 B2 H32 S8192 D64 causal 8.96 -> 6.5 ms against drawing in
// both, bf16 B8 Hq32 Hk8 S4096 D128 causal 10.2 -> 8.3 (two shares each).  Heads whose mask is above kMaskBytesMost draw
// in both kernels, as calls with scratch that has no room for a mask do.
constexpr size_t kMaskBytes = size_t(256) << 20, kMaskBytesMost = size_t(1) << 30;
constexpr int kMaskCtas = 1024;  // seven waves
// 32 x 32 bits across a warp: on entry bit k of lane l is A[l][k], on exit it is A[k][l].
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y & m) << j);
  }
  return x;
}

// Modes that move dS by a power of two before it is split: fp16 ones (bf16 has the range of fp32).
template <typename T, int MODE>
constexpr bool kScaledDs = MODE != kPlain && std::is_same<T, __half>::value;

template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<__half2*>(&w));
}
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
}

// The power of two for a head's dS, and its inverse.  |dS_ij| = P |keep dP_ij / (1 - p) - delta_i| is at most
// |dout_i| |v_j| / (1 - p) + |delta_i| (Cauchy-Schwarz, P <= 1); that bound goes to [2^13, 2^14), a quarter of fp16's
// range.  A bound of zero, infinity or NaN leaves dS as it is: infinities of the inputs reach the gradients.
struct GradScale {
  float mul, inv;
};
// largest of the warp's values, none of them negative (their bits order as they do)
__device__ __forceinline__ float warp_max(float x) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x)));
}
__device__ __forceinline__ GradScale grad_scale(const BwTcParams& p, int b, int h, int hk, int lane) {
  const float2* gs = p.g_stat + ((int64_t)b * p.Hq + h) * p.g_blocks;
  const float* vs = p.v_stat + ((int64_t)b * (p.Hq / p.G) + hk) * p.v_blocks;
  float g2 = 0.f, dl = 0.f, v2 = 0.f;
  for (int x = lane; x < p.g_blocks; x += 32) {
    const float2 s = gs[x];
    g2 = fmaxf(g2, s.x);
    dl = fmaxf(dl, s.y);
  }
  for (int x = lane; x < p.v_blocks; x += 32) v2 = fmaxf(v2, vs[x]);
  const float bound = fmaf(p.keep_scale * sqrtf(warp_max(g2)), sqrtf(warp_max(v2)), warp_max(dl));
  int k = 0;
  if (bound > 0.f && bound < __int_as_float(0x7f800000))
    k = max(-100, min(100, 13 - ((__float_as_int(bound) >> 23) - 127)));
  return {__int_as_float((127 + k) << 23), __int_as_float((127 - k) << 23)};
}

template <typename T, int D, bool KM, int MODE>
__global__ void __launch_bounds__(NTHREADS, 1)
tc_bwd_kernel(const __grid_constant__ BwMaps maps, const BwTcParams p, int* __restrict__ status) {
  using L = BwSmem<D, KM>;
  constexpr int NA = L::kStagesA, NB = L::kStagesB;
  constexpr int NSB = L::kSBufs, NDB = L::kDpBufs;
  constexpr uint32_t COL_DP = NSB * 128, COL_ACC = (NSB + NDB) * 128;
  extern __shared__ __align__(1024) unsigned char smem[];
  BwBars* bars = reinterpret_cast<BwBars*>(smem + L::bar_off);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (smem_u32(smem) & 1023u) {  // 128-byte swizzle atoms are 1 KB; the full shared memory leaves no slack to align by
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 1);
    return;
  }

  // Heaviest work first in launch order: key-major, the first key tiles see the most queries when
  // causal; query-major, the last query tiles see the most keys.
  const int own_tiles = (int)gridDim.z;
  const int own_tile = KM ? (int)blockIdx.z : (p.causal ? own_tiles - 1 - (int)blockIdx.z : (int)blockIdx.z);
  int h = blockIdx.x, b = blockIdx.y;
  if constexpr (MODE == kDrop) {  // the heads of a launch are consecutive, of several batches maybe
    const int bh = p.bh0 + b * (int)gridDim.x + h;
    b = bh / p.Hq;
    h = bh - b * p.Hq;
  }
  const int hk = h / p.G;
  const int own0 = own_tile * BT;  // first owned row: key n0 (key-major) or query i0 (query-major)

  // streamed tiles [u0, u0 + nu)
  int u0 = 0, nu;
  if (KM) {
    if (p.causal) u0 = max(0, own0 - p.p_seq) / BT;  // first query tile with a row that sees key own0
    nu = max(0, (p.M + BT - 1) / BT - u0);
  } else {
    int hi = p.N;
    if (p.causal) hi = max(0, min(p.N, p.p_seq + min(own0 + BT, p.M)));
    nu = (hi + BT - 1) / BT;
  }

  // Launch chain: pre-pass, query-major, key-major, group sum, each allowed to begin while the one before it drains.
  // Only the key-major kernel's partials and the pre-pass's arrays pass between them: the query-major kernel waits
  // for the pre-pass before it lets the key-major one begin, which therefore finds the arrays written and waits
  // for the query-major kernel only before it exits (so that its own completion stands for all of the chain).
  if (!KM) {
    griddep_wait();
    griddep_launch_dependents();
  }
  if (threadIdx.x == 0) {
    mbar_init(&bars->x_full, 1);
    mbar_init(&bars->y_full, 1);
    for (int s = 0; s < NA; ++s) {
      mbar_init(&bars->a_full[s], 1);
      mbar_init(&bars->a_empty[s], 1);
    }
    for (int s = 0; s < NB; ++s) {
      mbar_init(&bars->b_full[s], 1);
      mbar_init(&bars->b_empty[s], 1);
    }
    for (int w = 0; w < 2; ++w) {
      mbar_init(&bars->s_full[w], 1);
      mbar_init(&bars->dp_full[w], 1);
      mbar_init(&bars->vec_full[w], 1);
      mbar_init(&bars->vec_empty[w], 8);
      for (int c = 0; c < 2; ++c) mbar_init(&bars->p_ready[w][c], 256);
      mbar_init(&bars->ds_ready[w], 256);
    }
    mbar_init(&bars->s_free, 256);
    mbar_init(&bars->acc_done, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&maps.x);
    prefetch_tmap(&maps.y);
    prefetch_tmap(&maps.a);
    prefetch_tmap(&maps.b);
    prefetch_tmap(&maps.o0);
    if (KM) prefetch_tmap(&maps.o1);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  const int64_t vec_row = ((int64_t)b * p.Hq + h) * p.Mpad;  // this head's row of the padded L / delta arrays

  if (warp < 4) {
    reg_dealloc<REGS_AUX>();
    if (warp == 0 && lane == 0 && nu > 0) {
      // ---------------------------------------------------------- TMA producer
      const int x_head = KM ? hk : h, a_head = KM ? h : hk;
      auto load_tile = [&](int at, const CUtensorMap* m, uint64_t* bar, int row0, int head) {
        mbar_arrive_expect_tx(bar, L::kTile);
        for (int c = 0; c < D / 64; ++c) tma_load_4d(smem + at + c * L::kSub, m, bar, c * 64, row0, head, b);
      };
      load_tile(L::x_off, &maps.x, &bars->x_full, own0, x_head);
      for (int u = 0; u < nu; ++u) {
        const int row0 = (u0 + u) * BT, sa = u % NA, sb = u % NB;
        if (u >= NA && !mbar_wait(&bars->a_empty[sa], (u / NA - 1) & 1, abort_flag)) break;
        load_tile(L::a_off + sa * L::kTile, &maps.a, &bars->a_full[sa], row0, a_head);
        if (u == 0) load_tile(L::y_off, &maps.y, &bars->y_full, own0, x_head);
        if (u >= NB && !mbar_wait(&bars->b_empty[sb], (u / NB - 1) & 1, abort_flag)) break;
        load_tile(L::b_off + sb * L::kTile, &maps.b, &bars->b_full[sb], row0, a_head);
      }
    } else if (KM && warp == 2 && lane == 0) {
      // ---------------------------------------------------------- L and delta of the streamed query tiles
      for (int u = 0; u < nu; ++u) {
        const int s = u & 1;
        if (u >= 2 && !mbar_wait(&bars->vec_empty[s], (u / 2 - 1) & 1, abort_flag)) break;
        const int64_t at = vec_row + (u0 + u) * BT;
        mbar_arrive_expect_tx(&bars->vec_full[s], 1024);
        bulk_load_1d(smem + L::vec_off + s * 1024, p.negl2 + at, 512, &bars->vec_full[s]);
        bulk_load_1d(smem + L::vec_off + s * 1024 + 512, p.neg_delta + at, 512, &bars->vec_full[s]);
      }
    } else if (warp == 1 && nu > 0 && elect_one()) {
      // ---------------------------------------------------------- MMA issuer: one thread
      constexpr int kFmt = std::is_same<T, __half>::value ? 0 : 1;
      constexpr uint32_t idesc1 = make_idesc_f16(128, BT, kFmt, 0, 0);  // S', dP': 128 x 128, K = D
      // accumulators: 128 x D, K = streamed rows.  Head dims 16 and 32, in the fine modes of D = 64: no K-steps and, beyond
      // 32, no columns of padding (with the same in the forward pass: fp16 B16 H8 S785 D32 full 255 -> 247 us, B8 H16 S1500
      // D32 causal 370 -> 357).
      constexpr bool kPadded = D == 64 && MODE != kPlain;
      const int k_steps = kPadded ? p.D / 16 : D / 16;
      const uint32_t idesc2 = kPadded && p.D <= 32 ? make_idesc_f16(128, 32, kFmt, 0, 1) : make_idesc_f16(128, D, kFmt, 0, 1);
      const uint64_t x_desc = make_desc_sw128(smem_u32(smem + L::x_off), 16, 1024);
      const uint64_t y_desc = make_desc_sw128(smem_u32(smem + L::y_off), 16, 1024);
      const uint64_t ak_desc = make_desc_sw128(smem_u32(smem + L::a_off), 16, 1024);       // streamed tiles as K-major
      const uint64_t bk_desc = make_desc_sw128(smem_u32(smem + L::b_off), 16, 1024);
      const uint64_t am_desc = make_desc_sw128(smem_u32(smem + L::a_off), L::kSub, 1024);  // and as MN-major operands
      const uint64_t bm_desc = make_desc_sw128(smem_u32(smem + L::b_off), L::kSub, 1024);
      // 128 x 128 product of a stationary and a streamed tile over the head dimension
      auto issue_mma1 = [&](uint32_t d_col, uint64_t own_desc, uint64_t str_desc, uint64_t* full) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t off = (uint64_t)(((kk >> 2) * L::kSub + (kk & 3) * 32) >> 4);
          if (kk == 0) mma_ss(tmem_base + d_col, own_desc + off, str_desc + off, idesc1, 0u);
          else if (kk < k_steps) mma_ss_acc(tmem_base + d_col, own_desc + off, str_desc + off, idesc1);
        }
        mma_commit(full);
      };
      bool ok = true;
      auto wait = [&](uint64_t* bar, int phase) {
        if (ok) ok = mbar_wait(bar, phase & 1, abort_flag);
        tc_fence_after();
      };
      auto issue_s = [&](int u) {
        wait(&bars->a_full[u % NA], u / NA);
        if (!ok) return;
        issue_mma1((uint32_t)((u % NSB) * 128), x_desc, ak_desc + (uint64_t)((u % NA) * (L::kTile >> 4)),
                   &bars->s_full[u % NSB]);
      };
      auto issue_dp = [&](int u) {
        wait(&bars->b_full[u % NB], u / NB);
        if (!ok) return;
        issue_mma1(COL_DP + (uint32_t)((u % NDB) * 128), y_desc, bk_desc + (uint64_t)((u % NB) * (L::kTile >> 4)),
                   &bars->dp_full[u % NDB]);
      };
      // K-steps of 16 streamed rows of an accumulator: 32 rows of warpgroup e's 64 for dV, all 64 for dK / dQ.  The
      // 16-bit operands of a warpgroup's rows lie over its own 64 columns of S' or dP'.
      auto issue_dv = [&](int u, int e, int c) {
        const uint64_t tile = bm_desc + (uint64_t)((u % NB) * (L::kTile >> 4));
        const uint32_t t_p = tmem_base + (uint32_t)((u % NSB) * 128 + e * HALF);
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          const int k4 = c * 2 + k2;
          const uint64_t off = (uint64_t)(((e * 4 + k4) * 16 * 128) >> 4);
          if (e == 0 && k4 == 0) mma_ts(tmem_base + COL_ACC, t_p, tile, idesc2, u == 0 ? 0u : 1u);
          else mma_ts_acc(tmem_base + COL_ACC, t_p + (uint32_t)(k4 * 8), tile + off, idesc2);
        }
      };
      auto issue_ds = [&](int u, int e, uint32_t acc_col) {
        const uint64_t tile = am_desc + (uint64_t)((u % NA) * (L::kTile >> 4));
        const uint32_t t_ds = tmem_base + COL_DP + (uint32_t)((u % NDB) * 128 + e * HALF);
#pragma unroll
        for (int k4 = 0; k4 < HALF / 16; ++k4) {
          const uint64_t off = (uint64_t)(((e * 4 + k4) * 16 * 128) >> 4);
          constexpr int kStep = MODE != kPlain ? 16 : 8;  // fine modes: hi in 8 columns, lo in the 8 after them
          if (e == 0 && k4 == 0) mma_ts(tmem_base + acc_col, t_ds, tile, idesc2, u == 0 ? 0u : 1u);
          else mma_ts_acc(tmem_base + acc_col, t_ds + (uint32_t)(k4 * kStep), tile + off, idesc2);
          if (MODE != kPlain) mma_ts_acc(tmem_base + acc_col, t_ds + (uint32_t)(k4 * kStep + 8), tile + off, idesc2);
        }
      };
      wait(&bars->x_full, 0);
      issue_s(0);
      wait(&bars->y_full, 0);
      issue_dp(0);
      if (!KM && ok) mma_commit(&bars->b_empty[0]);
      for (int u = 0; ok && u < nu; ++u) {
        const bool more = u + 1 < nu;
        if constexpr (KM) {
          if (NSB == 2 && more) issue_s(u + 1);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            wait(&bars->p_ready[u % NSB][c], u / NSB);
            if (!ok) break;
            issue_dv(u, 0, c);
            issue_dv(u, 1, c);
          }
          if (!ok) break;
          mma_commit(&bars->b_empty[u % NB]);
          if (NSB == 1 && more) issue_s(u + 1);  // over P of this tile, which the MMAs before it have read
          wait(&bars->ds_ready[u % NDB], u / NDB);
          if (ok) issue_ds(u, 0, COL_ACC + D);
          if (ok) issue_ds(u, 1, COL_ACC + D);
          if (!ok) break;
          mma_commit(&bars->a_empty[u % NA]);
          if (more) issue_dp(u + 1);
        } else {
          if (more) {
            wait(&bars->s_free, u);
            if (ok) issue_s(u + 1);
            if (ok) issue_dp(u + 1);
            if (ok) mma_commit(&bars->b_empty[(u + 1) % NB]);
          }
          wait(&bars->ds_ready[u % NDB], u / NDB);
          if (ok) issue_ds(u, 0, COL_ACC);
          if (ok) issue_ds(u, 1, COL_ACC);
          if (ok) mma_commit(&bars->a_empty[u % NA]);
        }
      }
      if (ok) mma_commit(&bars->acc_done);
    }
  } else {
    reg_alloc<REGS_CONSUMER>();
    // ------------------------------------------------------------ consumers: thread = owned row
    const int e = (warp - 4) >> 2;  // half of the streamed rows this warpgroup handles
    const int lg = warp & 3;
    const int row = lg * 32 + lane;
    const int own = own0 + row;  // key j (key-major) or query i (query-major)
    const uint32_t t_lane = tmem_base + ((uint32_t)(lg * 32) << 16);
    const float c2 = p.sm_scale * kLog2e;
    const uint64_t c22 = pack_f32x2(c2, c2);
    float my_nl = 0.f, my_nd = 0.f;  // query-major: this thread's query
    if (!KM) {
      my_nl = p.negl2[vec_row + own];  // own < Mpad always
      my_nd = p.neg_delta[vec_row + own];
    }
    [[maybe_unused]] GradScale gsc{1.f, 1.f};
    if constexpr (kScaledDs<T, MODE>) {
      gsc = grad_scale(p, b, h, hk, lane);
      my_nd *= gsc.mul;
    }
    // what a kept entry's dP is multiplied by (keep_scale is 1 without dropout); query-major kernels put the power of
    // two here and on delta, key-major ones, whose delta comes with the streamed rows, on P
    const float kept = KM ? p.keep_scale : p.keep_scale * gsc.mul;

    // dropout: this thread's two words of the next tile's mask, fetched a tile ahead.  Query-major: entries [64 e, 64 e
    // + 64) of its query row; key-major: the word of the warp's 32 keys in rows 64 e + lane and 64 e + 32 + lane.
    [[maybe_unused]] uint32_t ahead[2] = {0u, 0u};
    [[maybe_unused]] auto fetch_mask = [&](int u) {
      const int bh = b * p.Hq + h - p.bh0, nqt = p.Mpad / BT, nkt = (p.N + BT - 1) / BT;
      if (KM) {
        const uint32_t* w = p.mask + mask_word(bh, u0 + u, own_tile, nqt, nkt) + (e * HALF + lane) * 4 + lg;
        ahead[0] = w[0];
        ahead[1] = w[128];
      } else {
        const uint2 w = *reinterpret_cast<const uint2*>(p.mask + mask_word(bh, own_tile, u, nqt, nkt) + row * 4 + e * 2);
        ahead[0] = w.x;
        ahead[1] = w.y;
      }
    };
    if constexpr (MODE == kDrop) {
      if (p.mask != nullptr && nu > 0) fetch_mask(0);
    }

    // One streamed tile, kMasked where an entry of this warpgroup's 128 x 64 block may be hidden.
    auto tile_body = [&](auto masked_tag, int u) -> bool {
      constexpr bool kMasked = decltype(masked_tag)::value;
      const int str0 = (u0 + u) * BT + e * HALF;  // first streamed row of this half
      // causal: (query i, key j) is visible iff j <= i + p_seq.  Column x of the half is streamed row
      // str0 + x.  Key-major (own = j, streamed = i): visible iff x >= own - p_seq - str0.
      // Query-major (own = i, streamed = j): visible iff x <= own + p_seq - str0.
      // Keys beyond N are masked too (query-major): their scores of zero against a very negative L would make
      // P infinite, and infinity times the zero K row is not zero.
      [[maybe_unused]] int x_lo = 0, x_hi = HALF - 1;
      if constexpr (kMasked) {
        if (p.causal && KM) x_lo = own - p.p_seq - str0;
        // Query rows beyond M are masked under dropout (key-major): against their zero dout rows stand weights of
        // 1 / (1 - p), which fp16 need not hold.
        if (KM && MODE == kDrop) x_hi = p.M - 1 - str0;
        if (!KM) x_hi = min(p.N - 1, p.causal ? own + p.p_seq : p.N - 1) - str0;
      }
      [[maybe_unused]] uint32_t keep[2] = {~0u, ~0u};  // bit x of the pair: entry x of this thread's 64 is kept
      if (MODE == kDrop && p.mask != nullptr) {
        keep[0] = KM ? warp_transpose_bits(ahead[0], lane) : ahead[0];
        keep[1] = KM ? warp_transpose_bits(ahead[1], lane) : ahead[1];
        if (u + 1 < nu) fetch_mask(u + 1);
      } else if constexpr (MODE == kDrop) {
        // Philox counter of the half's first entry of this thread, 32-bit wrap-around.  About 25 integer instructions
        // an entry bound the tile; a rolled loop of 16 keeps them in the instruction caches.
        const uint32_t bh = (uint32_t)(b * p.Hq + h);
        const uint32_t lin_step = KM ? (uint32_t)p.N : 1u;
        uint32_t lin = KM ? (bh * (uint32_t)p.M + (uint32_t)str0) * (uint32_t)p.N + (uint32_t)own
                          : (bh * (uint32_t)p.M + (uint32_t)own) * (uint32_t)p.N + (uint32_t)str0;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t bits = 0u;
#pragma unroll
          for (int x = 0; x < 16; ++x, lin += lin_step) bits |= dropout_keep(p.drop, lin) ? 1u << x : 0u;
          if (c < 2) keep[0] = c == 0 ? bits : keep[0] | bits << 16;
          else keep[1] = c == 2 ? bits : keep[1] | bits << 16;
        }
      }
      const uint32_t t_s = t_lane + (uint32_t)((u % NSB) * 128 + e * HALF);
      const uint32_t t_dp = t_lane + COL_DP + (uint32_t)((u % NDB) * 128 + e * HALF);
      const float* vl = reinterpret_cast<const float*>(smem + L::vec_off + (u & 1) * 1024) + e * HALF;
      if (KM && !mbar_wait(&bars->vec_full[u & 1], (u >> 1) & 1, abort_flag)) return false;
      if (!mbar_wait(&bars->s_full[u % NSB], (u / NSB) & 1, abort_flag)) return false;
      tc_fence_after();
      uint32_t sv[HALF];  // S', then P'
      tmem_ld32(t_s, reinterpret_cast<uint32_t(&)[32]>(sv[0]));
      tmem_ld32(t_s + 32, reinterpret_cast<uint32_t(&)[32]>(sv[32]));
      tmem_wait_ld();
      if (!KM) {  // the next tile's S' may be written
        tc_fence_before();
        mbar_arrive(&bars->s_free);
      }
      // ---- P' = exp2(S' c2 - L log2e); key-major, where it is the operand of dV, handed over in chunks of 32 rows
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int x = c * 32; x < c * 32 + 32; x += 4) {
          uint64_t n01 = pack_f32x2(my_nl, my_nl), n23 = n01;
          if (KM) {
            const float4 a = *reinterpret_cast<const float4*>(vl + x);
            n01 = pack_f32x2(a.x, a.y);
            n23 = pack_f32x2(a.z, a.w);
          }
          float t[4];
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[x]), __uint_as_float(sv[x + 1])), c22, n01), t[0], t[1]);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[x + 2]), __uint_as_float(sv[x + 3])), c22, n23), t[2], t[3]);
          float pr[4];
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            float pe = fast_exp2(t[y]);
            if (kMasked && !(x + y >= x_lo && x + y <= x_hi)) pe = 0.f;
            sv[x + y] = __float_as_uint(pe);
            pr[y] = pe;
            // a product, not a select: a weight that is not finite stays visible where it is dropped
            if constexpr (MODE == kDrop) pr[y] = pe * ((keep[c] >> (x + y - c * 32) & 1u) ? kept : 0.f);
          }
          pk[(x - c * 32) / 2] = pack2<T>(pr[0], pr[1]);
          pk[(x - c * 32) / 2 + 1] = pack2<T>(pr[2], pr[3]);
        }
        if (KM) {
          tmem_st16(t_s + c * 16, pk);
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(&bars->p_ready[u % NSB][c]);
        }
      }
      // ---- dS' = P' (dP' - delta)
      if (!mbar_wait(&bars->dp_full[u % NDB], (u / NDB) & 1, abort_flag)) return false;
      tc_fence_after();
      const float* vd = vl + 128;
      auto neg_delta4 = [&](int x, float (&nd)[4]) {
        if (KM) {
          const float4 d4 = *reinterpret_cast<const float4*>(vd + x);
          nd[0] = d4.x; nd[1] = d4.y; nd[2] = d4.z; nd[3] = d4.w;
        } else {
          nd[0] = nd[1] = nd[2] = nd[3] = my_nd;
        }
      };
      if constexpr (MODE == kPlain) {
        uint32_t dv[HALF], dk[HALF / 2];
        tmem_ld32(t_dp, reinterpret_cast<uint32_t(&)[32]>(dv[0]));
        tmem_ld32(t_dp + 32, reinterpret_cast<uint32_t(&)[32]>(dv[32]));
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < HALF; x += 4) {
          float nd[4];
          neg_delta4(x, nd);
#pragma unroll
          for (int y = 0; y < 4; y += 2) {
            const uint64_t t = add_f32x2(pack_f32x2(__uint_as_float(dv[x + y]), __uint_as_float(dv[x + y + 1])),
                                         pack_f32x2(nd[y], nd[y + 1]));
            float d0, d1;
            unpack_f32x2(mul_f32x2(t, pack_f32x2(__uint_as_float(sv[x + y]), __uint_as_float(sv[x + y + 1]))), d0, d1);
            dk[(x + y) / 2] = pack2<T>(d0, d1);
          }
        }
        tmem_st32(t_dp, dk);
      } else {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t dv[32], out[32];  // out: per 16 streamed rows 8 columns of hi, 8 of lo
          tmem_ld32(t_dp + c * 32, dv);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            float nd[4], ds[4];
            neg_delta4(c * 32 + x, nd);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
              const float ks = MODE == kDrop && !(keep[c] >> (x + y) & 1u) ? 0.f : kept;
              const float t = fmaf(__uint_as_float(dv[x + y]), ks, nd[y]);
              const float pe = __uint_as_float(sv[c * 32 + x + y]);
              ds[y] = (KM ? pe * gsc.mul : pe) * t;
            }
#pragma unroll
            for (int y = 0; y < 4; y += 2) {
              const uint32_t hi = pack2<T>(ds[y], ds[y + 1]);
              const float2 h2 = unpack2<T>(hi);
              const int at = (x >> 4) * 16 + ((x & 15) + y) / 2;
              out[at] = hi;
              out[at + 8] = pack2<T>(ds[y] - h2.x, ds[y + 1] - h2.y);
            }
          }
          tmem_st32(t_dp + c * 32, out);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->ds_ready[u % NDB]);
      if (KM) {  // this warp has read the tile's L and delta
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->vec_empty[u & 1]);
      }
      return true;
    };
    bool alive = true;
    for (int u = 0; alive && u < nu; ++u) {
      const int str0 = (u0 + u) * BT + e * HALF;
      bool masked;
      if (KM) masked = (p.causal && own0 + BT - 1 - p.p_seq > str0) || (MODE == kDrop && str0 + HALF > p.M);
      else masked = str0 + HALF > (p.causal ? min(p.N, own0 + p.p_seq + 1) : p.N);
      alive = masked ? tile_body(std::true_type{}, u) : tile_body(std::false_type{}, u);
    }

    // ---- epilogue: accumulators -> 16-bit -> swizzled smem -> TMA store (clips at the tensor's edge)
    if (alive && nu > 0) {
      if (!mbar_wait(&bars->acc_done, 0, abort_flag)) alive = false;
      tc_fence_after();
    }
    if (alive) {
      // Every MMA has completed, so the ring is free for staging: 32 rows x 64 columns (4 KB) per (warp, sub-tile).
      unsigned char* ost = smem + L::a_off + (warp - 4) * (32 * D * 2);
      // key-major: warpgroup 0 stores dV (acc0), warpgroup 1 stores dK (acc1, times sm_scale);
      // query-major: dQ (acc0, times sm_scale), warpgroup w takes the 64-column sub-tiles w, w + 2, ...
      const uint32_t t_acc = t_lane + COL_ACC + (KM ? (uint32_t)(e * D) : 0u);
      const float oscale = (KM && e == 0) ? 1.f : p.sm_scale * gsc.inv;
      const int sub_first = KM ? 0 : e, sub_step = KM ? 1 : 2;
      float* part = MODE == kPlain ? nullptr : (e == 0 ? p.part0 : p.part1);
      for (int sub = sub_first; sub < D / 64; sub += sub_step) {
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t ro[32];
          if (nu > 0) {
            tmem_ld32(t_acc + (uint32_t)(sub * 64 + c * 32), ro);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int x = 0; x < 32; ++x) ro[x] = 0u;  // no streamed tile at all: the gradient rows are zero
          }
          if constexpr (MODE != kPlain) {
            if (part != nullptr) {  // a row piece of up to 128 bytes per thread
              float* dst = part + (((int64_t)b * p.Hq + h) * p.N + own) * p.D + sub * 64 + c * 32;
#pragma unroll
              for (int g = 0; g < 8; ++g)
                if (own < p.N && sub * 64 + c * 32 + g * 4 < p.D)
                  *reinterpret_cast<float4*>(dst + g * 4) =
                      make_float4(__uint_as_float(ro[g * 4]) * oscale, __uint_as_float(ro[g * 4 + 1]) * oscale,
                                  __uint_as_float(ro[g * 4 + 2]) * oscale, __uint_as_float(ro[g * 4 + 3]) * oscale);
              continue;
            }
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 w;
            w.x = pack2<T>(__uint_as_float(ro[g * 8 + 0]) * oscale, __uint_as_float(ro[g * 8 + 1]) * oscale);
            w.y = pack2<T>(__uint_as_float(ro[g * 8 + 2]) * oscale, __uint_as_float(ro[g * 8 + 3]) * oscale);
            w.z = pack2<T>(__uint_as_float(ro[g * 8 + 4]) * oscale, __uint_as_float(ro[g * 8 + 5]) * oscale);
            w.w = pack2<T>(__uint_as_float(ro[g * 8 + 6]) * oscale, __uint_as_float(ro[g * 8 + 7]) * oscale);
            const int cc = c * 4 + g;  // 16-byte chunk inside the 64-column sub-tile
            *reinterpret_cast<uint4*>(ost + sub * 4096 + lane * 128 + ((cc ^ (lane & 7)) << 4)) = w;
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && part == nullptr) {
        const CUtensorMap* om = (KM && e == 1) ? &maps.o1 : &maps.o0;
        for (int sub = sub_first; sub < D / 64; sub += sub_step)
          tma_store_4d(om, ost + sub * 4096, sub * 64, own0 + lg * 32, h, b);
        tma_store_commit();
        tma_store_wait<0>();
      }
    }
  }

  // ------------------------------------------------------------ common exit
  if (KM) {
    griddep_launch_dependents();
    griddep_wait();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 1);
    for (int w = 0; w < 50; ++w) __nanosleep(20000);  // let copies in flight land before the smem goes away
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Pre-pass: delta_i = sum_d out_id * dout_id and -L_i * log2(e), both into arrays padded to whole
// 128-row tiles (zeros in the padding), so that the kernels can fetch a tile's 128 values with one
// aligned bulk copy.  Bound by HBM: D / 8 lanes per row, 16 bytes of each operand a lane, four rows in flight
// (bf16 B1 H28 S4096 D128: 15 us; 34 us with a warp and 4-byte loads to a row).
// STATS: each block also leaves bounds of its rows' |dout_i|^2 and |delta_i|, and further blocks one of |v_j|^2, for
// grad_scale.  The squared norms are bounded by D / 8 times the largest of a row's D / 8 pieces: at most 1.5 bits (3 in
// the product) above the norms themselves, which would take three or four shuffles a row.
constexpr int kPrepRows = 4;
struct BwStats {
  float2* g;
  float* v;
  int g_blocks, v_blocks;  // per query head, per kv head
};
template <typename T>
__device__ __forceinline__ float norm2(const uint4& w4) {
  const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
  float sum = 0.f;
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const float2 a = unpack2<T>(w[y]);
    sum = fmaf(a.x, a.x, fmaf(a.y, a.y, sum));
  }
  return sum;
}
// the block's (8 warps') largest x and y, in thread 0
__device__ __forceinline__ float2 block_max(float x, float y, float2 (&red)[8]) {
  x = warp_max(x);
  y = warp_max(y);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(x, y);
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      x = fmaxf(x, red[w].x);
      y = fmaxf(y, red[w].y);
    }
  }
  return make_float2(x, y);
}
// A word of the mask per thread, two blocks a tile; tiles without a visible entry are left out.  The mask's first head is bh0.
__device__ __forceinline__ void draw_mask(const BwdParams& p, uint32_t* mask, int bh0, int64_t block) {
  const int nqt = (p.M + BT - 1) / BT, nkt = (p.N + BT - 1) / BT;
  const int64_t tile = block >> 1;
  const int kt = (int)(tile % nkt);
  const int64_t rest = tile / nkt;
  const int qt = (int)(rest % nqt), bh = bh0 + (int)(rest / nqt);
  if (p.causal && kt * BT > qt * BT + BT - 1 + p.p_seq) return;
  const int at = (int)(block & 1) * 256 + threadIdx.x;
  uint32_t lin = ((uint32_t)bh * (uint32_t)p.M + (uint32_t)(qt * BT + (at >> 2))) * (uint32_t)p.N + (uint32_t)(kt * BT + (at & 3) * 32);
  uint32_t bits = 0u;
#pragma unroll 8
  for (int x = 0; x < 32; ++x) bits |= dropout_keep(p.drop, lin + (uint32_t)x) ? 1u << x : 0u;
  mask[tile * 512 + at] = bits;
}
// The mask alone, before a forward pass that reads it and leaves it to the backward pass, where the forward pass's own CTAs
// would not fill the chip with the draw: fp16 B1 H16 S1000 D64 causal, p = 0.1, forward and backward 77 us, 103 with the mask
// drawn in the forward kernel and kept, 117 drawn in both passes.
__global__ void __launch_bounds__(256) dropout_mask_kernel(BwdParams p, uint32_t* mask) {
  griddep_launch_dependents();
  griddep_wait();  // the mask's memory may have been another one's
  draw_mask(p, mask, 0, blockIdx.x);
}
template <typename T, bool STATS, bool DRAW>
__global__ void __launch_bounds__(256) bwd_prep_kernel(BwdParams p, float* negl2, float* neg_delta, int Mpad, BwStats st,
                                                       uint32_t* mask, int bh0, unsigned mask_block0) {
  griddep_launch_dependents();
  if (DRAW && blockIdx.x >= mask_block0) {
    draw_mask(p, mask, bh0, blockIdx.x - mask_block0);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lpr = p.D >> 3, rows_at_once = 32 / lpr, sub = lane & (lpr - 1);
  const int block_rows = 8 * kPrepRows * rows_at_once;
  const int row0 = warp * kPrepRows * rows_at_once + lane / lpr;  // within the block's rows
  [[maybe_unused]] __shared__ float2 red[8];
  if constexpr (STATS) {
    const int vb = (int)blockIdx.x - p.B * p.Hq * st.g_blocks;
    if (vb >= 0) {
      const int bk = vb / st.v_blocks, j0 = (vb - bk * st.v_blocks) * block_rows + row0;
      const T* v = reinterpret_cast<const T*>(p.v) + (bk / p.Hk) * p.v_sb + (bk % p.Hk) * p.v_sh + 8 * sub;
      uint4 vv[kPrepRows];
#pragma unroll
      for (int x = 0; x < kPrepRows; ++x) {
        const int j = j0 + x * rows_at_once;
        vv[x] = j < p.N ? *reinterpret_cast<const uint4*>(v + (int64_t)j * p.v_ss) : make_uint4(0u, 0u, 0u, 0u);
      }
      float v2 = 0.f;
#pragma unroll
      for (int x = 0; x < kPrepRows; ++x) v2 = fmaxf(v2, norm2<T>(vv[x]));
      v2 = block_max(v2, 0.f, red).x;
      if (threadIdx.x == 0) st.v[vb] = v2 * (float)lpr;
      return;
    }
  }
  const int bh = blockIdx.x / st.g_blocks;
  const int i0 = (blockIdx.x - bh * st.g_blocks) * block_rows + row0;
  const int h = bh % p.Hq, b = bh / p.Hq;
  const T* o = reinterpret_cast<const T*>(p.o) + b * p.o_sb + h * p.o_sh + 8 * sub;
  const T* g = reinterpret_cast<const T*>(p.dout) + b * p.do_sb + h * p.do_sh + 8 * sub;
  uint4 ov[kPrepRows], gv[kPrepRows];
  [[maybe_unused]] float g2 = 0.f, dl = 0.f;
#pragma unroll
  for (int x = 0; x < kPrepRows; ++x) {
    const int i = i0 + x * rows_at_once;
    ov[x] = gv[x] = make_uint4(0u, 0u, 0u, 0u);
    if (i < p.M) {
      ov[x] = *reinterpret_cast<const uint4*>(o + (int64_t)i * p.o_ss);
      gv[x] = *reinterpret_cast<const uint4*>(g + (int64_t)i * p.do_ss);
    }
  }
#pragma unroll
  for (int x = 0; x < kPrepRows; ++x) {
    const int i = i0 + x * rows_at_once;
    if constexpr (STATS) g2 = fmaxf(g2, norm2<T>(gv[x]));
    const uint32_t ow[4] = {ov[x].x, ov[x].y, ov[x].z, ov[x].w}, gw[4] = {gv[x].x, gv[x].y, gv[x].z, gv[x].w};
    float sum = 0.f;
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const float2 a = unpack2<T>(ow[y]), c = unpack2<T>(gw[y]);
      sum = fmaf(a.x, c.x, fmaf(a.y, c.y, sum));
    }
    for (int s = lpr >> 1; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
    if constexpr (STATS) dl = fmaxf(dl, fabsf(sum));
    if (sub == 0 && i < Mpad) {
      float nl = 0.f;
      if (i < p.M) {
        const float Li = p.L[(int64_t)bh * p.M + i];
        nl = (Li == __int_as_float(0xff800000)) ? 0.f : -Li * kLog2e;  // no visible key: every weight is masked anyway
      }
      neg_delta[(int64_t)bh * Mpad + i] = -sum;
      negl2[(int64_t)bh * Mpad + i] = nl;
    }
  }
  if constexpr (STATS) {
    const float2 m = block_max(g2, dl, red);
    if (threadIdx.x == 0) st.g[blockIdx.x] = make_float2(m.x * (float)lpr, m.y);
  }
}

// out[b,hk,j,:] = sum over the G query heads of the kv head, in head order, of part[b,hk*G+g,j,:]; one thread per 8
// elements, dK in the first half of the grid and dV in the second.  Bound by the reads (bf16 Hq28 Hk4 S4096 D128:
// 15 us for both; 2 x 17 us with a launch each and 4 bytes a thread).
struct GroupSumOut {
  void* out;
  int64_t sb, sh, ss;
};
template <typename T, typename P>
__global__ void __launch_bounds__(256) bwd_group_sum_kernel(const P* dk_part, const P* dv_part,
                                                            GroupSumOut dk, GroupSumOut dv, int B, int Hk, int G, int N,
                                                            int D) {
  griddep_wait();
  griddep_launch_dependents();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int chunks = D >> 3;
  if (idx >= (int64_t)B * Hk * N * chunks) return;
  const bool second = blockIdx.y != 0;
  const P* part = second ? dv_part : dk_part;
  const GroupSumOut o = second ? dv : dk;
  const int c = (int)(idx % chunks);
  const int64_t r = idx / chunks;
  const int j = (int)(r % N);
  const int64_t bk = r / N;
  const int hk = (int)(bk % Hk), b = (int)(bk / Hk);
  const P* src = part + (((bk * G) * N + j) * D + c * 8);
  const int64_t step = (int64_t)N * D;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int g = 0; g < G; ++g, src += step) {
    if constexpr (std::is_same<P, float>::value) {
      const float4 a = *reinterpret_cast<const float4*>(src), e = *reinterpret_cast<const float4*>(src + 4);
      s[0] += a.x; s[1] += a.y; s[2] += a.z; s[3] += a.w;
      s[4] += e.x; s[5] += e.y; s[6] += e.z; s[7] += e.w;
    } else {
      const uint4 a = *reinterpret_cast<const uint4*>(src);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const float2 v = unpack2<T>(w[y]);
        s[2 * y] += v.x;
        s[2 * y + 1] += v.y;
      }
    }
  }
  T* dst = reinterpret_cast<T*>(o.out) + b * o.sb + hk * o.sh + (int64_t)j * o.ss + c * 8;
  *reinterpret_cast<uint4*>(dst) =
      make_uint4(pack2<T>(s[0], s[1]), pack2<T>(s[2], s[3]), pack2<T>(s[4], s[5]), pack2<T>(s[6], s[7]));
}

// A launch that may begin while the kernel before it drains (programmatic stream serialization).
template <typename K, typename... A>
cudaError_t launch_overlapped(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  count_launch();
  return e;
}

int mpad_of(int M) { return (M + BT - 1) / BT * BT; }

// Blocks of the pre-pass that `rows` rows of one head take.
int prep_blocks(int rows, int D) {
  const int block_rows = 8 * kPrepRows * (256 / D);
  return (rows + block_rows - 1) / block_rows;
}

// Workspace: [-L*log2e | delta | pre-pass statistics (fine modes) | per-head dK | per-head dV | dropout mask]
struct BwWs {
  size_t delta, g_stat, v_stat, dk, dv, mask, total;
};
size_t head_mask_bytes(int M, int N) { return (size_t)(mpad_of(M) / BT) * ((N + BT - 1) / BT) * 2048; }
// (batch, head) pairs whose mask is held at a time; 0: none is.  Shares of as equal size as they come.
int mask_heads(int B, int Hq, int M, int N) {
  const size_t per = head_mask_bytes(M, N);
  const size_t heads = (size_t)B * Hq, ctas = std::min(mpad_of(M) / BT, (N + BT - 1) / BT);  // a head's, of the smaller launch
  const size_t fit = std::min(std::max(kMaskBytes / per, (kMaskCtas + ctas - 1) / ctas), kMaskBytesMost / per);
  if (fit == 0) return 0;
  const size_t shares = (heads + fit - 1) / fit;
  return (int)((heads + shares - 1) / shares);
}
BwWs bwd_ws(int B, int Hq, int Hk, int M, int N, int D, bool fine) {
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  BwWs w{};
  const size_t vec_bytes = up((size_t)B * Hq * mpad_of(M) * 4);
  const size_t part_bytes = Hq != Hk ? up((size_t)B * Hq * N * D * (fine ? 4 : 2)) : 0;
  w.delta = vec_bytes;
  w.g_stat = 2 * vec_bytes;
  w.v_stat = w.g_stat + (fine ? up((size_t)B * Hq * prep_blocks(mpad_of(M), D) * sizeof(float2)) : 0);
  w.dk = w.v_stat + (fine ? up((size_t)B * Hk * prep_blocks(N, D) * sizeof(float)) : 0);
  w.dv = w.dk + part_bytes;
  w.mask = w.dv + part_bytes;
  w.total = w.mask;  // without the mask
  return w;
}

template <typename T, int D, int MODE>
cudaError_t launch_bwd_td(const BwdParams& p, cudaStream_t s) {
  using Lk = BwSmem<D, true>;
  using Lq = BwSmem<D, false>;
  static PerDeviceOnce once_km, once_qm;
  cudaError_t e;
  if ((e = set_max_smem_once(once_km, tc_bwd_kernel<T, D, true, MODE>, Lk::total)) != cudaSuccess) return e;
  if ((e = set_max_smem_once(once_qm, tc_bwd_kernel<T, D, false, MODE>, Lq::total)) != cudaSuccess) return e;
  const int Mpad = mpad_of(p.M);
  const BwWs ws = bwd_ws(p.B, p.Hq, p.Hk, p.M, p.N, p.D, MODE != kPlain);
  char* base = reinterpret_cast<char*>(p.delta);
  float* negl2 = p.delta;
  float* neg_delta = reinterpret_cast<float*>(base + ws.delta);
  char *dk_part = base + ws.dk, *dv_part = base + ws.dv;
  uint32_t* mask = MODE == kDrop && p.mask_scratch && p.mask == nullptr ? reinterpret_cast<uint32_t*>(base + ws.mask) : nullptr;
  const int heads = p.B * p.Hq, share = mask != nullptr ? mask_heads(p.B, p.Hq, p.M, p.N) : heads;
  using Part = typename std::conditional<MODE == kPlain, T, float>::type;
  const BwStats st{reinterpret_cast<float2*>(base + ws.g_stat), reinterpret_cast<float*>(base + ws.v_stat),
                   prep_blocks(Mpad, p.D), prep_blocks(p.N, p.D)};
  // One round, or (dropout) one per share of the heads, whose pre-pass waits for the kernels that read the last mask: it is
  // launched plainly.  The rows' arrays of all heads come with the first.
  auto prepare = [&](int bh0) -> cudaError_t {
    constexpr bool kStats = kScaledDs<T, MODE>;
    const int n = std::min(share, heads - bh0);
    const unsigned rows_blocks = bh0 > 0 ? 0u : (unsigned)(p.B * p.Hq * st.g_blocks + (kStats ? p.B * p.Hk * st.v_blocks : 0));
    const unsigned mask_blocks = mask != nullptr ? (unsigned)(n * (head_mask_bytes(p.M, p.N) / 1024)) : 0u;
    bwd_prep_kernel<T, kStats, MODE == kDrop><<<rows_blocks + mask_blocks, 256, 0, s>>>(p, negl2, neg_delta, Mpad, st, mask, bh0,
                                                                                      rows_blocks);
    count_launch();
    return cudaGetLastError();
  };
  if ((e = prepare(0)) != cudaSuccess) return e;
  BwTcParams tp{};
  tp.Hq = p.Hq; tp.G = p.G; tp.M = p.M; tp.N = p.N; tp.p_seq = p.p_seq; tp.causal = p.causal; tp.Mpad = Mpad;
  tp.sm_scale = p.sm_scale; tp.negl2 = negl2; tp.neg_delta = neg_delta; tp.D = p.D;
  tp.drop = p.drop;
  tp.keep_scale = 1.f / (1.f - p.drop.p);
  tp.mask = p.mask != nullptr ? p.mask : mask;
  tp.g_stat = st.g; tp.v_stat = st.v; tp.g_blocks = st.g_blocks; tp.v_blocks = st.v_blocks;
  int* status_word = tc_status_word();
  const bool per_head = p.G > 1;
  const bool map_parts = per_head && MODE == kPlain;  // 16-bit partials go through the store maps
  BwTcParams tk = tp;  // the key-major launches': with the fp32 partials
  if (per_head && !map_parts) {
    tk.part0 = reinterpret_cast<float*>(dv_part);
    tk.part1 = reinterpret_cast<float*>(dk_part);
  }
  BwMaps qm, km;
  {  // query-major: dQ
    BwMaps& m = qm;
    if (!make_map_bhsd(&m.x, p.q, p.D, p.M, p.Hq, p.B, p.q_ss, p.q_sh, p.q_sb, 128) ||
        !make_map_bhsd(&m.y, p.dout, p.D, p.M, p.Hq, p.B, p.do_ss, p.do_sh, p.do_sb, 128) ||
        !make_map_bhsd(&m.a, p.k, p.D, p.N, p.Hk, p.B, p.k_ss, p.k_sh, p.k_sb, 128) ||
        !make_map_bhsd(&m.b, p.v, p.D, p.N, p.Hk, p.B, p.v_ss, p.v_sh, p.v_sb, 128) ||
        !make_map_bhsd(&m.o0, p.dq, p.D, p.M, p.Hq, p.B, p.dq_ss, p.dq_sh, p.dq_sb, 32))
      return cudaErrorInvalidValue;
    m.o1 = m.o0;
  }
  {  // key-major: dV, dK (per query head)
    BwMaps& m = km;
    void* dv_dst = map_parts ? static_cast<void*>(dv_part) : p.dv;
    void* dk_dst = map_parts ? static_cast<void*>(dk_part) : p.dk;
    const int o_heads = per_head && !map_parts ? p.Hk : p.Hq;  // (those maps are not used with fp32 partials)
    const int64_t ph_ss = p.D, ph_sh = (int64_t)p.N * p.D, ph_sb = (int64_t)p.Hq * p.N * p.D;
    if (!make_map_bhsd(&m.x, p.k, p.D, p.N, p.Hk, p.B, p.k_ss, p.k_sh, p.k_sb, 128) ||
        !make_map_bhsd(&m.y, p.v, p.D, p.N, p.Hk, p.B, p.v_ss, p.v_sh, p.v_sb, 128) ||
        !make_map_bhsd(&m.a, p.q, p.D, p.M, p.Hq, p.B, p.q_ss, p.q_sh, p.q_sb, 128) ||
        !make_map_bhsd(&m.b, p.dout, p.D, p.M, p.Hq, p.B, p.do_ss, p.do_sh, p.do_sb, 128) ||
        !make_map_bhsd(&m.o0, dv_dst, p.D, p.N, o_heads, p.B, map_parts ? ph_ss : p.dv_ss,
                       map_parts ? ph_sh : p.dv_sh, map_parts ? ph_sb : p.dv_sb, 32) ||
        !make_map_bhsd(&m.o1, dk_dst, p.D, p.N, o_heads, p.B, map_parts ? ph_ss : p.dk_ss,
                       map_parts ? ph_sh : p.dk_sh, map_parts ? ph_sb : p.dk_sb, 32))
      return cudaErrorInvalidValue;
  }
  for (int bh0 = 0; bh0 < heads; bh0 += share) {
    if (bh0 > 0 && (e = prepare(bh0)) != cudaSuccess) return e;
    tp.bh0 = tk.bh0 = bh0;
    const bool all = share == heads;
    const unsigned gx = all ? p.Hq : std::min(share, heads - bh0), gy = all ? p.B : 1;
    if ((e = launch_overlapped(tc_bwd_kernel<T, D, false, MODE>, dim3(gx, gy, (p.M + BT - 1) / BT), NTHREADS, Lq::total, s,
                               qm, tp, status_word)) != cudaSuccess)
      return e;
    if ((e = launch_overlapped(tc_bwd_kernel<T, D, true, MODE>, dim3(gx, gy, (p.N + BT - 1) / BT), NTHREADS, Lk::total, s,
                               km, tk, status_word)) != cudaSuccess)
      return e;
  }
  if (per_head) {
    const int64_t n = (int64_t)p.B * p.Hk * p.N * (p.D / 8);
    const dim3 grid((unsigned)((n + 255) / 256), 2, 1);
    const GroupSumOut dk{p.dk, p.dk_sb, p.dk_sh, p.dk_ss}, dv{p.dv, p.dv_sb, p.dv_sh, p.dv_ss};
    if ((e = launch_overlapped(bwd_group_sum_kernel<T, Part>, grid, 256, 0, s, reinterpret_cast<const Part*>(dk_part),
                               reinterpret_cast<const Part*>(dv_part), dk, dv, p.B, p.Hk, p.G, p.N, p.D)) !=
        cudaSuccess)
      return e;
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t launch_bwd_t(const BwdParams& p, cudaStream_t s) {
  if (p.drop.p > 0.f) return p.D == 128 ? launch_bwd_td<T, 128, kDrop>(p, s) : launch_bwd_td<T, 64, kDrop>(p, s);
  if (p.D < 64) return launch_bwd_td<T, 64, kFine>(p, s);
  return p.D == 128 ? launch_bwd_td<T, 128, kPlain>(p, s) : launch_bwd_td<T, 64, kPlain>(p, s);
}

}  // namespace

size_t tc_bwd_workspace_bytes(int B, int Hq, int Hk, int M, int N, int D, bool fine) {
  return bwd_ws(B, Hq, Hk, M, N, D, fine).total;
}

size_t tc_bwd_mask_bytes(int B, int Hq, int M, int N) {
  return mask_heads(B, Hq, M, N) * head_mask_bytes(M, N);
}

cudaError_t launch_dropout_mask(const FwdParams& p, uint32_t* mask, cudaStream_t s) {
  BwdParams b{};
  b.B = p.B; b.Hq = p.Hq; b.M = p.M; b.N = p.N; b.p_seq = p.p_seq; b.causal = p.causal;
  b.drop = p.drop;
  const unsigned blocks = (unsigned)((size_t)p.B * p.Hq * (head_mask_bytes(p.M, p.N) / 1024));
  const cudaError_t e = launch_overlapped(dropout_mask_kernel, dim3(blocks), 256, 0, s, b, mask);
  return e != cudaSuccess ? e : cudaGetLastError();
}

bool tc_bwd_supported(const BwdParams& p, int dtype) {
  (void)dtype;
  if (!tc_head_dim(p.D)) return false;
  if (!(p.sm_scale > 0.f)) return false;
  if (!device_is_sm100() || get_encode() == nullptr) return false;
  if ((p.N + BT - 1) / BT > 65535 || (p.M + BT - 1) / BT > 65535 || p.B > 65535) return false;
  return ok16(p.q, p.q_sb, p.q_sh, p.q_ss) && ok16(p.k, p.k_sb, p.k_sh, p.k_ss) &&
         ok16(p.v, p.v_sb, p.v_sh, p.v_ss) && ok16(p.o, p.o_sb, p.o_sh, p.o_ss) &&
         ok16(p.dout, p.do_sb, p.do_sh, p.do_ss) && ok16(p.dq, p.dq_sb, p.dq_sh, p.dq_ss) &&
         ok16(p.dk, p.dk_sb, p.dk_sh, p.dk_ss) && ok16(p.dv, p.dv_sb, p.dv_sh, p.dv_ss);
}

cudaError_t launch_tc_bwd(const BwdParams& p, int dtype, cudaStream_t s) {
  return dtype == FAWS_FP16 ? launch_bwd_t<__half>(p, s) : launch_bwd_t<__nv_bfloat16>(p, s);
}

}  // namespace faws
