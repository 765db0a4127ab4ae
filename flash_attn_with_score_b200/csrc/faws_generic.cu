// CUDA-core kernels of the attention-with-scores family.
//
// These cover every shape the operators accept (head dim 16/32/64/128, ragged
// lengths, M != N, unaligned views).  The tcgen05 kernels in faws_tc.cu take
// over whenever a problem fits them; these stay as the path for the rest and
// as the on-device cross-check in the tests.
//
// One CTA = 64 query rows of one (batch, query head); key tiles of 64 are
// streamed through shared memory.  The loop body is the FlashAttention-2
// forward step (flash.py:432-470) with the score-tile hooks of
// attention_with_scores.py:141-162 (store), attention_with_row_sum.py:146-156
// (row reduce) and attention_with_col_sum.py:170-191 (column reduce, written as
// a per-CTA partial instead of an atomic add).
#include "faws_internal.cuh"
#include "faws_tc_ptx.cuh"

namespace faws {
namespace {

constexpr int BM = kGenericBlockM;
constexpr int BN = kGenericBlockN;
constexpr int NT = 256;
constexpr int SLD = BN + 1;
constexpr float kLog2e = 1.4426950408889634f;
#define FAWS_NEG_INF (__int_as_float(0xff800000))

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// rows [r0, r0+64) of a (rows, D) matrix -> smem, zero outside [r_lo, r_hi)
template <typename T>
__device__ __forceinline__ void load_tile(T* dst, int lds, const T* src, int64_t stride_s, int r0,
                                          int r_lo, int r_hi, int D, int vec) {
  if (vec) {
    const int chunks = D >> 3;
    for (int idx = threadIdx.x; idx < 64 * chunks; idx += NT) {
      const int r = idx / chunks, c = idx - r * chunks;
      const int row = r0 + r;
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (row >= r_lo && row < r_hi)
        val = *reinterpret_cast<const uint4*>(src + (int64_t)row * stride_s + c * 8);
      *reinterpret_cast<uint4*>(dst + r * lds + c * 8) = val;
    }
  } else {
    for (int idx = threadIdx.x; idx < 64 * D; idx += NT) {
      const int r = idx / D, c = idx - r * D;
      const int row = r0 + r;
      T val = from_f<T>(0.f);
      if (row >= r_lo && row < r_hi) val = src[(int64_t)row * stride_s + c];
      dst[r * lds + c] = val;
    }
  }
}

// acc[r][c] = sum_d A[(ty*4+r)][d] * Bm[(tx+16c)][d]
template <typename T>
__device__ __forceinline__ void tile_dot(const T* A, const T* Bm, int lds, int D, int ty, int tx,
                                         float (&acc)[4][4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
  for (int d = 0; d < D; d += 2) {
    float ax[4], ay[4], bx[4], by[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      ax[r] = to_f(A[(ty * 4 + r) * lds + d]);
      ay[r] = to_f(A[(ty * 4 + r) * lds + d + 1]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      bx[c] = to_f(Bm[(tx + 16 * c) * lds + d]);
      by[c] = to_f(Bm[(tx + 16 * c) * lds + d + 1]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(ax[r], bx[c], fmaf(ay[r], by[c], acc[r][c]));
  }
}

template <typename T>
__global__ void __launch_bounds__(NT) generic_fwd_kernel(FwdParams p, int vec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int D = p.D, lds = D + 8;
  T* Qs = reinterpret_cast<T*>(smem_raw);
  T* Ks = Qs + BM * lds;
  T* Vs = Ks + BN * lds;
  float* Ss = reinterpret_cast<float*>(Vs + BN * lds);
  float* m_s = Ss + BM * SLD;
  float* l_s = m_s + BM;
  float* a_s = l_s + BM;

  const int tid = threadIdx.x;
  const int qb_abs = p.m_begin / BM + blockIdx.x;
  const int m0 = qb_abs * BM;
  const int h = blockIdx.y, b = blockIdx.z, hk = h / p.G;
  const int ty = tid >> 4, tx = tid & 15;

  const T* qp = reinterpret_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
  const T* kp = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh;
  const T* vp = reinterpret_cast<const T*>(p.v) + b * p.v_sb + hk * p.v_sh;
  T* op = reinterpret_cast<T*>(p.o) + b * p.o_sb + h * p.o_sh;
  const int64_t bh = (int64_t)b * p.Hq + h;

  load_tile(Qs, lds, qp, p.q_ss, m0, p.m_begin, p.m_end, D, vec);
  if (tid < BM) {
    m_s[tid] = FAWS_NEG_INF;
    l_s[tid] = 0.f;
    a_s[tid] = 1.f;
  }
  float o[4][8];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) o[r][c] = 0.f;
  float rs_acc = 0.f;
  const int ncd = D >> 4;  // output columns per thread in the PV step

  int hi = p.N;
  if (p.causal) {
    const int last = min(m0 + BM, p.m_end);
    hi = max(0, min(p.N, p.p_seq + last));
  }
  const int nt = (hi + BN - 1) / BN;
  const float masked_f = __uint_as_float(p.masked_bits);
  const bool part_on = p.col_partial != nullptr && qb_abs >= p.qb_first &&
                       (m0 + BM) > p.col_row_begin;

  for (int it = 0; it < nt; ++it) {
    int t = it;
    if (p.schedule == kReverse) t = nt - 1 - it;
    else if (p.schedule == kRoundRobin) t = (qb_abs + it) % nt;
    const int n0 = t * BN;
    __syncthreads();
    load_tile(Ks, lds, kp, p.k_ss, n0, 0, p.N, D, vec);
    load_tile(Vs, lds, vp, p.v_ss, n0, 0, p.N, D, vec);
    __syncthreads();

    float acc[4][4];
    tile_dot(Qs, Ks, lds, D, ty, tx, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = m0 + ty * 4 + r;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = n0 + tx + 16 * c;
        const float s = acc[r][c] * p.sm_scale;
        const bool inb = i >= p.m_begin && i < p.m_end && j < p.N;
        const bool vis = inb && (!p.causal || j <= i + p.p_seq);
        if (p.scores != nullptr && inb) {
          const int64_t off = (bh * p.M + i) * (int64_t)p.N + j;
          const float val = vis ? s : masked_f;
          if (p.scores_f32) reinterpret_cast<float*>(p.scores)[off] = val;
          else reinterpret_cast<T*>(p.scores)[off] = from_f<T>(val);
        }
        if (p.s_scratch != nullptr && inb && i >= p.split && j < p.split)
          p.s_scratch[(bh * (p.M - p.split) + (i - p.split)) * (int64_t)p.split + j] =
              vis ? s : FAWS_NEG_INF;
        Ss[(ty * 4 + r) * SLD + tx + 16 * c] = vis ? s : FAWS_NEG_INF;
      }
    }
    __syncthreads();

    if (p.col_partial != nullptr) {  // uniform branch
      if (part_on && tid < BN && n0 + tid < p.ncols_pad) {
        float sum = 0.f;
        for (int r = 0; r < BM; ++r) {
          const float val = Ss[r * SLD + tid];
          if (m0 + r >= p.col_row_begin && val != FAWS_NEG_INF) sum += val;
        }
        p.col_partial[(bh * p.n_qb_part + (qb_abs - p.qb_first)) * (int64_t)p.ncols_pad + n0 + tid] = sum;
      }
      __syncthreads();
    }

    {  // online softmax, 4 threads per row
      const int row = tid >> 2, qd = tid & 3;
      float mx = FAWS_NEG_INF;
#pragma unroll
      for (int c = 0; c < 16; ++c) mx = fmaxf(mx, Ss[row * SLD + qd + 4 * c]);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_old = m_s[row];
      const float l_old = l_s[row];
      const float m_new = fmaxf(m_old, mx);
      const float alpha = (m_new == FAWS_NEG_INF) ? 1.f : exp2f((m_old - m_new) * kLog2e);
      float psum = 0.f, rsum = 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const float s = Ss[row * SLD + qd + 4 * c];
        const bool hid = (s == FAWS_NEG_INF);
        const float pr = hid ? 0.f : exp2f((s - m_new) * kLog2e);
        rsum += hid ? 0.f : s;
        psum += pr;  // the normaliser is taken before dropout (flash.py:459-460)
        bool keep = true;
        if (p.drop.p > 0.f)
          keep = dropout_keep(p.drop, ((uint32_t)bh * (uint32_t)p.M + (uint32_t)(m0 + row)) * (uint32_t)p.N +
                                          (uint32_t)(n0 + qd + 4 * c));
        Ss[row * SLD + qd + 4 * c] = keep ? to_f(from_f<T>(pr)) : 0.f;
      }
      psum += __shfl_xor_sync(0xffffffffu, psum, 1);
      psum += __shfl_xor_sync(0xffffffffu, psum, 2);
      rs_acc += rsum;
      __syncwarp();
      if (qd == 0) {
        m_s[row] = m_new;
        l_s[row] = l_old * alpha + psum;
        a_s[row] = alpha;
      }
    }
    __syncthreads();

#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float a = a_s[ty * 4 + r];
#pragma unroll
      for (int c = 0; c < 8; ++c) o[r][c] *= a;
    }
    for (int n = 0; n < BN; ++n) {
      float pv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) pv[r] = Ss[(ty * 4 + r) * SLD + n];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c < ncd) {
          const float vv = to_f(Vs[n * lds + tx + 16 * c]);
#pragma unroll
          for (int r = 0; r < 4; ++r) o[r][c] = fmaf(pv[r], vv, o[r][c]);
        }
      }
    }
  }
  __syncthreads();

#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = m0 + ty * 4 + r;
    if (i >= p.m_begin && i < p.m_end) {
      const float l = l_s[ty * 4 + r];
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const float oscale = p.drop.p > 0.f ? p.drop.out_scale : 1.f;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < ncd) op[(int64_t)i * p.o_ss + tx + 16 * c] = from_f<T>(o[r][c] * inv * oscale);
    }
  }
  if (p.L != nullptr && tid < BM) {
    const int i = m0 + tid;
    if (i >= p.m_begin && i < p.m_end) {
      const float l = l_s[tid];
      p.L[bh * p.M + i] = l > 0.f ? m_s[tid] + logf(l) : FAWS_NEG_INF;
    }
  }
  if (p.row_sum != nullptr) {
    rs_acc += __shfl_xor_sync(0xffffffffu, rs_acc, 1);
    rs_acc += __shfl_xor_sync(0xffffffffu, rs_acc, 2);
    const int i = m0 + (tid >> 2);
    if ((tid & 3) == 0 && i >= p.m_begin && i < p.m_end) p.row_sum[bh * p.M + i] = rs_acc;
  }
  if (p.scores != nullptr) {  // key tiles the causal loop never visits: all hidden
    const int c_begin = nt * BN;
    const int width = p.N - c_begin;
    if (width > 0) {
      for (int idx = tid; idx < BM * width; idx += NT) {
        const int r = idx / width, j = c_begin + (idx - r * width);
        const int i = m0 + r;
        if (i >= p.m_begin && i < p.m_end) {
          const int64_t off = (bh * p.M + i) * (int64_t)p.N + j;
          if (p.scores_f32) reinterpret_cast<float*>(p.scores)[off] = masked_f;
          else reinterpret_cast<T*>(p.scores)[off] = from_f<T>(masked_f);
        }
      }
    }
  }
}

// Score-only operator: one CTA writes a 64 x 64 tile of q.k^T * sm_scale (attention_scores.py:56-151).
template <typename T>
__global__ void __launch_bounds__(NT) generic_scores_only_kernel(ScoresOnlyParams p, int vec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int D = p.D, lds = D + 8;
  T* Qs = reinterpret_cast<T*>(smem_raw);
  T* Ks = Qs + BM * lds;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int n_nt = (p.N + BN - 1) / BN;
  const int m0 = (blockIdx.x / n_nt) * BM, n0 = (blockIdx.x % n_nt) * BN;
  const int h = blockIdx.y, b = blockIdx.z, hk = h / (p.Hq / p.Hk);
  const T* qp = reinterpret_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
  const T* kp = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh;
  load_tile(Qs, lds, qp, p.q_ss, m0, 0, p.M, D, vec);
  load_tile(Ks, lds, kp, p.k_ss, n0, 0, p.N, D, vec);
  __syncthreads();
  float acc[4][4];
  tile_dot(Qs, Ks, lds, D, ty, tx, acc);
  const int64_t bh = (int64_t)b * p.Hq + h;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = m0 + ty * 4 + r;
    if (i >= p.M) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = n0 + tx + 16 * c;
      if (j >= p.N) continue;
      const int64_t off = (bh * p.M + i) * (int64_t)p.N + j;
      const float val = acc[r][c] * p.sm_scale;
      if (p.scores_f32) reinterpret_cast<float*>(p.scores)[off] = val;
      else reinterpret_cast<T*>(p.scores)[off] = from_f<T>(val);
    }
  }
}

// Key-major softmax column sums (the structure of total.py:50-142): a CTA owns
// 64 keys and walks the query tiles; thread c < 64 accumulates column c in a
// register in a fixed order, so there are no atomics and no partials.
template <typename T>
__global__ void __launch_bounds__(NT) generic_colsoftmax_kernel(ColSoftmaxParams p, int vec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int D = p.D, lds = D + 8;
  T* Ks = reinterpret_cast<T*>(smem_raw);
  T* Qs = Ks + BN * lds;
  float* Ss = reinterpret_cast<float*>(Qs + BM * lds);
  float* Ls = Ss + BM * SLD;

  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * BN;
  const int h = blockIdx.y, b = blockIdx.z, hk = h / p.G;
  const int ty = tid >> 4, tx = tid & 15;
  const T* qp = reinterpret_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
  const T* kp = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh;
  const int64_t bh = (int64_t)b * p.Hq + h;
  const bool from_scratch = p.s_scratch != nullptr;

  if (!from_scratch) load_tile(Ks, lds, kp, p.k_ss, n0, 0, min(p.N, p.n_end), D, vec);
  int i_lo = max(p.i_begin, p.m_begin);
  int i_start = i_lo;
  if (p.causal) i_start = max(i_start, n0 - p.p_seq);
  float colacc = 0.f;
  for (int m0 = (i_start / BM) * BM; m0 < p.m_end; m0 += BM) {
    __syncthreads();
    if (!from_scratch) load_tile(Qs, lds, qp, p.q_ss, m0, i_lo, p.m_end, D, vec);
    if (tid < BM) {
      const int i = m0 + tid;
      Ls[tid] = (i >= i_lo && i < p.m_end) ? p.L[bh * p.M + i] : FAWS_NEG_INF;
    }
    __syncthreads();
    float acc[4][4];
    if (!from_scratch) tile_dot(Qs, Ks, lds, D, ty, tx, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = m0 + ty * 4 + r;
      const float Li = Ls[ty * 4 + r];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = n0 + tx + 16 * c;
        const bool vis = i >= i_lo && i < p.m_end && j < p.n_end && j < p.N &&
                         (!p.causal || j <= i + p.p_seq) && Li != FAWS_NEG_INF;
        float s = 0.f;
        if (vis) {
          s = from_scratch
                  ? p.s_scratch[(bh * (p.M - p.split) + (i - p.split)) * (int64_t)p.split + j]
                  : acc[r][c] * p.sm_scale;
        }
        bool keep = vis;
        if (vis && p.drop.p > 0.f)
          keep = dropout_keep(p.drop, ((uint32_t)bh * (uint32_t)p.M + (uint32_t)i) * (uint32_t)p.N + (uint32_t)j);
        Ss[(ty * 4 + r) * SLD + tx + 16 * c] = keep ? exp2f((s - Li) * kLog2e) : 0.f;
      }
    }
    __syncthreads();
    if (tid < BN) {
      for (int r = 0; r < BM; ++r) colacc += Ss[r * SLD + tid];
    }
  }
  if (tid < BN && n0 + tid < p.n_end) p.out[bh * p.n_end + n0 + tid] = colacc;
}

// Second pass of the buffered cross-token variant: the scaled scores of the cross region were
// stored by the forward pass as (B,Hq,M-split,split) fp32; this kernel streams them back
// (attention_cross_token_softmax_sum.py:581-627, without atomics).  HBM-bound, so it is built to keep
// many bytes in flight: a CTA owns 128 key columns of one output head; a thread owns 4 adjacent columns
// (one 16-byte load per row) and one of 8 row groups, and issues 8 independent row loads before it
// uses any (32 threads x 8 row groups x 8 rows x 16 B = 32 KB in flight per CTA).  The exponentials are
// accumulated per thread in registers and the 8 row groups are added in a fixed order at the end.
constexpr int kScRowGroups = 8;
constexpr int kScUnroll = 8;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(32 * kScRowGroups) scratch_colsum_kernel(ColSoftmaxParams p, int heads_per_cta, int Hout) {
  __shared__ float4 red[kScRowGroups - 1][32];
  const int ct = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int j0 = blockIdx.x * 128 + ct * 4;  // first of this thread's 4 columns
  const int ho = blockIdx.y, b = blockIdx.z;
  const int i_lo = max(max(p.i_begin, p.m_begin), p.split);
  const int rows = p.M - p.split;
  const int n_lim = min(p.n_end, p.split);
  const bool vec_ok = (p.split % 4 == 0) && (j0 + 3 < n_lim);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int g = 0; g < heads_per_cta; ++g) {
    const int h = ho * heads_per_cta + g;
    const int64_t bh = (int64_t)b * p.Hq + h;
    const float* sbase = p.s_scratch + bh * (int64_t)rows * p.split;
    const float* Lbase = p.L + bh * p.M;
    // key j is visible to query i iff j <= i + p_seq: rows before i_first see none of this CTA's columns
    int i_first = i_lo;
    if (p.causal) i_first = max(i_first, (int)blockIdx.x * 128 - p.p_seq);  // signed: p_seq may exceed the tile start
    for (int i0 = i_first + rg * kScUnroll; i0 < p.m_end; i0 += kScRowGroups * kScUnroll) {
      float4 sv[kScUnroll];
      float Lv[kScUnroll];
#pragma unroll
      for (int r = 0; r < kScUnroll; ++r) {  // loads first: eight rows in flight per thread
        const int i = i0 + r;
        sv[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        Lv[r] = FAWS_NEG_INF;
        if (i < p.m_end) {
          const float* rowp = sbase + (int64_t)(i - p.split) * p.split + j0;
          if (vec_ok) {
            sv[r] = __ldcs(reinterpret_cast<const float4*>(rowp));  // streamed once
          } else {
            if (j0 < n_lim) sv[r].x = rowp[0];
            if (j0 + 1 < n_lim) sv[r].y = rowp[1];
            if (j0 + 2 < n_lim) sv[r].z = rowp[2];
            if (j0 + 3 < n_lim) sv[r].w = rowp[3];
          }
          Lv[r] = Lbase[i];
        }
      }
#pragma unroll
      for (int r = 0; r < kScUnroll; ++r) {
        const int i = i0 + r;
        if (Lv[r] == FAWS_NEG_INF) continue;  // row outside the window, or a row without a visible key
        const float nl = -Lv[r] * kLog2e;
        const int jmax = p.causal ? i + p.p_seq : 0x7fffffff;  // last visible key of this row
        acc.x += (j0 <= jmax) ? ex2_approx(fmaf(sv[r].x, kLog2e, nl)) : 0.f;
        acc.y += (j0 + 1 <= jmax) ? ex2_approx(fmaf(sv[r].y, kLog2e, nl)) : 0.f;
        acc.z += (j0 + 2 <= jmax) ? ex2_approx(fmaf(sv[r].z, kLog2e, nl)) : 0.f;
        acc.w += (j0 + 3 <= jmax) ? ex2_approx(fmaf(sv[r].w, kLog2e, nl)) : 0.f;
      }
    }
  }
  if (rg > 0) red[rg - 1][ct] = acc;
  __syncthreads();
  if (rg == 0) {
#pragma unroll
    for (int w = 0; w < kScRowGroups - 1; ++w) {  // row groups 0, 1, 2, ... in this order
      const float4 o = red[w][ct];
      acc.x += o.x; acc.y += o.y; acc.z += o.z; acc.w += o.w;
    }
    float* dst = p.out + ((int64_t)b * Hout + ho) * p.n_end + j0;
    if (j0 < n_lim) dst[0] = acc.x;
    if (j0 + 1 < n_lim) dst[1] = acc.y;
    if (j0 + 2 < n_lim) dst[2] = acc.z;
    if (j0 + 3 < n_lim) dst[3] = acc.w;
  }
}

// out[b,ho,j] = sum over the group's heads (or the single head) and over the
// query blocks that visited column j, in a fixed order.
__global__ void reduce_partials_kernel(ReducePartialParams p) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.n_end) return;
  const int ho = blockIdx.y, b = blockIdx.z;
  const int h0 = p.per_q_head ? ho : ho * p.G;
  const int nh = p.per_q_head ? 1 : p.G;
  const int Hout = p.per_q_head ? p.Hq : p.Hk;
  const int tile_start = (j / p.block_n) * p.block_n;
  float sum = 0.f;
  for (int g = 0; g < nh; ++g) {
    const float* base = p.partial + ((int64_t)(b * p.Hq + h0 + g) * p.n_qb_part) * p.ncols_pad;
    for (int qb = 0; qb < p.n_qb_part; ++qb) {
      if (p.causal) {
        const int last = min((p.qb_first + qb + 1) * p.block_m, p.m_end);
        const int hi = min(p.N, p.p_seq + last);
        if (tile_start >= hi) continue;  // the forward kernel never visited this key tile
      }
      sum += base[(int64_t)qb * p.ncols_pad + j];
    }
  }
  p.out[((int64_t)b * Hout + ho) * p.n_end + j] = sum;
}

// Column sums with the linear part: a block owns one 128-wide key tile t of one output head.
// out[j] = sm_scale * k_j . V(t) + sum_h sum_{qb hooked} partial[h][qb][j], where V(t) is the sum of
// qsum[h][qb] over the output head's query heads and the query tiles for which col_tile_linear(qb, t)
// holds: one contiguous range of tiles, as is the range of those that saw the key tile at all.
// One key row of D / 8 lanes at a time, 16 bytes a lane, all of a warp's rows in flight before V is known; the loads
// of V and of the partial rows, (query head, query tile) pairs, are dealt to four thread groups, whose sums are added
// in the fixed order 0..3.
// Bound by the loads' latency and L2 (fp16 B1 H32 S8192 D128 causal: 29 us; 88 us with the K tile staged in shared
// memory, a dot product per query head and every query tile tested by predicate, which was bound by issue).  Dealing
// pairs and not the tiles of one head after another keeps eight loads in flight where a head has few tiles (fp16 B1
// Hq28 Hk4 S128 D64 full, whole operator: 9.6 and 12.6 us).
constexpr int kLinGroups = 4;

// Sum of the (query head g, query tile r) entries at base + g * head_stride + r * tile_stride, g < nh, r < len, that fall
// to thread group tg.
__device__ __forceinline__ float sum_dealt_pairs(const float* base, int64_t head_stride, int tile_stride, int nh, int len,
                                                 int tg) {
  if (len <= 0) return 0.f;
  int r = tg % len, left = (nh * len - tg + kLinGroups - 1) / kLinGroups;
  const float* at = base + (tg / len) * head_stride + r * tile_stride;
  const int64_t wrap = head_stride - (int64_t)len * tile_stride;
  auto next = [&] {
    const float x = *at;
    at += kLinGroups * tile_stride;
    r += kLinGroups;
    while (r >= len) {
      r -= len;
      at += wrap;
    }
    return x;
  };
  float s = 0.f;
  for (; left > 0; left -= 8) {  // (the last few together as well: one after the other each would wait for its load)
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = e < left ? next() : 0.f;
    s += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  return s;
}

// CTAS: resident per SM.  Two leave 64 registers, and no spill code (24 / 44 bytes of it in fp16, 36 / 108 in bf16 with three):
// bf16 B16 H4 S200 D64 full 15.9 -> 14.1 us, B6 H8 S174 D64 causal 12.4 -> 11.7, whole operator.  raw_col_sums chooses.
template <typename T, int CTAS>
__global__ void __launch_bounds__(128 * kLinGroups, CTAS) reduce_colsum_lin_kernel(ReducePartialParams p) {
  constexpr int kRowsPerWarp = 128 / (4 * kLinGroups);
  __shared__ __align__(16) float V[kLinGroups][128];
  __shared__ float part[kLinGroups][128];
  __shared__ float lin[128];
  const int t = blockIdx.x, tid = threadIdx.x & 127, tg = threadIdx.x >> 7;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = t * 128 + tid;
  const int ho = blockIdx.y, b = blockIdx.z;
  const int h0 = p.per_q_head ? ho : ho * p.G;
  const int nh = p.per_q_head ? 1 : p.G;
  const int Hout = p.per_q_head ? p.Hq : p.Hk;
  const int hk = h0 / p.G;

  // this warp's key rows (the forward kernel ran on tcgen05: rows are 16-byte aligned, D / 8 a power of two)
  const int lpr = p.D >> 3, rows_at_once = 32 / lpr;  // lanes per row; rows of one warp-wide load
  const int sub = lane & (lpr - 1), row0 = warp * kRowsPerWarp + lane / lpr;
  const T* kbase = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh + 8 * sub;
  uint4 kr[kRowsPerWarp / 2];  // (at D = 128 two rows a load; fewer loads below)
#pragma unroll
  for (int x = 0; x < kRowsPerWarp / 2; ++x) {
    const int jr = t * 128 + row0 + x * rows_at_once;
    kr[x] = make_uint4(0u, 0u, 0u, 0u);
    if (x * rows_at_once < kRowsPerWarp && jr < p.N)
      kr[x] = *reinterpret_cast<const uint4*>(kbase + (int64_t)jr * p.k_ss);
  }

  ptx::griddep_wait();  // the sums and partial rows come from the forward pass, which this launch may overlap; k does not
  // linear query tiles [lin_lo, lin_hi) and, among [seen_lo, seen_hi), the others, which left partial rows:
  // col_tile_linear and the forward kernel's visits, as ranges
  int lin_lo = (p.row_lo + 127) / 128, lin_hi = p.m_end / 128;
  int seen_lo = p.qb_first;
  const int seen_hi = p.qb_first + p.n_qb_part;
  if (p.causal) {
    lin_lo = max(lin_lo, (max(0, t * 128 + 127 - p.p_seq) + 127) / 128);
    seen_lo = max(seen_lo, max(0, t * 128 - p.p_seq) / 128);  // first tile whose last row reaches the key tile
    if (t * 128 >= p.p_seq + p.m_end) seen_lo = seen_hi;
  }
  if (t * 128 + 128 > p.N) lin_hi = 0;
  lin_hi = max(lin_lo, lin_hi);

  float v = 0.f;
  if (tid < p.D)
    v = sum_dealt_pairs(p.qsum + (((int64_t)b * p.Hq + h0) * p.nqb_total + lin_lo) * 128 + tid, (int64_t)p.nqb_total * 128,
                        128, nh, lin_hi - lin_lo, tg);
  float p0 = 0.f;
  if (j < p.n_end) {
    const float* base = p.partial + ((int64_t)(b * p.Hq + h0) * p.n_qb_part - p.qb_first) * p.ncols_pad + j;
    const int64_t head = (int64_t)p.n_qb_part * p.ncols_pad;
    const int first_end = min(lin_lo, seen_hi), second = max(seen_lo, lin_hi);  // seen tiles before and behind the linear ones
    p0 = sum_dealt_pairs(base + (int64_t)seen_lo * p.ncols_pad, head, p.ncols_pad, nh, first_end - seen_lo, tg) +
         sum_dealt_pairs(base + (int64_t)second * p.ncols_pad, head, p.ncols_pad, nh, seen_hi - second, tg);
  }
  V[tg][tid] = v;
  part[tg][tid] = p0;
  __syncthreads();
  if (tg == 0) V[0][tid] = (V[0][tid] + V[1][tid]) + (V[2][tid] + V[3][tid]);
  __syncthreads();
  const float4 va = *reinterpret_cast<const float4*>(&V[0][8 * sub]), vb = *reinterpret_cast<const float4*>(&V[0][8 * sub + 4]);
#pragma unroll
  for (int x = 0; x < kRowsPerWarp / 2; ++x) {
    if (x * rows_at_once >= kRowsPerWarp) break;
    const T* k8 = reinterpret_cast<const T*>(&kr[x]);
    float d = to_f(k8[0]) * va.x;
    d = fmaf(to_f(k8[1]), va.y, d);
    d = fmaf(to_f(k8[2]), va.z, d);
    d = fmaf(to_f(k8[3]), va.w, d);
    float d2 = to_f(k8[4]) * vb.x;
    d2 = fmaf(to_f(k8[5]), vb.y, d2);
    d2 = fmaf(to_f(k8[6]), vb.z, d2);
    d2 = fmaf(to_f(k8[7]), vb.w, d2);
    d += d2;
    for (int w = lpr >> 1; w > 0; w >>= 1) d += __shfl_xor_sync(0xffffffffu, d, w);
    const int row = row0 + x * rows_at_once;
    if (sub == 0 && row < (warp + 1) * kRowsPerWarp) lin[row] = d;
  }
  __syncthreads();
  if (tg == 0 && j < p.n_end)
    p.out[((int64_t)b * Hout + ho) * p.n_end + j] =
        j < p.N ? fmaf(p.sm_scale, lin[tid], (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid])) : 0.f;
}
static_assert(kLinGroups == 4, "the sums of the thread groups are written out");

__global__ void group_sum_kernel(const float* in, float* out, int Hk, int G, int len) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= len) return;
  const int hk = blockIdx.y, b = blockIdx.z;
  float sum = 0.f;
  for (int g = 0; g < G; ++g) sum += in[((int64_t)(b * Hk + hk) * G + g) * len + j];
  out[((int64_t)b * Hk + hk) * len + j] = sum;
}

__global__ void reduce_ranks_kernel(const float* parts, int n_ranks, int64_t count, float* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  float sum = 0.f;
  for (int r = 0; r < n_ranks; ++r) sum += parts[(int64_t)r * count + i];
  out[i] = sum;
}

// Split-KV combine (the role of _fwd_combine_kv_splits, split_kv.py:163-227): every key range s left
// a normalised partial result o_s and its log-normaliser L_s; out = sum_s exp(L_s - L) o_s with
// L = log sum_s exp(L_s), added in the order s = 0, 1, ...  One warp per query row.
// A few hundred rows of latency: the launch overlaps the forward pass (programmatic dependent launch; it waits
// before its first load), a lane owns 2 or 4 neighbouring dims and has the loads of four ranges in flight.
// One-row decoding, bf16 Hq32 Hk8 N9001 D128: B8 59.6 -> 57.1 us, B1 20.7 -> 14.4 us against a plain launch of
// scalar loads.
template <typename T, int V>
__device__ __forceinline__ void combine_row(const float* o_part, const float* Ls, int64_t M, T* orow,
                                            int64_t s_step, int d, float mx, float inv, int S) {
  static_assert(V == 2 || V == 4, "dims of a lane");
  float acc[V];
#pragma unroll
  for (int x = 0; x < V; ++x) acc[x] = 0.f;
  for (int s0 = 0; s0 < S; s0 += 4) {
    __align__(16) float w[4][V];
    float l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      l[e] = FAWS_NEG_INF;
      if (s0 + e < S) {
        l[e] = Ls[(int64_t)(s0 + e) * M];
        const float* src = o_part + (int64_t)(s0 + e) * s_step + d;
        if constexpr (V == 4) *reinterpret_cast<float4*>(w[e]) = *reinterpret_cast<const float4*>(src);
        else *reinterpret_cast<float2*>(w[e]) = *reinterpret_cast<const float2*>(src);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (l[e] == FAWS_NEG_INF) continue;
      const float f = exp2f((l[e] - mx) * kLog2e);
#pragma unroll
      for (int x = 0; x < V; ++x) acc[x] += f * w[e][x];
    }
  }
  __align__(8) T res[V];  // (rows of 16-byte alignment: the forward kernel's condition)
#pragma unroll
  for (int x = 0; x < V; ++x) res[x] = from_f<T>(acc[x] * inv);
  if constexpr (V == 4) *reinterpret_cast<uint2*>(orow + d) = *reinterpret_cast<const uint2*>(res);
  else *reinterpret_cast<uint32_t*>(orow + d) = *reinterpret_cast<const uint32_t*>(res);
}

template <typename T>
__global__ void combine_splits_kernel(const float* o_part, const float* L_part, T* out,
                                      int64_t o_sb, int64_t o_sh, int64_t o_ss, float* L, int B, int Hq, int M, int D,
                                      int S) {
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= (int64_t)B * Hq * M) return;
  const int i = (int)(row % M);
  const int64_t bh = row / M;
  const int h = (int)(bh % Hq), b = (int)(bh / Hq);
  const float* Ls = L_part + bh * S * M + i;
  float mx = FAWS_NEG_INF;
  for (int s = lane; s < S; s += 32) mx = fmaxf(mx, Ls[(int64_t)s * M]);
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
  float den = 0.f;
  for (int s = 0; s < S; ++s) {
    const float l = Ls[(int64_t)s * M];
    den += (l == FAWS_NEG_INF) ? 0.f : exp2f((l - mx) * kLog2e);
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  T* orow = out + b * o_sb + h * o_sh + (int64_t)i * o_ss;
  const float* part = o_part + (bh * S * M + i) * (int64_t)D;
  const int64_t s_step = (int64_t)M * D;
  if (D == 128) combine_row<T, 4>(part, Ls, M, orow, s_step, lane * 4, mx, inv, S);
  else if (lane * 2 < D) combine_row<T, 2>(part, Ls, M, orow, s_step, lane * 2, mx, inv, S);
  if (L != nullptr && lane == 0) L[row] = den > 0.f ? mx + logf(den) : FAWS_NEG_INF;
}

size_t fwd_smem(int D) { return (size_t)(3 * 64 * (D + 8)) * 2 + (size_t)(BM * SLD + 3 * BM) * 4; }
size_t cs_smem(int D) { return (size_t)(2 * 64 * (D + 8)) * 2 + (size_t)(BM * SLD + BM) * 4; }

template <typename K>
cudaError_t set_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

bool aligned16(const void* ptr, int64_t a, int64_t b, int64_t c) {
  return (reinterpret_cast<uintptr_t>(ptr) % 16 == 0) && a % 8 == 0 && b % 8 == 0 && c % 8 == 0;
}

}  // namespace

cudaError_t launch_generic_fwd(const FwdParams& p, int dtype, cudaStream_t s) {
  const int vec = aligned16(p.q, p.q_sb, p.q_sh, p.q_ss) && aligned16(p.k, p.k_sb, p.k_sh, p.k_ss) &&
                  aligned16(p.v, p.v_sb, p.v_sh, p.v_ss);
  const int nqb = (p.m_end + BM - 1) / BM - p.m_begin / BM;
  if (nqb <= 0) return cudaSuccess;
  dim3 grid(nqb, p.Hq, p.B);
  const size_t smem = fwd_smem(p.D);
  cudaError_t e;
  if (dtype == FAWS_FP16) {
    if ((e = set_smem(generic_fwd_kernel<__half>, smem)) != cudaSuccess) return e;
    generic_fwd_kernel<__half><<<grid, NT, smem, s>>>(p, vec);
  } else {
    if ((e = set_smem(generic_fwd_kernel<__nv_bfloat16>, smem)) != cudaSuccess) return e;
    generic_fwd_kernel<__nv_bfloat16><<<grid, NT, smem, s>>>(p, vec);
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_generic_scores_only(const ScoresOnlyParams& p, int dtype, cudaStream_t s) {
  const int vec = aligned16(p.q, p.q_sb, p.q_sh, p.q_ss) && aligned16(p.k, p.k_sb, p.k_sh, p.k_ss);
  const long long tiles = (long long)((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  if (tiles <= 0 || tiles > 0x7fffffffLL) return tiles <= 0 ? cudaSuccess : cudaErrorInvalidValue;
  dim3 grid((unsigned)tiles, p.Hq, p.B);
  const size_t smem = (size_t)(2 * 64 * (p.D + 8)) * 2;
  if (dtype == FAWS_FP16) generic_scores_only_kernel<__half><<<grid, NT, smem, s>>>(p, vec);
  else generic_scores_only_kernel<__nv_bfloat16><<<grid, NT, smem, s>>>(p, vec);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_generic_colsoftmax(const ColSoftmaxParams& p, int dtype, cudaStream_t s) {
  const int vec = aligned16(p.q, p.q_sb, p.q_sh, p.q_ss) && aligned16(p.k, p.k_sb, p.k_sh, p.k_ss);
  if (p.n_end <= 0) return cudaSuccess;
  dim3 grid((p.n_end + BN - 1) / BN, p.Hq, p.B);
  const size_t smem = cs_smem(p.D);
  cudaError_t e;
  if (dtype == FAWS_FP16) {
    if ((e = set_smem(generic_colsoftmax_kernel<__half>, smem)) != cudaSuccess) return e;
    generic_colsoftmax_kernel<__half><<<grid, NT, smem, s>>>(p, vec);
  } else {
    if ((e = set_smem(generic_colsoftmax_kernel<__nv_bfloat16>, smem)) != cudaSuccess) return e;
    generic_colsoftmax_kernel<__nv_bfloat16><<<grid, NT, smem, s>>>(p, vec);
  }
  count_launch();
  return cudaGetLastError();
}

// group_sum != 0: p.out is (B,Hk,n_end) and a CTA adds the G heads of its kv head; else (B,Hq,n_end).
cudaError_t launch_scratch_colsum(const ColSoftmaxParams& p, int group_sum, cudaStream_t s) {
  if (p.n_end <= 0) return cudaSuccess;
  const int hpc = group_sum ? p.G : 1;
  const int Hout = p.Hq / hpc;
  dim3 grid((p.n_end + 127) / 128, Hout, p.B);
  scratch_colsum_kernel<<<grid, 32 * kScRowGroups, 0, s>>>(p, hpc, Hout);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_reduce_partials(const ReducePartialParams& p, int dtype, cudaStream_t s) {
  if (p.n_end <= 0) return cudaSuccess;
  if (p.lin) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((p.n_end + 127) / 128, p.per_q_head ? p.Hq : p.Hk, p.B);
    cfg.blockDim = dim3(128 * kLinGroups, 1, 1);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.overlap;
    const auto kernel =
        dtype == FAWS_FP16 ? (p.resident == 3 ? reduce_colsum_lin_kernel<__half, 3> : reduce_colsum_lin_kernel<__half, 2>)
                           : (p.resident == 3 ? reduce_colsum_lin_kernel<__nv_bfloat16, 3> : reduce_colsum_lin_kernel<__nv_bfloat16, 2>);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
    if (e != cudaSuccess) return e;
  } else {
    dim3 grid((p.n_end + 255) / 256, p.per_q_head ? p.Hq : p.Hk, p.B);
    reduce_partials_kernel<<<grid, 256, 0, s>>>(p);
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_group_sum(const float* in, float* out, int B, int Hk, int G, int len,
                             cudaStream_t s) {
  if (len <= 0) return cudaSuccess;
  dim3 grid((len + 255) / 256, Hk, B);
  group_sum_kernel<<<grid, 256, 0, s>>>(in, out, Hk, G, len);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_combine_splits(const float* o_part, const float* L_part, void* out, int64_t o_sb, int64_t o_sh,
                                  int64_t o_ss, float* L, int B, int Hq, int M, int D, int n_splits, int dtype,
                                  cudaStream_t s) {
  const int64_t rows = (int64_t)B * Hq * M;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((rows + 3) / 4), 1, 1);
  cfg.blockDim = dim3(128, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e;
  if (dtype == FAWS_FP16)
    e = cudaLaunchKernelEx(&cfg, combine_splits_kernel<__half>, o_part, L_part, static_cast<__half*>(out), o_sb, o_sh, o_ss, L, B, Hq, M, D, n_splits);
  else
    e = cudaLaunchKernelEx(&cfg, combine_splits_kernel<__nv_bfloat16>, o_part, L_part, static_cast<__nv_bfloat16*>(out), o_sb, o_sh, o_ss, L, B, Hq, M, D, n_splits);
  if (e != cudaSuccess) return e;
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_reduce_ranks(const float* parts, int n_ranks, int64_t count, float* out,
                                cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  reduce_ranks_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(parts, n_ranks, count, out);
  count_launch();
  return cudaGetLastError();
}

}  // namespace faws
