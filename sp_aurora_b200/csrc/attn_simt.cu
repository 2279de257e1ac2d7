// CUDA-core (fp32 FMA) flash-attention forward and backward.
//
// This is the path fp32 tensors take: every product and accumulation is fp32,
// so results agree with the reference's fp32 PyTorch math
// (sp_aurora/intel_flash_attn.py:95-126) to ~1e-6, inside the 1e-4 budget that
// tensor-core bf16/tf32 products cannot meet. It also accepts bf16/fp16 data
// (converted on load) so tests can cross-check the tcgen05 kernels on the GPU.
//
// Bound by the fp32 FMA pipes. A CTA owns 64 rows and streams 64-row tiles; its threads are a
// grid of 16 columns (tx) by 64/R rows (ty), and a thread owns R rows {ty + i*64/R} by 4 columns
// {tx + 16*j} of a score tile, so one float4 of each operand feeds 4*R*4 multiply-adds. The 16
// threads of a row are half a warp: row maxima are shuffles, and the probabilities that become
// the next product's operand go through shared memory rows that only their own warp reads (no
// block barrier). Tile rows are padded by four floats, which puts the 16 rows a half-warp reads
// at once in different banks. B=2, S=1024, 32 heads, D=64, causal, fp32: forward + backward
// 2486 -> 1154 us against four threads per row with one float4 load per four multiply-adds; the
// three kernels take 293, 368 and 496 us, 31, 37 and 37 TFLOP/s of executed tiles of the 73 that an
// FMA-only loop reaches.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "spa_internal.h"
#include "tc05.cuh"

namespace spa {
namespace {

constexpr int kRows = 64;        // rows per CTA
constexpr int kTile = 64;        // rows of the streamed operand per shared-memory tile
constexpr int kCols = kTile / 16;   // score columns per thread
constexpr int kLdP = kTile + 4;  // row stride of the probability tile

template <typename T>
__device__ __forceinline__ float4 load4(const T* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
template <>
__device__ __forceinline__ float4 load4<__half>(const __half* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const __half2 a = *reinterpret_cast<const __half2*>(&u.x);
  const __half2 b = *reinterpret_cast<const __half2*>(&u.y);
  const float2 fa = __half22float2(a), fb = __half22float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, float4 v);
template <>
__device__ __forceinline__ void store4<float>(float* p, float4 v) {
  *reinterpret_cast<float4*>(p) = v;
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a);
  u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}
template <>
__device__ __forceinline__ void store4<__half>(__half* p, float4 v) {
  __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a);
  u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// Shape of a kernel instance: R rows per thread.
template <int D, int R>
struct SimtShape {
  static constexpr int kTy = kRows / R;          // rows of the thread grid
  static constexpr int kThreads = 16 * kTy;
  static constexpr int kLd = D + 4;              // row stride of an operand tile
  static constexpr int kTileFloats = kTile * kLd;
  static constexpr int kNC = D / 16;             // head-dim columns per thread
  static constexpr int kVec = kNC < 4 ? kNC : 4; // of which this many are adjacent
  // i-th head-dim column of thread column tx
  __device__ static __forceinline__ int col(int tx, int i) { return (i / kVec) * 64 + tx * kVec + i % kVec; }
};

// Cooperative load of kTile rows x D (element type T, row stride `stride` elements) into an fp32
// operand tile; rows outside [first, end) are filled with zeros. The streamed operands are cut to
// the rows that the block's own rows see or are seen by: a masked weight is 0, but 0 * Inf is not.
template <int D, int R, typename T>
__device__ __forceinline__ void load_tile(float* dst, const T* src, int64_t stride, int end, int first = 0) {
  using S = SimtShape<D, R>;
  constexpr int kVecs = D / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < kTile * kVecs; i += S::kThreads) {
    const int r = i / kVecs, f = i % kVecs;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r >= first && r < end) v = load4<T>(src + (int64_t)r * stride + 4 * f);
    *reinterpret_cast<float4*>(dst + r * S::kLd + 4 * f) = v;
  }
}

// acc[i][j] = row (ty + i*kTy) of a . row (tx + 16*j) of b. The even and the odd elements are
// summed apart (the packed multiply-add works on pairs) and joined every 32 elements, at D = 32
// every 16, so that no chain is longer than that of four threads per row, D / 4. Joined at the end
// only, results were up to 14 % (D = 128), 4 % (D = 64) and 20 % (scores at D = 32) further from
// 64-bit ones; joining costs 2 % of the time (1127 -> 1151 us for the call above), at D = 32 up to 7 %
// (1024 rows of 2 x 8 heads 309 -> 322 us, 3000 of 8 in bf16 927 -> 990, 3000 of 32 2725 -> 2703).
template <int D, int R>
__device__ __forceinline__ void dot_tiles(float (&acc)[R][kCols], const float* a, const float* b, int ty, int tx) {
  using S = SimtShape<D, R>;
  constexpr int kJoin = D == 32 ? 16 : 32;
#pragma unroll
  for (int f0 = 0; f0 < D; f0 += kJoin) {
    float2 p[R][kCols];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < kCols; ++j) p[i][j] = make_float2(0.f, 0.f);
#pragma unroll(kJoin / 16)   // two steps at D = 32 spill: 322 -> 324, 990 -> 954, 2703 -> 2773 us
    for (int f = f0; f < f0 + kJoin; f += 4) {
      float4 bv[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) bv[j] = *reinterpret_cast<const float4*>(b + (tx + 16 * j) * S::kLd + f);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 av = *reinterpret_cast<const float4*>(a + (ty + i * S::kTy) * S::kLd + f);
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          fma2(p[i][j].x, p[i][j].y, av.x, av.y, bv[j].x, bv[j].y, p[i][j].x, p[i][j].y);
          fma2(p[i][j].x, p[i][j].y, av.z, av.w, bv[j].z, bv[j].w, p[i][j].x, p[i][j].y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[i][j] = f0 == 0 ? p[i][j].x + p[i][j].y : acc[i][j] + (p[i][j].x + p[i][j].y);
  }
}

// The thread's part of a score tile -> the probability tile (read back by the same warp).
template <int D, int R>
__device__ __forceinline__ void put_scores(float* p_s, const float (&v)[R][kCols], int ty, int tx) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < kCols; ++j) p_s[(ty + i * SimtShape<D, R>::kTy) * kLdP + tx + 16 * j] = v[i][j];
}

// o[i][c] += sum over the tile's kTile rows k of p[ty + i*kTy][k] * b[k][col(c)].
template <int D, int R>
__device__ __forceinline__ void add_product(float (&o)[R][D / 16], const float* p_s, const float* b, int ty, int tx) {
  using S = SimtShape<D, R>;
#pragma unroll 2
  for (int k = 0; k < kTile; k += 4) {
    float4 pv[R];
#pragma unroll
    for (int i = 0; i < R; ++i) pv[i] = *reinterpret_cast<const float4*>(p_s + (ty + i * S::kTy) * kLdP + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float bv[S::kNC];
      const float* br = b + (k + kk) * S::kLd;
#pragma unroll
      for (int c = 0; c < S::kNC; c += S::kVec) {
        if constexpr (S::kVec == 4) {
          const float4 x = *reinterpret_cast<const float4*>(br + S::col(tx, c));
          bv[c] = x.x; bv[c + 1] = x.y; bv[c + 2] = x.z; bv[c + 3] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(br + S::col(tx, c));
          bv[c] = x.x; bv[c + 1] = x.y;
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float pe = kk == 0 ? pv[i].x : kk == 1 ? pv[i].y : kk == 2 ? pv[i].z : pv[i].w;
#pragma unroll
        for (int c = 0; c < S::kNC; ++c) o[i][c] = fmaf(pe, bv[c], o[i][c]);
      }
    }
  }
}

// Adjacent head-dim columns of a row: 2 or 4 elements.
template <int V, typename T>
__device__ __forceinline__ void load_cols(float* v, const T* p) {
  if constexpr (V == 4) {
    const float4 x = load4<T>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
    v[0] = static_cast<float>(p[0]);
    v[1] = static_cast<float>(p[1]);
  }
}
template <int V, typename T>
__device__ __forceinline__ void store_cols(T* p, const float* v) {
  if constexpr (V == 4) {
    store4<T>(p, make_float4(v[0], v[1], v[2], v[3]));
  } else {
    p[0] = static_cast<T>(v[0]);
    p[1] = static_cast<T>(v[1]);
  }
}

// Row tile, head and batch of a CTA: heads fastest, tiles slowest, so that under a causal mask
// all the long tiles start first (`last_first`: the last rows are the long ones).
__device__ __forceinline__ void decode_cta(int rows, int heads, int batch, bool last_first, int& r0, int& h, int& b) {
  int w = blockIdx.x;
  h = w % heads;
  w /= heads;
  b = w % batch;
  w /= batch;
  const int tiles = (rows + kRows - 1) / kRows;
  r0 = (last_first ? tiles - 1 - w : w) * kRows;
}

struct SimtFwdParams {
  const void *q, *k, *v;
  int64_t q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh;
  void* out;
  int64_t o_sb, o_ss, o_sh;
  float* out_acc;
  float* lse;
  int64_t lse_sb, lse_sh;
  int B, Sq, Sk, Hq, Hkv, causal, causal_off, merge_prev;
  float scale;
};

template <int D, typename T, int R>
__global__ void __launch_bounds__(SimtShape<D, R>::kThreads)
attn_fwd_simt_kernel(const SimtFwdParams p) {
  using S = SimtShape<D, R>;
  extern __shared__ __align__(16) float simt_smem[];
  float* q_s = simt_smem;
  float* k_s = q_s + S::kTileFloats;
  float* v_s = k_s + S::kTileFloats;
  float* p_s = v_s + S::kTileFloats;
  int r0, h, b;
  decode_cta(p.Sq, p.Hq, p.B, p.causal, r0, h, b);
  const int hk = h / (p.Hq / p.Hkv);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_tile<D, R, T>(q_s, reinterpret_cast<const T*>(p.q) + b * p.q_sb + (int64_t)r0 * p.q_ss + h * p.q_sh,
                     p.q_ss, p.Sq - r0);
  float o[R][S::kNC], m[R], l[R];   // l: this thread's columns only, joined at the end
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < S::kNC; ++c) o[i][c] = 0.f;
  }

  int n_keys = p.Sk;
  if (p.causal) {
    const long long last = (long long)min(r0 + kRows, p.Sq) - 1 + p.causal_off;
    n_keys = (int)max(0ll, min((long long)p.Sk, last + 1));
  }
  const T* kbase = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh;
  const T* vbase = reinterpret_cast<const T*>(p.v) + b * p.v_sb + hk * p.v_sh;

  for (int k0 = 0; k0 < n_keys; k0 += kTile) {
    __syncthreads();
    load_tile<D, R, T>(k_s, kbase + (int64_t)k0 * p.k_ss, p.k_ss, n_keys - k0);
    load_tile<D, R, T>(v_s, vbase + (int64_t)k0 * p.v_ss, p.v_ss, n_keys - k0);
    __syncthreads();
    float s[R][kCols], alpha[R];
    dot_tiles<D, R>(s, q_s, k_s, ty, tx);
    const bool need_mask = k0 + kTile > p.Sk || (p.causal && (long long)k0 + kTile - 1 > (long long)r0 + p.causal_off);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < kCols; ++j) {
        float x = s[i][j] * p.scale;
        if (need_mask) {
          const int kidx = k0 + tx + 16 * j;
          const long long my_last = p.causal ? (long long)r0 + ty + i * S::kTy + p.causal_off : (long long)p.Sk;
          if (kidx >= p.Sk || (long long)kidx > my_last) x = -INFINITY;
        }
        s[i][j] = x;
        mx = fmaxf(mx, x);
      }
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      const float m_new = fmaxf(m[i], mx);
      const float m_eff = m_new == -INFINITY ? 0.f : m_new;   // nothing visible yet: all p = 0
      alpha[i] = expf(m[i] - m_eff);                          // m = -inf -> 0
      float psum = 0.f;
#pragma unroll
      for (int j = 0; j < kCols; ++j) {
        s[i][j] = expf(s[i][j] - m_eff);
        psum += s[i][j];
      }
      l[i] = l[i] * alpha[i] + psum;
      m[i] = m_new;
    }
    put_scores<D, R>(p_s, s, ty, tx);
    __syncwarp();
    float tile[R][S::kNC];   // summed apart from the running output: shorter chains of roundings
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < S::kNC; ++c) tile[i][c] = 0.f;
    add_product<D, R>(tile, p_s, v_s, ty, tx);
    // A row that has seen no key yet keeps its zeros: its weights are 0, but 0 * Inf in V is not.
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < S::kNC; ++c)
        o[i][c] = m[i] == -INFINITY ? 0.f : fmaf(o[i][c], alpha[i], tile[i][c]);
  }

#pragma unroll
  for (int i = 0; i < R; ++i) {
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], d);
    const int row = r0 + ty + i * S::kTy;
    const size_t lse_idx = (size_t)b * p.lse_sb + (size_t)h * p.lse_sh + row;
    // one thread of the row reads the old lse, and only that thread writes the new one
    float lse_old = p.merge_prev && tx == 0 && row < p.Sq ? p.lse[lse_idx] : 0.f;
    lse_old = __shfl_sync(0xffffffffu, lse_old, threadIdx.x & 16);
    if (row >= p.Sq) continue;
    const bool have = l[i] > 0.f;
    const float inv_l = have ? 1.f / l[i] : l[i];   // 0 without a key, NaN stays NaN
    const float lse_blk = have ? m[i] + logf(l[i]) : -INFINITY;
    float w_old = 0.f, w_blk = have ? 1.f : 0.f, lse_new = lse_blk;
    if (p.merge_prev) {
      const float mx = fmaxf(lse_old, lse_blk);
      if (mx == -INFINITY) {
        w_blk = 0.f;
        lse_new = -INFINITY;
      } else {
        const float e_old = expf(lse_old - mx), e_blk = expf(lse_blk - mx);
        const float sum = e_old + e_blk;
        lse_new = mx + logf(sum);
        w_old = e_old / sum;
        w_blk = e_blk / sum;
      }
    }
    if (tx == 0) p.lse[lse_idx] = lse_new;
    float* acc_row = p.out_acc ? p.out_acc + (((size_t)b * p.Sq + row) * p.Hq + h) * D : nullptr;
    T* out_row = p.out ? reinterpret_cast<T*>(p.out) + b * p.o_sb + (int64_t)row * p.o_ss + h * p.o_sh : nullptr;
    const float osc = inv_l * w_blk;
#pragma unroll
    for (int c = 0; c < S::kNC; c += S::kVec) {
      const int e = S::col(tx, c);
      float a[S::kVec];
#pragma unroll
      for (int u = 0; u < S::kVec; ++u) a[u] = o[i][c + u] * osc;
      if (p.merge_prev) {
        float old[S::kVec];
        load_cols<S::kVec, float>(old, acc_row + e);
#pragma unroll
        for (int u = 0; u < S::kVec; ++u) a[u] = fmaf(w_old, old[u], a[u]);
      }
      if (acc_row) store_cols<S::kVec, float>(acc_row + e, a);
      if (out_row) store_cols<S::kVec, T>(out_row + e, a);
    }
  }
}

struct SimtBwdParams {
  const void *q, *k, *v, *dout;
  int64_t q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, do_sb, do_ss, do_sh;
  const float* lse;
  const float* delta;
  int64_t lse_sb, lse_sh;
  float* dq_acc;
  void* dq;
  int64_t dq_sb, dq_ss, dq_sh;
  int dq_overwrite;
  void* dk;
  void* dv;
  int64_t dkv_sb, dkv_ss, dkv_sh;
  int dkv_fp32, dkv_accumulate;
  int B, Sq, Sk, Hq, Hkv, causal, causal_off;
  float scale;
};

// dQ: query rows stationary, keys streamed. The CTA owns its dq rows, so the
// accumulation into dq_acc is a plain read-modify-write.
template <int D, typename T, int R>
__global__ void __launch_bounds__(SimtShape<D, R>::kThreads)
attn_bwd_dq_simt_kernel(const SimtBwdParams p) {
  using S = SimtShape<D, R>;
  extern __shared__ __align__(16) float simt_smem[];
  float* q_s = simt_smem;
  float* do_s = q_s + S::kTileFloats;
  float* k_s = do_s + S::kTileFloats;
  float* v_s = k_s + S::kTileFloats;
  float* ds_s = v_s + S::kTileFloats;
  int r0, h, b;
  decode_cta(p.Sq, p.Hq, p.B, p.causal, r0, h, b);
  const int hk = h / (p.Hq / p.Hkv);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_tile<D, R, T>(q_s, reinterpret_cast<const T*>(p.q) + b * p.q_sb + (int64_t)r0 * p.q_ss + h * p.q_sh,
                     p.q_ss, p.Sq - r0);
  load_tile<D, R, T>(do_s, reinterpret_cast<const T*>(p.dout) + b * p.do_sb + (int64_t)r0 * p.do_ss + h * p.do_sh,
                     p.do_ss, p.Sq - r0);
  float dq[R][S::kNC], lse[R], delta[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = r0 + ty + i * S::kTy;
    const size_t sidx = (size_t)b * p.lse_sb + (size_t)h * p.lse_sh + min(row, p.Sq - 1);
    lse[i] = row < p.Sq ? p.lse[sidx] : INFINITY;   // +inf: P = 0
    delta[i] = p.delta[sidx];
#pragma unroll
    for (int c = 0; c < S::kNC; ++c) dq[i][c] = 0.f;
  }

  int n_keys = p.Sk;
  if (p.causal) {
    const long long last = (long long)min(r0 + kRows, p.Sq) - 1 + p.causal_off;
    n_keys = (int)max(0ll, min((long long)p.Sk, last + 1));
  }
  const T* kbase = reinterpret_cast<const T*>(p.k) + b * p.k_sb + hk * p.k_sh;
  const T* vbase = reinterpret_cast<const T*>(p.v) + b * p.v_sb + hk * p.v_sh;

  for (int k0 = 0; k0 < n_keys; k0 += kTile) {
    __syncthreads();
    load_tile<D, R, T>(k_s, kbase + (int64_t)k0 * p.k_ss, p.k_ss, n_keys - k0);
    load_tile<D, R, T>(v_s, vbase + (int64_t)k0 * p.v_ss, p.v_ss, n_keys - k0);
    __syncthreads();
    float s[R][kCols], dp[R][kCols];
    dot_tiles<D, R>(s, q_s, k_s, ty, tx);
    const bool need_mask = k0 + kTile > p.Sk || (p.causal && (long long)k0 + kTile - 1 > (long long)r0 + p.causal_off);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < kCols; ++j) {
        float pe = expf(s[i][j] * p.scale - lse[i]);
        if (need_mask) {
          const int kidx = k0 + tx + 16 * j;
          const long long my_last = p.causal ? (long long)r0 + ty + i * S::kTy + p.causal_off : (long long)p.Sk;
          if (kidx >= p.Sk || (long long)kidx > my_last) pe = 0.f;
        }
        s[i][j] = pe;
      }
    dot_tiles<D, R>(dp, do_s, v_s, ty, tx);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < kCols; ++j) s[i][j] *= dp[i][j] - delta[i];
    put_scores<D, R>(ds_s, s, ty, tx);
    __syncwarp();
    add_product<D, R>(dq, ds_s, k_s, ty, tx);
  }
  // total = (earlier ring steps' sum, unless this is the first) + this block; it goes to
  // dq in the element type and / or back to the fp32 accumulator, whichever is given.
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = r0 + ty + i * S::kTy;
    if (row >= p.Sq) continue;
    float* acc = p.dq_acc ? p.dq_acc + (((size_t)b * p.Sq + row) * p.Hq + h) * D : nullptr;
    T* dst = p.dq ? reinterpret_cast<T*>(p.dq) + b * p.dq_sb + (int64_t)row * p.dq_ss + h * p.dq_sh : nullptr;
#pragma unroll
    for (int c = 0; c < S::kNC; c += S::kVec) {
      const int e = S::col(tx, c);
      float a[S::kVec];
#pragma unroll
      for (int u = 0; u < S::kVec; ++u) a[u] = 0.f;
      if (!p.dq_overwrite) load_cols<S::kVec, float>(a, acc + e);
#pragma unroll
      for (int u = 0; u < S::kVec; ++u) a[u] = fmaf(p.scale, dq[i][c + u], a[u]);
      if (dst) store_cols<S::kVec, T>(dst + e, a);
      if (acc) store_cols<S::kVec, float>(acc + e, a);
    }
  }
}

// dK/dV: key rows stationary, queries (of every head of the GQA group) streamed.
template <int D, typename T, int R>
__global__ void __launch_bounds__(SimtShape<D, R>::kThreads)
attn_bwd_dkv_simt_kernel(const SimtBwdParams p) {
  using S = SimtShape<D, R>;
  extern __shared__ __align__(16) float simt_smem[];
  float* k_s = simt_smem;
  float* v_s = k_s + S::kTileFloats;
  float* q_s = v_s + S::kTileFloats;
  float* do_s = q_s + S::kTileFloats;
  float* p_s = do_s + S::kTileFloats;
  float* lse_s = p_s + kRows * kLdP;
  float* dl_s = lse_s + kTile;
  int r0, g, b;
  decode_cta(p.Sk, p.Hkv, p.B, false, r0, g, b);
  const int G = p.Hq / p.Hkv;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_tile<D, R, T>(k_s, reinterpret_cast<const T*>(p.k) + b * p.k_sb + (int64_t)r0 * p.k_ss + g * p.k_sh,
                     p.k_ss, p.Sk - r0);
  load_tile<D, R, T>(v_s, reinterpret_cast<const T*>(p.v) + b * p.v_sb + (int64_t)r0 * p.v_ss + g * p.v_sh,
                     p.v_ss, p.Sk - r0);
  float dk[R][S::kNC], dv[R][S::kNC];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < S::kNC; ++c) dk[i][c] = dv[i][c] = 0.f;
  int q_first = 0;   // first query that sees a key of this block
  if (p.causal) q_first = (int)max(0ll, min((long long)p.Sq, (long long)r0 - p.causal_off));
  for (int hh = 0; hh < G; ++hh) {
    const int h = g * G + hh;
    const T* qbase = reinterpret_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
    const T* dobase = reinterpret_cast<const T*>(p.dout) + b * p.do_sb + h * p.do_sh;
    const size_t sbase = (size_t)b * p.lse_sb + (size_t)h * p.lse_sh;
    for (int q0 = q_first / kTile * kTile; q0 < p.Sq; q0 += kTile) {
      __syncthreads();
      load_tile<D, R, T>(q_s, qbase + (int64_t)q0 * p.q_ss, p.q_ss, p.Sq - q0, q_first - q0);
      load_tile<D, R, T>(do_s, dobase + (int64_t)q0 * p.do_ss, p.do_ss, p.Sq - q0, q_first - q0);
      if (threadIdx.x < kTile) {
        const int qi = q0 + threadIdx.x;
        const bool in = qi >= q_first && qi < p.Sq;
        lse_s[threadIdx.x] = in ? p.lse[sbase + qi] : INFINITY;
        dl_s[threadIdx.x] = in ? p.delta[sbase + qi] : 0.f;
      }
      __syncthreads();
      float s[R][kCols], dp[R][kCols];
      dot_tiles<D, R>(s, k_s, q_s, ty, tx);
      const bool need_mask =
          q0 + kTile > p.Sq || (p.causal && (long long)r0 + kRows - 1 > (long long)q0 + p.causal_off);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          float pe = expf(s[i][j] * p.scale - lse_s[tx + 16 * j]);
          if (need_mask) {
            const int qi = q0 + tx + 16 * j;
            const long long krow = (long long)r0 + ty + i * S::kTy;
            if (qi >= p.Sq || (p.causal && krow > (long long)qi + p.causal_off)) pe = 0.f;
          }
          s[i][j] = pe;
        }
      put_scores<D, R>(p_s, s, ty, tx);
      __syncwarp();
      add_product<D, R>(dv, p_s, do_s, ty, tx);
      dot_tiles<D, R>(dp, v_s, do_s, ty, tx);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < kCols; ++j) s[i][j] *= dp[i][j] - dl_s[tx + 16 * j];
      __syncwarp();   // P has been read
      put_scores<D, R>(p_s, s, ty, tx);
      __syncwarp();
      add_product<D, R>(dk, p_s, q_s, ty, tx);
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int krow = r0 + ty + i * S::kTy;
    if (krow >= p.Sk) continue;
    const size_t off = (((size_t)b * p.Sk + krow) * p.Hkv + g) * D;                   // fp32: contiguous
    const int64_t off_t = b * p.dkv_sb + (int64_t)krow * p.dkv_ss + g * p.dkv_sh;     // element type: strided
#pragma unroll
    for (int c = 0; c < S::kNC; c += S::kVec) {
      const int e = S::col(tx, c);
      float a[S::kVec], w[S::kVec], x[S::kVec], y[S::kVec];
#pragma unroll
      for (int u = 0; u < S::kVec; ++u) {
        a[u] = dk[i][c + u] * p.scale;
        w[u] = dv[i][c + u];
        x[u] = y[u] = 0.f;
      }
      if (p.dkv_fp32) {
        float* pk = reinterpret_cast<float*>(p.dk) + off + e;
        float* pv = reinterpret_cast<float*>(p.dv) + off + e;
        if (p.dkv_accumulate) {
          load_cols<S::kVec, float>(x, pk);
          load_cols<S::kVec, float>(y, pv);
        }
#pragma unroll
        for (int u = 0; u < S::kVec; ++u) { a[u] += x[u]; w[u] += y[u]; }
        store_cols<S::kVec, float>(pk, a);
        store_cols<S::kVec, float>(pv, w);
      } else {
        T* pk = reinterpret_cast<T*>(p.dk) + off_t + e;
        T* pv = reinterpret_cast<T*>(p.dv) + off_t + e;
        if (p.dkv_accumulate) {
          load_cols<S::kVec, T>(x, pk);
          load_cols<S::kVec, T>(y, pv);
        }
#pragma unroll
        for (int u = 0; u < S::kVec; ++u) { a[u] += x[u]; w[u] += y[u]; }
        store_cols<S::kVec, T>(pk, a);
        store_cols<S::kVec, T>(pv, w);
      }
    }
  }
}

// Launch one of the kernels: 64-row tiles x heads x batch CTAs in a linear grid.
template <typename Shape, typename P>
int launch_simt(void (*kern)(P), const P& p, int operand_tiles, int extra_floats, int rows, int heads, int batch,
                void* stream, const char* what) {
  const int smem = (operand_tiles * Shape::kTileFloats + kRows * kLdP + extra_floats) * (int)sizeof(float);
  int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem, what);
  if (rc) return rc;
  const long long grid = (long long)ceil_div(rows, kRows) * heads * batch;
  if (grid > 0x7fffffffll) {
    set_error("%s grid out of range", what);
    return SPA_EINVAL;
  }
  kern<<<(unsigned)grid, Shape::kThreads, smem, (cudaStream_t)stream>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s launch: %s", what, cudaGetErrorString(e));
    return SPA_ECUDA;
  }
  return SPA_OK;
}

// Rows per thread: 8 load less per multiply-add. At D = 64 they are faster although the backward
// kernels spill 40 (dK/dV) and 88 bytes (dQ) at 255 registers (S=1024, 32 heads: dK/dV 479 us with 8,
// 502 with 4); at D = 128 the accumulators of 8 rows spill far more (S=2900, 8 heads: 2825 and 2196).
template <int D>
constexpr int kSimtR = D == 128 ? 4 : 8;

template <int D, typename T>
int launch_fwd_simt_typed(const spa_fwd_args* a) {
  SimtFwdParams p;
  p.q = a->q; p.k = a->k; p.v = a->v;
  p.q_sb = a->q_sb; p.q_ss = a->q_ss; p.q_sh = a->q_sh;
  p.k_sb = a->k_sb; p.k_ss = a->k_ss; p.k_sh = a->k_sh;
  p.v_sb = a->v_sb; p.v_ss = a->v_ss; p.v_sh = a->v_sh;
  p.out = a->out; p.o_sb = a->o_sb; p.o_ss = a->o_ss; p.o_sh = a->o_sh;
  p.out_acc = a->out_acc; p.lse = a->lse;
  p.lse_sb = a->lse_sb; p.lse_sh = a->lse_sh;
  p.B = a->B; p.Sq = a->Sq; p.Sk = a->Sk; p.Hq = a->Hq; p.Hkv = a->Hkv;
  p.causal = a->causal; p.causal_off = a->causal_off; p.merge_prev = a->merge_prev;
  p.scale = a->scale;
  constexpr int R = kSimtR<D>;
  return launch_simt<SimtShape<D, R>>(attn_fwd_simt_kernel<D, T, R>, p, 3, 0, a->Sq, a->Hq, a->B, a->stream, "fwd simt");
}

template <int D, typename T>
int launch_bwd_simt_typed(const spa_bwd_args* a) {
  SimtBwdParams p;
  p.q = a->q; p.k = a->k; p.v = a->v; p.dout = a->dout;
  p.q_sb = a->q_sb; p.q_ss = a->q_ss; p.q_sh = a->q_sh;
  p.k_sb = a->k_sb; p.k_ss = a->k_ss; p.k_sh = a->k_sh;
  p.v_sb = a->v_sb; p.v_ss = a->v_ss; p.v_sh = a->v_sh;
  p.do_sb = a->do_sb; p.do_ss = a->do_ss; p.do_sh = a->do_sh;
  p.lse = a->lse; p.delta = a->delta; p.lse_sb = a->lse_sb; p.lse_sh = a->lse_sh;
  p.dq_acc = a->dq_acc; p.dq = a->dq; p.dq_sb = a->dq_sb; p.dq_ss = a->dq_ss; p.dq_sh = a->dq_sh;
  p.dq_overwrite = a->dq_overwrite;
  p.dk = a->dk; p.dv = a->dv; p.dkv_sb = a->dkv_sb; p.dkv_ss = a->dkv_ss; p.dkv_sh = a->dkv_sh;
  p.dkv_fp32 = a->dkv_fp32; p.dkv_accumulate = a->dkv_accumulate;
  p.B = a->B; p.Sq = a->Sq; p.Sk = a->Sk; p.Hq = a->Hq; p.Hkv = a->Hkv;
  p.causal = a->causal; p.causal_off = a->causal_off; p.scale = a->scale;
  constexpr int R = kSimtR<D>;
  using Shape = SimtShape<D, R>;
  int rc = SPA_OK;
  if (a->passes != SPA_BWD_DKV_ONLY)
    rc = launch_simt<Shape>(attn_bwd_dq_simt_kernel<D, T, R>, p, 4, 0, a->Sq, a->Hq, a->B, a->stream, "bwd dq simt");
  if (rc == SPA_OK && a->passes != SPA_BWD_DQ_ONLY)
    rc = launch_simt<Shape>(attn_bwd_dkv_simt_kernel<D, T, R>, p, 4, 2 * kTile, a->Sk, a->Hkv, a->B, a->stream,
                            "bwd dkv simt");
  return rc;
}

template <typename F32, typename BF, typename HF>
int dispatch_dtype(int dtype, F32 f32, BF bf, HF hf) {
  switch (dtype) {
    case SPA_DTYPE_F32: return f32();
    case SPA_DTYPE_BF16: return bf();
    case SPA_DTYPE_F16: return hf();
  }
  set_error("unknown dtype %d", dtype);
  return SPA_EINVAL;
}

}  // namespace

int launch_fwd_simt(const spa_fwd_args* a) {
  switch (a->D) {
    case 32:
      return dispatch_dtype(a->dtype, [&] { return launch_fwd_simt_typed<32, float>(a); },
                            [&] { return launch_fwd_simt_typed<32, __nv_bfloat16>(a); },
                            [&] { return launch_fwd_simt_typed<32, __half>(a); });
    case 64:
      return dispatch_dtype(a->dtype, [&] { return launch_fwd_simt_typed<64, float>(a); },
                            [&] { return launch_fwd_simt_typed<64, __nv_bfloat16>(a); },
                            [&] { return launch_fwd_simt_typed<64, __half>(a); });
    case 128:
      return dispatch_dtype(a->dtype, [&] { return launch_fwd_simt_typed<128, float>(a); },
                            [&] { return launch_fwd_simt_typed<128, __nv_bfloat16>(a); },
                            [&] { return launch_fwd_simt_typed<128, __half>(a); });
  }
  set_error("CUDA-core forward supports head_dim 32, 64, 128, got %d", a->D);
  return SPA_EUNSUPPORTED;
}

int launch_bwd_simt(const spa_bwd_args* a) {
  switch (a->D) {
    case 32:
      return dispatch_dtype(a->dtype, [&] { return launch_bwd_simt_typed<32, float>(a); },
                            [&] { return launch_bwd_simt_typed<32, __nv_bfloat16>(a); },
                            [&] { return launch_bwd_simt_typed<32, __half>(a); });
    case 64:
      return dispatch_dtype(a->dtype, [&] { return launch_bwd_simt_typed<64, float>(a); },
                            [&] { return launch_bwd_simt_typed<64, __nv_bfloat16>(a); },
                            [&] { return launch_bwd_simt_typed<64, __half>(a); });
    case 128:
      return dispatch_dtype(a->dtype, [&] { return launch_bwd_simt_typed<128, float>(a); },
                            [&] { return launch_bwd_simt_typed<128, __nv_bfloat16>(a); },
                            [&] { return launch_bwd_simt_typed<128, __half>(a); });
  }
  set_error("CUDA-core backward supports head_dim 32, 64, 128, got %d", a->D);
  return SPA_EUNSUPPORTED;
}

}  // namespace spa
