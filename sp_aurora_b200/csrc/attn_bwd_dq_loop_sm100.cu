// Flash-attention backward, dQ pass, for many short query tiles (tcgen05 + TMEM + TMA): the kernel
// of attn_bwd_dq_sm100.cu with CTAs that work through several query tiles (worklist.cuh).
//
// The set-up and the fill and drain of the pipeline cost 3 us a query tile, as much as three K/V
// tiles. Across the query tiles of one CTA the K/V ring keeps running, the next Q is fetched while
// the last product finishes, and the next S and dP run under the epilogue. 2 x 3001 causal rows of
// 32 / 8 heads, D=128: 251 -> 224 us; 4 x 2048 rows of 16 heads, no mask: 241 -> 222.
//
// A kernel of its own, because the hand-offs between query tiles cost the single-tile form 3 to 6 %
// where the walks are long. Products, layout, warp roles, TMEM columns and the order of summation
// are the same, so are the results, bit for bit.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include <type_traits>

#include "spa_internal.h"
#include "tc05.cuh"
#include "varlen.cuh"
#include "worklist.cuh"

namespace spa {
namespace {

constexpr int kTileM = 128;   // query rows per CTA
constexpr int kTileN = 128;   // keys per K/V tile
constexpr int kThreads = 576;
constexpr int kComputeThreads = 512;
constexpr int kWarpTma = 16, kWarpMma = 17;
constexpr int kStages = 3;
constexpr float kLog2e = 1.4426950408889634f;
constexpr uint32_t kColS = 0, kColDP = 128, kColDQ = 256, kColDS = 384, kColQ = 448;

struct DqParams {
  int B, Sq, Sk, Hq, Hkv;
  int causal, causal_off;
  int dq_overwrite;
  int n_qblk;
  int chunk;   // query tiles per scheduling chunk (n_qblk or 1)
  int n_items; // (query tile, head, batch) triples of the launch
  int may_skip;   // some query tile sees no key at all
  float scale, scale_log2;
  const void* q;
  int64_t q_sb, q_ss, q_sh;
  const float* lse;
  const float* delta;
  int64_t lse_sb, lse_sh;
  float* dq_acc;
  void* dq;
  int64_t dq_sb, dq_ss, dq_sh;
  int* status;
};

template <int D>
struct DqSmem {
  static constexpr int kSlab = kTileN * 128;                 // 128 rows x 128 B
  static constexpr int kTile = (D / 64) * kSlab;             // one dO / K / V tile
  static constexpr int kStageBytes = 2 * kTile;              // K + V
  static constexpr int kDoOff = 0;
  static constexpr int kKVOff = kDoOff + kTile;
  static constexpr int kItemOff = kKVOff + kStages * kStageBytes;
  static constexpr int kMaxItems = 48;                       // per CTA
  static constexpr int kBarOff = kItemOff + kMaxItems * (int)sizeof(WorkItem);
  static constexpr int kNumBars = 2 + 2 * kStages + 6;
  static constexpr int kTotal = kBarOff + kNumBars * 8 + 16;
};

template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// kVar: one launch over the sequences of a packed batch (B = 1); K and V are then read through
// the maps of the sequence's table entry, dO through tm_do over the whole packed tensor.
template <int D, typename T, bool kVar>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_dq_loop_sm100_kernel(const __grid_constant__ CUtensorMap tm_k,
                         const __grid_constant__ CUtensorMap tm_v,
                         const __grid_constant__ CUtensorMap tm_do, const DqParams p,
                         const __grid_constant__ VarTable<kVar, 2> var) {
  using L = DqSmem<D>;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* do_full = bars;
  uint64_t* q_ready = bars + 1;
  uint64_t* kv_full = bars + 2;
  uint64_t* kv_empty = kv_full + kStages;
  uint64_t* sdp_full = kv_empty + kStages;    // S(j) and dP(j) are complete
  uint64_t* sdp_free = sdp_full + 1;          // S(j) and dP(j) are in registers
  uint64_t* ds_full = sdp_free + 1;
  uint64_t* dq_done = ds_full + 1;
  uint64_t* dq_free = dq_done + 1;            // the finished dQ is in registers
  uint64_t* do_empty = dq_free + 1;           // every dP of the query tile is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::kNumBars);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // Work decode of item w: query tiles of one chunk fastest (longest first under a causal
  // mask), then heads, batch, chunks; the CTAs resident together stream the K/V of one kv head.
  // Packed sequences: heads fastest, then the tiles of all sequences, longest walk first.
  auto decode = [&](int w) -> WorkItem {
    int qblk;
    WorkItem t = {};
    if constexpr (kVar) {
      t.h = w % p.Hq;
      qblk = var.decode(w / p.Hq, t.sg);
    } else {
      const int q_lo = w % p.chunk;
      w /= p.chunk;
      t.h = w % p.Hq;
      w /= p.Hq;
      t.b = w % p.B;
      qblk = p.n_qblk - 1 - ((w / p.B) * p.chunk + q_lo);
    }
    const int Sq = kVar ? var.seq(t.sg).sq : p.Sq;
    const int Sk = kVar ? var.seq(t.sg).sk : p.Sk;
    t.r0 = qblk * kTileM;
    t.n0 = (Sk + kTileN - 1) / kTileN;   // K/V tiles the query tile can see
    if (p.causal) {
      const int off = kVar ? var.seq(t.sg).off : p.causal_off;
      const long long last_key = (long long)min(t.r0 + kTileM, Sq) - 1 + off;  // inclusive
      const int nc = last_key < 0 ? 0 : (int)(last_key / kTileN) + 1;
      t.n0 = min(t.n0, nc);
    }
    return t;
  };
  WorkItem* items = reinterpret_cast<WorkItem*>(smem + L::kItemOff);
  const int n_items = item_count(p.n_items);
  for (int i = threadIdx.x; i < n_items; i += kThreads) items[i] = decode(item_index(i));
  // First item from i on that sees a key.
  auto skip_empty = [&](int i) -> int {
    while (i < n_items && items[i].n0 == 0) ++i;
    return i;
  };

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    mbar_init(do_full, 1);
    mbar_init(q_ready, kComputeThreads / 32);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    mbar_init(sdp_full, 1);
    mbar_init(sdp_free, kComputeThreads / 32);
    mbar_init(ds_full, kComputeThreads / 32);
    mbar_init(dq_done, 1);
    mbar_init(dq_free, kComputeThreads / 32);
    mbar_init(do_empty, 1);
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == kWarpMma) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wc{p.status, cta_abort};
  grid_release();   // as in attn_bwd_dq_sm100.cu

  if (warp == kWarpTma) {
    // ------------------------------------------------------------------ TMA
    if (lane == 0) {
      tma_prefetch_desc(&tm_do);
      uint32_t used[kStages] = {};   // fills of each ring slot so far; every item starts at slot 0
      int n = 0;                     // items so far
      for (int i = skip_empty(0); i < n_items; i = skip_empty(i + 1), ++n) {
        const WorkItem t = items[i];
        const CUtensorMap* const k_map = kVar ? var.map(t.sg, 0) : &tm_k;
        const CUtensorMap* const v_map = kVar ? var.map(t.sg, 1) : &tm_v;
        const int q_row = t.r0 + (kVar ? var.seq(t.sg).q0 : 0);
        const int hk = t.h / (p.Hq / p.Hkv);
        bool ok = true;
        for (int j0 = 0; j0 < t.n0 && ok; j0 += kStages) {
#pragma unroll
          for (int slot = 0; slot < kStages; ++slot) {
          const int j = j0 + slot;
          if (j >= t.n0 || !ok) break;
          ok = mbar_wait(&kv_empty[slot], (used[slot] & 1) ^ 1, wc, 0, j);
          if (!ok) break;
          ++used[slot];
          uint8_t* st = smem + L::kKVOff + slot * L::kStageBytes;
          mbar_arrive_expect_tx(&kv_full[slot], L::kStageBytes);
          for (int s = 0; s < D / 64; ++s) {
            tma_load_4d(st + s * L::kSlab, k_map, &kv_full[slot], s * 64, j * kTileN, hk, t.b);
            tma_load_4d(st + L::kTile + s * L::kSlab, v_map, &kv_full[slot], s * 64, j * kTileN, hk, t.b);
          }
          if (j == 0) {
            if (n > 0) ok = mbar_wait(do_empty, (n - 1) & 1, wc, 5, n);
            if (!ok) break;
            mbar_arrive_expect_tx(do_full, L::kTile);
            for (int s = 0; s < D / 64; ++s)
              tma_load_4d(smem + L::kDoOff + s * L::kSlab, &tm_do, do_full, s * 64, q_row, t.h, t.b);
          }
          }
        }
        if (!ok) break;
      }
    }
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------------ MMA
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc(128, kTileN, kBf16, false, false);
      constexpr uint32_t idesc_dq = make_idesc(128, D, kBf16, false, true);
      const uint32_t do_base = smem_u32(smem + L::kDoOff);
      const uint32_t kv_base = smem_u32(smem + L::kKVOff);
      const SmemDesc do_km = make_smem_desc(do_base, 16, 1024);          // dO, K-major (A of dP)
      const SmemDesc kv_km = make_smem_desc(kv_base, 16, 1024);          // K / V, K-major (B of S, dP)
      const SmemDesc k_mn = make_smem_desc(kv_base, L::kSlab, 1024);     // K, MN-major (B of dQ)
      // `slot` is a compile-time constant at every call site (the tile loop is unrolled
      // over the ring period): runtime descriptor words cost issue time.
      // S(j) = Q K_j^T : A = Q from TMEM, B = K tile (K-major).
      // `use` is the number of earlier fills of the slot.
      auto issue_s = [&](uint32_t use, const int slot) -> bool {
        if (!mbar_wait(&kv_full[slot], use & 1, wc, 3, slot)) return false;
        tc_fence_after();
        const uint32_t b0 = (slot * L::kStageBytes) >> 4;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk / 4) * L::kSlab + (kk % 4) * 32) >> 4;
          mma_ts_d(tmem_base + kColS, tmem_base + kColQ + kk * 8, kv_km, b0 + off, idesc_s, kk > 0);
        }
        return true;
      };
      // dP(j) = dO V_j^T : A = dO tile (shared memory), B = V tile (K-major).
      auto issue_dp = [&](const int slot) {
        const uint32_t b0 = (slot * L::kStageBytes + L::kTile) >> 4;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk / 4) * L::kSlab + (kk % 4) * 32) >> 4;
          mma_ss_d(tmem_base + kColDP, do_km, off, kv_km, b0 + off, idesc_s, kk > 0);
        }
        mma_commit(sdp_full);
      };

      uint32_t used[kStages] = {};   // as in the producer
      uint32_t g = 0;                // K/V tiles so far
      int n = 0;                     // items so far
      bool ok = true;
      for (int i = skip_empty(0); ok && i < n_items; i = skip_empty(i + 1), ++n) {
        const int n_kv = items[i].n0;
        ok = mbar_wait(q_ready, n & 1, wc, 2, n);
        if (ok) ok = mbar_wait(do_full, n & 1, wc, 1, n);
        tc_fence_after();
        // dS of the last tile has been handed in, so its S and dP columns are free too.
        if (ok) ok = issue_s(used[0], 0);
        if (!ok) break;
        issue_dp(0);
        if (n_kv == 1) mma_commit(do_empty);
        for (int j0 = 0; j0 < n_kv && ok; j0 += kStages) {
#pragma unroll
          for (int sl = 0; sl < kStages; ++sl) {
            const int j = j0 + sl;
            if (j >= n_kv || !ok) break;
            ++used[sl];
            if (j + 1 < n_kv) {
              ok = mbar_wait(sdp_free, g & 1, wc, 4, j);    // S(j) and dP(j) are in registers
              if (!ok) break;
              tc_fence_after();
              ok = issue_s(used[(sl + 1) % kStages], (sl + 1) % kStages);
              if (!ok) break;
              issue_dp((sl + 1) % kStages);
              if (j + 2 == n_kv) mma_commit(do_empty);
            }
            ok = mbar_wait(ds_full, g & 1, wc, 6, j);
            if (ok && j == 0 && n > 0) ok = mbar_wait(dq_free, (n - 1) & 1, wc, 7, n);
            if (!ok) break;
            tc_fence_after();
            // dQ += dS(j) K_j : A = dS from TMEM, B = K tile MN-major (rows = keys).
            const uint32_t b0 = (sl * L::kStageBytes) >> 4;
#pragma unroll
            for (int kk = 0; kk < kTileN / 16; ++kk)
              mma_ts_d(tmem_base + kColDQ, tmem_base + kColDS + kk * 8, k_mn, b0 + ((kk * 2048) >> 4),
                       idesc_dq, (j > 0 || kk > 0));
            mma_commit(&kv_empty[sl]);
            mma_commit(dq_done);
            ++g;
          }
        }
      }
    }
  } else {
    // -------------------------------------------------------------- compute
    const int grp = warp >> 2;                 // key-column quarter of the tile
    const int quad = warp & 3;
    const int r = quad * 32 + lane;            // query row in tile = TMEM lane
    const int c_base = grp * 32;
    constexpr int kOutCols = D / 4;            // dQ columns (and Q elements) per group
    constexpr int kWords = D / 8;              // 32-bit words (two Q elements each) per group
    const uint32_t lane_field = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem_base + lane_field + kColS + c_base;
    const uint32_t t_dp = tmem_base + lane_field + kColDP + c_base;
    const uint32_t t_ds = tmem_base + lane_field + kColDS + grp * 16;
    const uint32_t t_dq = tmem_base + lane_field + kColDQ + grp * kOutCols;
    const uint32_t t_q = tmem_base + lane_field + kColQ + grp * (D / 8);
    bool ok = true;

    // Length of the item's sequence, its first row in the packed tensors.
    auto seq_q = [&](const WorkItem& t) -> int { return kVar ? var.seq(t.sg).sq : p.Sq; };
    auto row_base = [&](const WorkItem& t) -> int { return kVar ? var.seq(t.sg).q0 : 0; };
    // A quarter of the thread's Q row, the A operand of S (zeros past the end of the sequence).
    auto load_q = [&](const WorkItem& t, uint32_t (&qw)[kWords]) {
      const int qrow = t.r0 + r;
      if (qrow < seq_q(t)) {
        const uint4* src = reinterpret_cast<const uint4*>(
            reinterpret_cast<const T*>(p.q) + (size_t)t.b * p.q_sb + (size_t)(row_base(t) + qrow) * p.q_ss +
            (size_t)t.h * p.q_sh + grp * (D / 4));
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i) {
          const uint4 v = src[i];
          qw[4 * i] = v.x; qw[4 * i + 1] = v.y; qw[4 * i + 2] = v.z; qw[4 * i + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < kWords; ++i) qw[i] = 0u;
      }
    };
    auto store_q = [&](const uint32_t (&qw)[kWords]) {
      if constexpr (D == 128) tmem_st16(t_q, qw); else tmem_st8(t_q, qw);
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(q_ready);
    };
    // Row statistics, negated for the packed multiply-adds: -inf in place of -lse makes
    // out-of-range rows give P = 0.
    auto load_stats = [&](const WorkItem& t, float& nlse2, float& ndlt) {
      const int qrow = t.r0 + r;
      const size_t sidx = (size_t)t.b * p.lse_sb + (size_t)t.h * p.lse_sh + (qrow < seq_q(t) ? row_base(t) + qrow : 0);
      nlse2 = qrow < seq_q(t) ? -p.lse[sidx] * kLog2e : -INFINITY;
      ndlt = qrow < seq_q(t) ? -p.delta[sidx] : 0.f;
    };
    // total = (earlier ring steps' sum unless dq_overwrite) + o; it goes to dq in the element
    // type and / or back to the fp32 accumulator, whichever is given.
    auto write_rows = [&](const WorkItem& t, float (&o)[kOutCols]) {
      const int qrow = t.r0 + r;
      if (qrow >= seq_q(t)) return;
      const size_t acc_off = (((size_t)t.b * p.Sq + qrow) * p.Hq + t.h) * D + grp * kOutCols;
      if (!p.dq_overwrite && p.dq_acc) {
        const float4* a4 = reinterpret_cast<const float4*>(p.dq_acc + acc_off);
#pragma unroll
        for (int i = 0; i < kOutCols / 4; ++i) {
          const float4 a = a4[i];
          o[4 * i] += a.x; o[4 * i + 1] += a.y; o[4 * i + 2] += a.z; o[4 * i + 3] += a.w;
        }
      }
      if (p.dq) {
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.dq) + (size_t)t.b * p.dq_sb +
                                              (size_t)(row_base(t) + qrow) * p.dq_ss + (size_t)t.h * p.dq_sh +
                                              grp * kOutCols);
#pragma unroll
        for (int i = 0; i < kOutCols / 8; ++i)
          dst[i] = make_uint4(pack2<T>(o[8 * i], o[8 * i + 1]), pack2<T>(o[8 * i + 2], o[8 * i + 3]),
                              pack2<T>(o[8 * i + 4], o[8 * i + 5]), pack2<T>(o[8 * i + 6], o[8 * i + 7]));
      }
      if (p.dq_acc) {
        float4* dst = reinterpret_cast<float4*>(p.dq_acc + acc_off);
#pragma unroll
        for (int i = 0; i < kOutCols / 4; ++i)
          dst[i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      }
    };

    // Query tiles without a visible key take no part in the pipeline: their total is what it was.
    if (p.may_skip && (p.dq_overwrite || p.dq)) {
      for (int e = 0; e < n_items; ++e) {
        const WorkItem t = items[e];
        if (t.n0 > 0) continue;
        float o[kOutCols];
#pragma unroll
        for (int i = 0; i < kOutCols; ++i) o[i] = 0.f;
        write_rows(t, o);
      }
    }

    int g = 0;   // K/V tiles so far
    int cur = skip_empty(0);
    float nlse2 = 0.f, ndlt = 0.f;
    if (cur < n_items) {
      const WorkItem t = items[cur];
      uint32_t qw[kWords];
      load_q(t, qw);
      store_q(qw);
      load_stats(t, nlse2, ndlt);
    }
    while (cur < n_items) {
      const WorkItem t = items[cur];
      const int qrow = t.r0 + r;
      const int Sk = kVar ? var.seq(t.sg).sk : p.Sk;
      const int off = kVar ? var.seq(t.sg).off : p.causal_off;
      for (int j = 0; j < t.n0; ++j, ++g) {
        // dP(j) follows S(j) on the in-order tensor pipe, so its completion covers both. Both are
        // taken into registers before the exponentials: the issuer can then put S(j+1) and
        // dP(j+1) on the pipe back to back while this tile is turned into dS.
        ok = warp_wait(sdp_full, g & 1, wc, 8, g);
        if (!ok) break;
        tc_fence_after();
        uint32_t sr[32], dpr[32];
        tmem_ld32(t_s, sr);
        tmem_ld32(t_dp, dpr);
        tmem_ld_wait();
        tc_fence_before();
        warp_arrive(sdp_free);
        float* pr = reinterpret_cast<float*>(sr);   // scores, then probabilities, in place

        const int k0 = j * kTileN;
        const bool need_mask =
            (k0 + kTileN > Sk) ||
            (p.causal && ((long long)k0 + kTileN - 1 > (long long)t.r0 + off));
        if (!need_mask) {                            // tiles below the diagonal: no selects
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float x0, x1;
            fma2(x0, x1, pr[c], pr[c + 1], p.scale_log2, p.scale_log2, nlse2, nlse2);
            pr[c] = fast_exp2(x0);
            pr[c + 1] = fast_exp2(x1);
          }
        } else {
          long long lim = Sk - 1;
          if (p.causal) lim = min(lim, (long long)qrow + off);
          const int limit = (int)max(0ll, min(lim - k0 - c_base + 1, 32ll));   // first masked column
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float x0, x1;
            fma2(x0, x1, pr[c], pr[c + 1], p.scale_log2, p.scale_log2, nlse2, nlse2);
            pr[c] = c < limit ? fast_exp2(x0) : 0.f;
            pr[c + 1] = c + 1 < limit ? fast_exp2(x1) : 0.f;
          }
        }
        uint32_t dsp[16];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float e0, e1, d0, d1;
          add2(e0, e1, __uint_as_float(dpr[c]), __uint_as_float(dpr[c + 1]), ndlt, ndlt);
          mul2(d0, d1, pr[c], pr[c + 1], e0, e1);
          dsp[c >> 1] = pack2<T>(d0, d1);
        }
        if (g > 0) {
          // The previous tile's dQ product has finished reading the dS columns.
          ok = warp_wait(dq_done, (g - 1) & 1, wc, 10, g);
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st16(t_ds, dsp);
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(ds_full);
      }
      if (!ok) break;
      // Every S product of this item is complete (its last scores have been read): Q may go.
      const int nxt = skip_empty(cur + 1);
      if (nxt < n_items) {
        const WorkItem nt = items[nxt];
        uint32_t qw[kWords];
        load_q(nt, qw);
        load_stats(nt, nlse2, ndlt);
        store_q(qw);
      }
      // ----------------------------------------------------------- epilogue
      ok = warp_wait(dq_done, (g - 1) & 1, wc, 11, g);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[kOutCols];
      if constexpr (kOutCols == 32) tmem_ld32(t_dq, v); else tmem_ld16(t_dq, v);
      tmem_ld_wait();
      tc_fence_before();
      warp_arrive(dq_free);
      float o[kOutCols];
#pragma unroll
      for (int i = 0; i < kOutCols; ++i) o[i] = __uint_as_float(v[i]) * p.scale;
      write_rows(t, o);
      cur = nxt;
    }
  }

  // Common exit: give in-flight copies/MMAs of an aborted CTA time to land, then free TMEM.
  tc_fence_before();
  __syncthreads();
  if (*cta_abort) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D, typename T, bool kVar>
int launch_dq_loop_typed(const spa_bwd_args* a, int is_bf16, const spa_seq* seqs, int n_seq) {
  using L = DqSmem<D>;
  CUtensorMap tk, tv, tdo;
  if (encode_rows_map(&tdo, a->dout, is_bf16, D, a->Sq, a->Hq, a->B, a->do_ss, a->do_sh, a->do_sb,
                      kTileM))
    return SPA_ECUDA;
  if (encode_rows_map(&tk, a->k, is_bf16, D, a->Sk, a->Hkv, a->B, a->k_ss, a->k_sh, a->k_sb, kTileN))
    return SPA_ECUDA;
  if (encode_rows_map(&tv, a->v, is_bf16, D, a->Sk, a->Hkv, a->B, a->v_ss, a->v_sh, a->v_sb, kTileN))
    return SPA_ECUDA;
  DqParams p;
  p.B = a->B; p.Sq = a->Sq; p.Sk = a->Sk; p.Hq = a->Hq; p.Hkv = a->Hkv;
  p.causal = a->causal; p.causal_off = a->causal_off;
  p.dq_overwrite = a->dq_overwrite;
  p.n_qblk = ceil_div(a->Sq, kTileM);
  p.chunk = (!a->causal || p.n_qblk >= 512) ? p.n_qblk : 1;
  p.scale = a->scale; p.scale_log2 = a->scale * kLog2e;
  p.q = a->q; p.q_sb = a->q_sb; p.q_ss = a->q_ss; p.q_sh = a->q_sh;
  p.lse = a->lse; p.delta = a->delta; p.lse_sb = a->lse_sb; p.lse_sh = a->lse_sh;
  p.dq_acc = a->dq_acc; p.dq = a->dq; p.dq_sb = a->dq_sb; p.dq_ss = a->dq_ss; p.dq_sh = a->dq_sh;
  p.status = device_status_word();
  if (!p.status) return SPA_ECUDA;
  const int smem_bytes = L::kTotal + 1024;
  auto kern = attn_bwd_dq_loop_sm100_kernel<D, T, kVar>;
  int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes, "bwd dq sm100");
  if (rc) return rc;
  long long grid = (long long)p.n_qblk * a->B * a->Hq;
  VarTable<kVar, 2> var;
  if constexpr (kVar) {
    grid = fill_var_table(&var, seqs, n_seq, kTileM, /*by_key=*/false) * a->Hq;
    for (int i = 0; i < n_seq; ++i) {
      const VarSeq& q = var.s[i];
      if (encode_rows_map(&var.tm[i][0], row_ptr(a->k, q.k0, a->k_ss), is_bf16, D, q.sk, a->Hkv, 1, a->k_ss,
                          a->k_sh, a->k_sb, kTileN) ||
          encode_rows_map(&var.tm[i][1], row_ptr(a->v, q.k0, a->v_ss), is_bf16, D, q.sk, a->Hkv, 1, a->v_ss,
                          a->v_sh, a->v_sb, kTileN))
        return SPA_ECUDA;
    }
  }
  if (grid <= 0 || grid > 0x7fffffffll) {
    set_error("bwd dq grid out of range");
    return SPA_EINVAL;
  }
  p.n_items = (int)grid;
  p.may_skip = a->causal && a->causal_off < 0;
  for (int i = 0; i < n_seq; ++i) p.may_skip |= a->causal && seqs[i].causal_off < 0;
  grid = worklist_grid(grid, device_sm_count(), L::kMaxItems);
  kern<<<(unsigned)grid, kThreads, smem_bytes, (cudaStream_t)a->stream>>>(tk, tv, tdo, p, var);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("bwd dq sm100 launch: %s", cudaGetErrorString(e));
    return SPA_ECUDA;
  }
  return SPA_OK;
}

template <bool kVar>
int launch_dq_loop_any(const spa_bwd_args* a, const spa_seq* seqs, int n_seq) {
  const bool bf = a->dtype == SPA_DTYPE_BF16;
  if (a->D == 128)
    return bf ? launch_dq_loop_typed<128, __nv_bfloat16, kVar>(a, 1, seqs, n_seq)
              : launch_dq_loop_typed<128, __half, kVar>(a, 0, seqs, n_seq);
  return bf ? launch_dq_loop_typed<64, __nv_bfloat16, kVar>(a, 1, seqs, n_seq)
            : launch_dq_loop_typed<64, __half, kVar>(a, 0, seqs, n_seq);
}

// K/V tiles that the `blocks` query tiles of a sequence go through all together.
long long walk_tiles(long long blocks, int sk, bool causal, int causal_off) {
  const long long n = ceil_div(sk, kTileN);
  if (!causal) return blocks * n;
  // Tile i (the last one taken as full) sees first + i K/V tiles, cut to 0..n.
  const long long last_key = kTileM - 1 + (long long)causal_off;   // of tile 0
  const long long first = last_key >= 0 ? last_key / kTileN + 1 : -((-last_key - 1) / kTileN);
  auto sum_to = [](long long x) { return x > 0 ? x * (x + 1) / 2 : 0ll; };
  return sum_to(first + blocks - 1) - sum_to(first - 1) - sum_to(first + blocks - 1 - n) + sum_to(first - 1 - n);
}

}  // namespace

// Several items for every SM and short walks: at most 24 K/V tiles on average without a mask, or 48
// query tiles that start at the diagonal (24.5). Measured: 12 tiles 251 -> 224 us, 16 tiles 241 ->
// 222, 32 tiles even; beyond that a fixed schedule loses, its CTAs drift apart and stop sharing K/V
// in L2: 32768 rows 11.8 -> 14.3 ms.
bool dq_loops(const spa_bwd_args* a, const spa_seq* seqs, int n_seq) {
  if (a->D != 64 && a->D != 128) return false;
  long long items = 0, walk = 0;
  for (int i = 0; i < (n_seq > 0 ? n_seq : 1); ++i) {
    const long long blocks = ceil_div(n_seq > 0 ? seqs[i].sq : a->Sq, kTileM);
    items += blocks;
    walk += n_seq > 0 ? walk_tiles(blocks, seqs[i].sk, a->causal, seqs[i].causal_off)
                      : walk_tiles(blocks, a->Sk, a->causal, a->causal_off);
  }
  return items * a->Hq * a->B >= 3ll * device_sm_count() && 2 * walk <= 49 * items;
}

int launch_bwd_dq_loop_sm100(const spa_bwd_args* a, const spa_seq* seqs, int n_seq) {
  return n_seq > 0 ? launch_dq_loop_any<true>(a, seqs, n_seq) : launch_dq_loop_any<false>(a, nullptr, 0);
}

}  // namespace spa
