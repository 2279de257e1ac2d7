// Packed sequences in one launch: the table that tells a CTA of the tensor-core kernels which
// sequence and which block of it it owns.
//
// A launch per sequence (and per group of heads) leaves the chip almost empty: eight documents
// of 16k tokens, 8 kv heads taken one at a time, were 192 attention launches of 4 to 150 CTAs.
// Forward and backward of those documents (32 / 8 heads, D = 128, bf16): 8.32 -> 2.24 ms, with
// the later steps 2.12; four sequences of 64 to 512 tokens (8 heads, D = 64, fp16): 1264 -> 275 us,
// through the C++ node 111, host time for the most part.
// The table travels as a kernel parameter, by value: nothing is copied to the device, nothing
// outlives the launch, and a stream capture records it with the launch.
//
// Tiles may run past the end of a sequence into the next one's rows. That is harmless for the
// stationary rows (they are not stored) but not for the dimension a product sums over: the
// masked weight is 0 there, and 0 * Inf or 0 * NaN of a neighbouring sequence would leak. Those
// operands (V forward; K, V in the dQ pass; Q, dO in the dK/dV pass) are read through a TMA map
// of the sequence alone, which fills rows past its end with zeros, as a call on the sequence
// by itself would see them.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include <algorithm>

#include "spa_internal.h"

namespace spa {

constexpr int kVarMaxSeqs = 32;   // sequences per launch (the table stays under 10 KB)

struct VarSeq {
  int q0, sq, k0, sk;   // first row and length in the packed query / key tensors
  int off;              // causal offset of this sequence
  int nblk;             // blocks of the kernel's stationary dimension
};

template <bool kVar, int kMaps>
struct VarTable {       // plain launches pass an empty parameter; the accessors are never reached
  __device__ __forceinline__ VarSeq seq(int) const { return VarSeq{}; }
  __device__ __forceinline__ const CUtensorMap* map(int, int) const { return nullptr; }
};

template <int kMaps>
struct alignas(64) VarTable<true, kMaps> {
  CUtensorMap tm[kVarMaxSeqs][kMaps];
  VarSeq s[kVarMaxSeqs];   // longest (most blocks) first
  int n;

  __device__ __forceinline__ const VarSeq& seq(int i) const { return s[i]; }
  __device__ __forceinline__ const CUtensorMap* map(int i, int m) const { return &tm[i][m]; }
  // The w-th (sequence, block) pair: blocks of equal index belong together, the highest index
  // first. Between nblk[i + 1] and nblk[i] exactly the first i + 1 sequences have blocks.
  // With the causal cost proportional to the index this is longest-first over all sequences.
  __device__ __forceinline__ int decode(int w, int& sg) const {
    int i = 0;
    int hi = s[0].nblk;
    while (true) {
      const int lo = i + 1 < n ? s[i + 1].nblk : 0;
      const int band = (i + 1) * (hi - lo);
      if (w < band || i + 1 >= n) {
        sg = w % (i + 1);
        return hi - 1 - w / (i + 1);
      }
      w -= band;
      hi = lo;
      ++i;
    }
  }
};

// Host: enter the sequences, most blocks first, and return the number of (sequence, block)
// pairs. `block` rows per block of the stationary dimension (queries, or keys with by_key).
template <int kMaps>
inline long long fill_var_table(VarTable<true, kMaps>* t, const spa_seq* seqs, int n, int block, bool by_key) {
  long long total = 0;
  for (int i = 0; i < n; ++i) {
    const spa_seq& q = seqs[i];
    VarSeq& v = t->s[i];
    v.q0 = q.q0; v.sq = q.sq; v.k0 = q.k0; v.sk = q.sk; v.off = q.causal_off;
    v.nblk = ceil_div(by_key ? q.sk : q.sq, block);
    total += v.nblk;
  }
  std::stable_sort(t->s, t->s + n, [](const VarSeq& a, const VarSeq& b) { return a.nblk > b.nblk; });
  t->n = n;
  return total;
}

// Row `row` of a 16-bit tensor with `stride` elements between rows.
inline const void* row_ptr(const void* base, int row, int64_t stride) {
  return static_cast<const char*>(base) + (int64_t)row * stride * 2;
}

}  // namespace spa
