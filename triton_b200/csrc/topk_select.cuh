// Best-k selection in registers, shared by the stand-alone top-k kernels and the router kernel.
//
// Order: larger value first, equal values to the smaller expert index (triton_kernels
// topk_details/_topk_forward.py:29-35 packs `PAD - index` under the value for the same effect).
#pragma once
#include <cstdint>

// order-preserving map float -> uint32 (larger float <=> larger key), never 0: that is an empty place's key, and the NaN whose bits
// are all ones must fill one like any other value
__device__ __forceinline__ uint32_t sel_float_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return max(b ^ ((b & 0x80000000u) ? 0xFFFFFFFFu : 0x80000000u), 1u);
}
__device__ __forceinline__ float sel_key_float(uint32_t k) {
  return __uint_as_float(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xFFFFFFFFu));
}

// The K best (value key, expert) pairs, best first.  An insertion compares the candidate with all K places at once
// (independent compares, then two selects per place) instead of bubbling it down: a thread walks its share of a row
// alone, so the length of the dependent chain is what the selection costs.  `push` takes experts in ascending order
// and keeps the earlier of two equal values ahead with a strict compare; `merge` joins two lists of any experts and
// compares the expert index too (a third of the instructions of inserting one list into the other).
template <int K>
struct TopK {
  uint32_t key[K];
  int idx[K];
  __device__ __forceinline__ TopK() {
#pragma unroll
    for (int i = 0; i < K; ++i) { key[i] = 0u; idx[i] = 0x7FFFFFFF; }
  }
  __device__ __forceinline__ void place(uint32_t c, int ci, const bool (&gt)[K]) {
#pragma unroll
    for (int i = K - 1; i > 0; --i) {               // descending: place i - 1 still holds its old entry
      key[i] = gt[i] ? (gt[i - 1] ? key[i - 1] : c) : key[i];
      idx[i] = gt[i] ? (gt[i - 1] ? idx[i - 1] : ci) : idx[i];
    }
    key[0] = gt[0] ? c : key[0];
    idx[0] = gt[0] ? ci : idx[0];
  }
  __device__ __forceinline__ void push(float v, int e) {
    const uint32_t c = sel_float_key(v);
    bool gt[K];
#pragma unroll
    for (int i = 0; i < K; ++i) gt[i] = c > key[i];
    place(c, e, gt);
  }
  __device__ __forceinline__ static bool ahead(uint32_t a, int ai, uint32_t b, int bi) { return a > b || (a == b && ai < bi); }
  // the best K of this list and another, both best first: place by place the better of one list's i-th and the other's
  // (K - 1 - i)-th, which leaves a bitonic list to sort (K a power of two)
  __device__ __forceinline__ void merge(const uint32_t (&k2)[K], const int (&i2)[K]) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const bool other = ahead(k2[K - 1 - i], i2[K - 1 - i], key[i], idx[i]);
      key[i] = other ? k2[K - 1 - i] : key[i];
      idx[i] = other ? i2[K - 1 - i] : idx[i];
    }
#pragma unroll
    for (int s = K / 2; s > 0; s >>= 1)
#pragma unroll
      for (int i = 0; i < K; ++i)
        if ((i & s) == 0) {
          const bool swap = ahead(key[i + s], idx[i + s], key[i], idx[i]);
          const uint32_t ka = key[i], kb = key[i + s];
          const int ia = idx[i], ib = idx[i + s];
          key[i] = swap ? kb : ka; key[i + s] = swap ? ka : kb;
          idx[i] = swap ? ib : ia; idx[i + s] = swap ? ia : ib;
        }
  }
  // the lists of the lanes lane ^ 1, lane ^ 2, ... lane ^ (parts - 1) meet: afterwards every lane of the group holds
  // the best K of the group (parts a power of two, groups aligned in the warp; all 32 lanes must call)
  __device__ __forceinline__ void merge_lanes(int parts) {
    for (int m = 1; m < parts; m <<= 1) {
      uint32_t ok_[K];
      int oi[K];
#pragma unroll
      for (int i = 0; i < K; ++i) {
        ok_[i] = __shfl_xor_sync(0xFFFFFFFFu, key[i], m);
        oi[i] = __shfl_xor_sync(0xFFFFFFFFu, idx[i], m);
      }
      merge(ok_, oi);
    }
  }
};
