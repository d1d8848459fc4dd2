// Kernel parameter blocks shared by the dense (flash / piecewise) kernels and
// the host-side glue that fills them from the C ABI structs.
#pragma once

#include "common.cuh"

namespace fa {

struct Strides {
  int64_t b, h, l;
};

__host__ __device__ inline Strides strides_of(const fa_tensor4 *t) {
  return Strides{t->stride_b, t->stride_h, t->stride_l};
}

// Forward (flash, piecewise and split-KV stage 1).
struct FwdParams {
  const void *q, *k, *v, *q2, *k2;
  void *o;
  float *lse;
  Strides sq, sk, sv, sq2, sk2, so;
  int B, H, Hk, M, N;
  int causal;
  int w;  // piecewise distance threshold
  float sm_scale;
  // dropout (flash forward only): keep iff uniform(seed, offset + linear index) > dropout_p
  float dropout_p;
  uint64_t seed, offset;
  // split-KV
  int num_splits, n_split_size;
  float *o_partial;    // (B,H,S,M,D)
  float *lse_partial;  // (B,H,S,M)
};

// Backward (flash and piecewise).  In the flash kernels q2/k2/dq2/dk2 are unused.
struct BwdParams {
  const void *q, *k, *v, *q2, *k2, *d_o;
  const float *lse, *delta;
  void *dq, *dq2, *dk, *dk2, *dv;
  Strides sq, sk, sv, sq2, sk2, sdo, sdq, sdq2, sdk, sdk2, sdv;
  int B, H, Hk, M, N;
  int causal;
  int w;
  float sm_scale;
  float dropout_p;
  uint64_t seed, offset;
};

// First output word of Philox-4x32 with 6 rounds, counter (c0, c1, 0, 0), key (k0, k1).
__host__ __device__ __forceinline__ uint32_t philox4x32_6(uint32_t k0, uint32_t k1, uint32_t c0,
                                                          uint32_t c1) {
  uint32_t c2 = 0, c3 = 0;
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    const uint32_t a0 = c0, a2 = c2;
    const uint64_t pb = (uint64_t)0xCD9E8D57u * a2, pa = (uint64_t)0xD2511F53u * a0;
    c0 = (uint32_t)(pb >> 32) ^ c1 ^ k0;
    c2 = (uint32_t)(pa >> 32) ^ c3 ^ k1;
    c1 = (uint32_t)pb;
    c3 = (uint32_t)pa;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c0;
}
// Dropout decision of attention element `idx` (= ((b*H + h)*M + m)*N + n): true = keep.
__host__ __device__ __forceinline__ bool dropout_keep(uint64_t seed, uint64_t offset, uint64_t idx,
                                                      float dropout_p) {
  const uint64_t ctr = offset + idx;
  int32_t x = (int32_t)philox4x32_6((uint32_t)seed, (uint32_t)(seed >> 32), (uint32_t)ctr,
                                    (uint32_t)(ctr >> 32));
  if (x < 0) x = -x - 1;
  return (float)x * 4.6566127342e-10f > dropout_p;
}

// ---- the same decision for the tcgen05 kernels ----
// dropout_keep() as one unsigned range check: with x = u or ~u of the Philox word u (whichever is not
// negative), (float)x * c > dropout_p holds from some smallest x = t on, hence for u in [t, 2^32 - t).
// t by bisection with the very float operations of dropout_keep(); no x satisfies it: an empty range.
struct DropoutRule {
  uint64_t seed, offset;
  uint32_t first, width;   // keep iff u - first < width
  float rp;                // 1 / (1 - dropout_p)
  // Where the forward leaves the decisions for the backward (null: nowhere, the backward draws again): bit n % 32 of
  // word ((b * H + h) * words + n / 32) * rows + m, 1 = keep.  rows: M rounded up to 128, words: N / 32 rounded up to 4.
  uint32_t *bits;
  int rows, words;
};
inline DropoutRule make_dropout_rule(float dropout_p, uint64_t seed, uint64_t offset) {
  uint64_t lo = 0, hi = 1ull << 31;   // smallest x in [lo, hi] that is kept (2^31: none)
  while (lo < hi) {
    const uint64_t mid = (lo + hi) / 2;
    const volatile float u = (float)(int32_t)mid * 4.6566127342e-10f;
    if (u > dropout_p) hi = mid;
    else lo = mid + 1;
  }
  return DropoutRule{seed, offset, (uint32_t)lo, (uint32_t)(0u - 2u * (uint32_t)lo), 1.f / (1.f - dropout_p), nullptr, 0, 0};
}

// The buffer of a call: B H words rows 4-byte words.  Kept while it takes no more memory than q and o together (N / 8
// bytes a query row against 4 D): up to 32 D keys.
inline int64_t keep_bits_bytes(const fa_flash_shape *s) {
  if (!(s->dropout_p > 0.f) || s->N > 32 * s->D) return 0;
  return (int64_t)s->B * s->H * ((s->N + 127) / 128 * 4) * (((int64_t)s->M + 127) / 128 * 128) * 4;
}
inline void keep_bits_in(DropoutRule &r, const fa_flash_shape *s, void *bits) {
  r.bits = static_cast<uint32_t *>(bits);
  r.rows = (s->M + 127) / 128 * 128, r.words = (s->N + 127) / 128 * 4;
}

// Keep bits of the elements whose counters are ctr + at(0), ctr + at(1), .. ctr + at(31) (bit i: the i-th), none
// larger than `most`.
// What bounds a kernel with dropout is this: Philox costs 10 multiplications an element and only its first output word
// is used.  While the counters share their upper 32 bits (all but one in 2^32 / most calls) one product of round 2
// depends on nothing else and is taken out of the loop; words of rounds 4 to 6 that do not reach the first output are
// not computed: 9 multiplications and 9 three-input xors an element.
template <typename At>
__device__ __forceinline__ uint32_t dropout_keep_bits32(const DropoutRule &r, uint64_t ctr, uint64_t most, At at) {
  constexpr uint32_t A = 0xD2511F53u, B = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  const uint32_t k0 = (uint32_t)r.seed, k1 = (uint32_t)(r.seed >> 32);
  const uint32_t lo = (uint32_t)ctr;
  uint32_t bits = 0;
  if ((uint64_t)lo + most >> 32) {   // the upper half of the counter changes on the way
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {
      const uint64_t c = ctr + at(i);
      const uint32_t u = philox4x32_6(k0, k1, (uint32_t)c, (uint32_t)(c >> 32));
      if (u - r.first < r.width) bits |= 1u << i;
    }
    return bits;
  }
  const uint64_t fixed = (uint64_t)A * ((uint32_t)(ctr >> 32) ^ k0);   // round 2
  const uint32_t fx = (uint32_t)(fixed >> 32) ^ (k1 + W1), fy = (uint32_t)fixed ^ (k1 + 2u * W1);
#pragma unroll 8
  for (int i = 0; i < 32; ++i) {
    uint64_t pa = (uint64_t)A * (lo + (uint32_t)at(i));   // round 1
    uint32_t c2 = (uint32_t)(pa >> 32) ^ k1;
    uint64_t pb = (uint64_t)B * c2;   // round 2
    uint32_t c0 = (uint32_t)(pb >> 32) ^ (k0 + W0), c1 = (uint32_t)pb;
    c2 = (uint32_t)pa ^ fx;
    pb = (uint64_t)B * c2, pa = (uint64_t)A * c0;   // round 3
    c0 = (uint32_t)(pb >> 32) ^ c1 ^ (k0 + 2u * W0);
    c2 = (uint32_t)(pa >> 32) ^ fy;
    const uint32_t c3 = (uint32_t)pa;
    pa = (uint64_t)A * c0;   // round 4
    c0 = __umulhi(B, c2) ^ (uint32_t)pb ^ (k0 + 3u * W0);
    c2 = (uint32_t)(pa >> 32) ^ c3 ^ (k1 + 3u * W1);
    const uint32_t d2 = __umulhi(A, c0) ^ (uint32_t)pa ^ (k1 + 4u * W1);   // round 5
    const uint32_t u = __umulhi(B, d2) ^ (B * c2) ^ (k0 + 5u * W0);        // round 6
    if (u - r.first < r.width) bits |= 1u << i;
  }
  return bits;
}

template <typename T>
__device__ __forceinline__ const T *row_ptr(const void *base, const Strides &s, int b, int h,
                                            int l) {
  return reinterpret_cast<const T *>(base) + (int64_t)b * s.b + (int64_t)h * s.h +
         (int64_t)l * s.l;
}
template <typename T>
__device__ __forceinline__ T *row_ptr_mut(void *base, const Strides &s, int b, int h, int l) {
  return reinterpret_cast<T *>(base) + (int64_t)b * s.b + (int64_t)h * s.h + (int64_t)l * s.l;
}

// Which score branch a (BM x BN) tile needs under the piecewise rule
// "branch 2 iff (m + P_SEQ) - n >= w".
struct PwClass {
  bool need1, need2;
};
__device__ __forceinline__ PwClass pw_classify(int m0, int rows, int n0, int cols, int p_seq,
                                               int w) {
  int dmin = m0 + p_seq - (n0 + cols - 1);
  int dmax = m0 + rows - 1 + p_seq - n0;
  PwClass c;
  c.need2 = dmax >= w;  // some element is far
  c.need1 = dmin < w;   // some element is near
  return c;
}

}  // namespace fa
