// C ABI entry points of the flash_attention forward: the one-pass kernel, the
// split-KV two-stage path for decode-shaped M, and the split-count heuristic.
#include <cmath>

#include "dense_fwd.cuh"
#include "dense_host.cuh"

namespace fa {

template <int D>
struct FwdTile {
  static constexpr int BM = 128;
  static constexpr int BN = 64;
};
struct SplitTile {
  static constexpr int BM = 64;
  static constexpr int BN = 64;
};

struct FwdLaunch {
  FwdParams p;
  cudaStream_t stream;
  template <typename T, int D>
  int operator()() const {
    constexpr int BM = FwdTile<D>::BM, BN = FwdTile<D>::BN;
    using L = FwdSmemLayout<D, BM, BN, false>;
    auto kern = dense_fwd_kernel<T, D, BM, BN, false, false>;
    static unsigned long long done = 0;
    if (int st = ensure_dyn_smem(kern, L::kTotal, &done)) return st;
    dim3 grid((p.M + BM - 1) / BM, p.B * p.H, 1);
    kern<<<grid, BM / 16 * 32, L::kTotal, stream>>>(p);
    FA_CHECK_LAUNCH();
    return FA_OK;
  }
};

struct SplitLaunch {
  FwdParams p;
  cudaStream_t stream;
  template <typename T, int D>
  int operator()() const {
    constexpr int BM = SplitTile::BM, BN = SplitTile::BN;
    using L = FwdSmemLayout<D, BM, BN, false>;
    auto kern = dense_fwd_kernel<T, D, BM, BN, false, true>;
    static unsigned long long done = 0;
    if (int st = ensure_dyn_smem(kern, L::kTotal, &done)) return st;
    dim3 grid((p.M + BM - 1) / BM, p.B * p.H, p.num_splits);
    kern<<<grid, BM / 16 * 32, L::kTotal, stream>>>(p);
    FA_CHECK_LAUNCH();
    return FA_OK;
  }
};

static FwdParams make_fwd_params(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                                 const fa_tensor4 *v) {
  FwdParams p{};
  p.q = q->ptr, p.k = k->ptr, p.v = v->ptr;
  p.sq = strides_of(q), p.sk = strides_of(k), p.sv = strides_of(v);
  p.B = s->B, p.H = s->H, p.Hk = s->Hk, p.M = s->M, p.N = s->N;
  p.causal = s->causal, p.sm_scale = s->sm_scale;
  p.dropout_p = s->dropout_p, p.seed = s->philox_seed, p.offset = s->philox_offset;
  p.num_splits = 1;
  return p;
}

namespace tc {
int flash_fwd_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                 const fa_tensor4 *v, const fa_tensor4 *o, float *lse, cudaStream_t stream, void *bits);
int flash_fwd_fine_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k, const fa_tensor4 *v,
                      const fa_tensor4 *o, float *lse, cudaStream_t stream);
double fine_microseconds(const fa_flash_shape *s, int sms);
}

}  // namespace fa

using namespace fa;

extern "C" int fa_flash_fwd(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                            const fa_tensor4 *v, const fa_tensor4 *o, float *lse, void *stream) {
  if (int st = validate_shape(s)) return st;
  if (int st = validate_tensors({q, k, v, o})) return st;
  if (!lse) return FA_ERR_BAD_ARG;
  // what a tensor map can express runs on tcgen05; everything else on the shape-generic kernel
  const int tc_status = tc::flash_fwd_tc(s, q, k, v, o, lse, static_cast<cudaStream_t>(stream), nullptr);
  if (tc_status <= 0) return tc_status;
  FwdParams p = make_fwd_params(s, q, k, v);
  p.o = o->ptr, p.so = strides_of(o), p.lse = lse;
  return dispatch_dtype_d(s->dtype, s->D, FwdLaunch{p, static_cast<cudaStream_t>(stream)});
}

extern "C" int fa_flash_fwd_keep(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                                 const fa_tensor4 *v, const fa_tensor4 *o, float *lse, void *bits, int64_t bits_bytes,
                                 void *stream) {
  if (int st = validate_shape(s)) return st;
  if (int st = validate_tensors({q, k, v, o})) return st;
  if (!lse || !bits || (reinterpret_cast<uintptr_t>(bits) & 15)) return FA_ERR_BAD_ARG;
  const int64_t need = fa_flash_keep_bits_bytes(s);
  if (need == 0) return FA_ERR_UNSUPPORTED;
  if (bits_bytes < need) return FA_ERR_WORKSPACE;
  const int tc_status = tc::flash_fwd_tc(s, q, k, v, o, lse, static_cast<cudaStream_t>(stream), bits);
  return tc_status == 1 ? FA_ERR_UNSUPPORTED : tc_status;   // 1: nothing launched
}

extern "C" int fa_flash_fwd_few_rows(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                                     const fa_tensor4 *v, const fa_tensor4 *o, float *lse, void *stream) {
  if (int st = validate_shape(s)) return st;
  if (int st = validate_tensors({q, k, v, o})) return st;
  if (!lse) return FA_ERR_BAD_ARG;
  if (s->M < 32) return FA_ERR_UNSUPPORTED;   // H=4 M=17 N=131072 157 -> 192 us
  const int tc_status = tc::flash_fwd_fine_tc(s, q, k, v, o, lse, static_cast<cudaStream_t>(stream));
  return tc_status == 1 ? FA_ERR_UNSUPPORTED : tc_status;   // 1: nothing launched
}

// The split-KV kernels give a query tile of 64 rows to as many CTAs as the heuristic says, at 0.67 / 0.81 / 1.17 us a tile
// of 64 keys (head_dim up to 32 / 64 / 128), and then combine; the cluster form has tiles of 128 rows, at most 8 CTAs each and
// one launch.  The rule is the smaller of two fits (260 calls of 32..400 queries, each 5 % off).  bf16, split-KV -> cluster, us:
//   taken    H=8 M=32 N=16384 D=128 43.7 -> 30.2, H=4 M=128 N=16384 79.8 -> 31.4, H=16 M=64 N=4096 43.6 -> 17.4,
//            H=12 M=88 N=11400 109 -> 24.4, H=2 M=45 N=180 D=128 8.2 -> 6.9
//   refused  H=3 M=37 N=424 D=64 6.9 -> 9.0, H=1 M=41 N=8859 D=64 14.8 -> 19.0, H=1 M=222 N=921 D=64 8.1 -> 9.7,
//            H=4 M=46 N=9570 D=32 16.7 -> 19.2, B=8 H=4 M=37 N=346 D=64 8.0 -> 8.9, H=4 M=32 N=1000 9.1 -> 10.9
extern "C" int32_t fa_flash_few_rows_pays(const fa_flash_shape *s, int32_t num_sms) {
  if (validate_shape(s) != FA_OK || s->M < 32 || s->dropout_p > 0.f || num_sms <= 0) return 0;
  const double cluster = tc::fine_microseconds(s, num_sms);
  if (cluster <= 0.0) return 0;
  const int splits = fa_num_splits_heuristic(s->B, s->H, s->M, s->N, 16, 128, num_sms, 128);
  const int tiles = (s->N + SplitTile::BN - 1) / SplitTile::BN, per_split = (tiles + splits - 1) / splits;
  const double used = (tiles + per_split - 1) / per_split;
  const double fixed = s->D == 128 ? 5.65 : (s->D == 64 ? 4.9 : 4.65), a_tile = s->D == 128 ? 1.17 : (s->D == 64 ? 0.81 : 0.67);
  return cluster < fixed + a_tile * per_split + 0.166 * used;
}

extern "C" int fa_splitkv_fwd(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                              const fa_tensor4 *v, int32_t num_splits, int32_t n_split_size,
                              float *o_partial, float *lse_partial, void *stream) {
  if (int st = validate_shape(s)) return st;
  if (int st = validate_tensors({q, k, v})) return st;
  if (!o_partial || !lse_partial) return FA_ERR_WORKSPACE;
  if (s->dropout_p > 0.f) return FA_ERR_UNSUPPORTED;  // no dropout on the split-KV path
  if (num_splits < 1 || num_splits > 65535 || n_split_size <= 0 ||
      n_split_size % SplitTile::BN != 0)
    return FA_ERR_BAD_ARG;
  if ((int64_t)num_splits * n_split_size < s->N) return FA_ERR_BAD_ARG;
  FwdParams p = make_fwd_params(s, q, k, v);
  p.num_splits = num_splits, p.n_split_size = n_split_size;
  p.o_partial = o_partial, p.lse_partial = lse_partial;
  return dispatch_dtype_d(s->dtype, s->D, SplitLaunch{p, static_cast<cudaStream_t>(stream)});
}

extern "C" int fa_splitkv_combine(const fa_flash_shape *s, int32_t num_splits,
                                  const float *o_partial, const float *lse_partial,
                                  const fa_tensor4 *o, float *lse, void *stream) {
  if (int st = validate_shape(s)) return st;
  if (int st = validate_tensors({o})) return st;
  if (!o_partial || !lse_partial) return FA_ERR_WORKSPACE;
  if (!lse || num_splits < 1) return FA_ERR_BAD_ARG;
  const int64_t total = (int64_t)s->B * s->H * s->M * (s->D / 4);
  const int threads = 256;
  const int blocks = (int)std::min<int64_t>((total + threads - 1) / threads, 148 * 16);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s->dtype == FA_F16)
    splitkv_combine_kernel<__half><<<blocks, threads, 0, st>>>(
        o_partial, lse_partial, o->ptr, strides_of(o), lse, s->B, s->H, s->M, s->D, num_splits);
  else
    splitkv_combine_kernel<__nv_bfloat16><<<blocks, threads, 0, st>>>(
        o_partial, lse_partial, o->ptr, strides_of(o), lse, s->B, s->H, s->M, s->D, num_splits);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

extern "C" int64_t fa_splitkv_workspace_bytes(const fa_flash_shape *s, int32_t num_splits) {
  if (!s || num_splits < 1) return 0;
  const int64_t rows = (int64_t)s->B * s->H * num_splits * s->M;
  return rows * s->D * 4 + rows * 4;
}

// Restates src/flag_attn/split_kv.py:234-262: no split when the unsplit grid
// already fills 80% of the SMs; otherwise the smallest split count whose wave
// efficiency is within 85% of the best one, among counts that leave no split
// empty.
extern "C" int32_t fa_num_splits_heuristic(int32_t B, int32_t H, int32_t M, int32_t N,
                                           int32_t block_m, int32_t block_n, int32_t num_sms,
                                           int32_t max_splits) {
  const int64_t blocks = (int64_t)B * H * ((M + block_m - 1) / block_m);
  if ((double)blocks >= 0.8 * num_sms) return 1;
  const int n_blocks = (N + block_n - 1) / block_n;
  max_splits = std::min(std::min(num_sms, n_blocks), max_splits);
  auto available = [&](int sp) {
    const int per = (n_blocks + sp - 1) / sp;
    return sp == 1 || (per * sp - n_blocks < per);
  };
  auto efficiency = [&](int sp) {
    const double waves = (double)(blocks * sp) / num_sms;
    return waves / std::ceil(waves);
  };
  double best = 0.0;
  for (int sp = 1; sp <= max_splits; ++sp)
    if (available(sp)) best = std::max(best, efficiency(sp));
  for (int sp = 1; sp <= max_splits; ++sp)
    if (available(sp) && efficiency(sp) >= 0.85 * best) return sp;
  return 1;
}
