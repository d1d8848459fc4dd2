// Launcher of the tcgen05 total_attention kernel.
#include "total_attn_tc.cuh"
#include "tma_host.cuh"
#include "../common.cuh"

namespace fa {
int *device_status_word();

namespace tc {

bool generic_forced();

template <typename T, int D, bool PAIRS_FIRST>
static int launch_total_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                           const float *lse, float *total, cudaStream_t stream) {
  using C = TotalTcCfg<D>;
  CUtensorMap mq, mk;
  if (!make_map_bhld(&mq, q, s->dtype, s->B, s->H, s->M, s->D, C::BM) ||
      !make_map_bhld(&mk, k, s->dtype, s->B, s->Hk, s->N, s->D, C::BN))
    return 1;   // layout not expressible as a tensor map: the caller uses the generic kernel
  auto kern = total_attention_tc_kernel<T, D, PAIRS_FIRST>;
  static unsigned long long done = 0;
  if (int st = ensure_dyn_smem(kern, C::kTotal, &done)) return st;
  TotalTcParams p{};
  p.lse = lse, p.total = total;
  p.B = s->B, p.H = s->H, p.Hk = s->Hk, p.M = s->M, p.N = s->N;
  p.causal = s->causal, p.sm_scale = s->sm_scale;
  p.status = device_status_word();
  const int pairs = s->B * s->H, blocks = (s->N + C::BN - 1) / C::BN;
  const dim3 grid = PAIRS_FIRST ? dim3(pairs, blocks) : dim3(blocks, pairs);
  kern<<<grid, C::kThreads, C::kTotal, stream>>>(mq, mk, p);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

// Returns FA_OK / a negative status, or 1 when this path does not cover the call.
int total_attention_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                       const float *lse, float *total, cudaStream_t stream) {
  if (generic_forced() || !(s->sm_scale > 0.f)) return 1;
  // head_dim 16 and 32, padded to 64: bf16 causal, shape-generic -> this, us: 16: B=16 H=16 L=512 27.8 -> 34.3, L=896
  // 64.7 -> 69.4, B=4 H=16 L=1024 31 -> 26, L=2048 87 -> 65, M=64 N=4096 12.4 -> 44.7; 32: L=896 65.8 -> 69.2,
  // L=2048 91 -> 65.
  if (s->D < 64 && s->M < 1024) return 1;
  // The CTAs of a (batch, head) pair share its Q and lse.  Heaviest blocks of all pairs first where that fits in L2
  // (see forward_group_size()).
  const bool first = (s->N + 127) / 128 <= 65535 &&
                     one_group_in_l2((int64_t)s->M * ((s->D == 128 ? 128 : 64) * 2 + 4), s->B * s->H, s->causal);
#define FA_TOTAL(T, D) \
  (first ? launch_total_tc<T, D, true>(s, q, k, lse, total, stream) : launch_total_tc<T, D, false>(s, q, k, lse, total, stream))
  if (s->dtype == FA_F16) return s->D == 128 ? FA_TOTAL(__half, 128) : FA_TOTAL(__half, 64);
  return s->D == 128 ? FA_TOTAL(__nv_bfloat16, 128) : FA_TOTAL(__nv_bfloat16, 64);
#undef FA_TOTAL
}

}  // namespace tc
}  // namespace fa
