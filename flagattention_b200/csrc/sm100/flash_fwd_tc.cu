// Launcher of the tcgen05 flash_attention forward.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "flash_fwd_tc.cuh"
#include "flash_fwd_persist_tc.cuh"
#include "tma_host.cuh"
#include "../common.cuh"
#include "../dense_host.cuh"

namespace fa {
int *device_status_word();

namespace tc {

// Kernel family switch (fa_set_kernel_family): 0 = tcgen05 kernels wherever they cover the call,
// 1 = shape-generic kernels only.  The environment variable FLAGATTN_B200_GENERIC=1 only sets the
// value the process starts with.
static std::atomic<int> g_kernel_family{[] {
  const char *e = std::getenv("FLAGATTN_B200_GENERIC");
  return (e && e[0] == '1') ? 1 : 0;
}()};
bool generic_forced() { return g_kernel_family.load(std::memory_order_relaxed) == 1; }
// family 2 (test suites, A/B timing): tcgen05 kernels, but the forward with one CTA per query tile
static bool one_cta_per_tile_forced() { return g_kernel_family.load(std::memory_order_relaxed) == 2; }
int set_kernel_family(int family) {
  return g_kernel_family.exchange(family == 1 ? 1 : (family == 2 ? 2 : 0));
}

// CTAs that share the walk of a query tile (SPLIT): 1, 2, 4 or 8, and the estimated time in tiles.  One CTA walks a 64-key
// tile in 0.62 us (0.66 at head_dim 128), so an SM with a single CTA, or none, is idle for want of query tiles.  Sharing
// costs the set-up and the combining, 3.75 tiles (4.25).  The CTAs of a cluster take SMs of their own while there are
// any: 74 clusters of 2, 33 of 4, 15 of 8.  Beyond that two share an SM, which costs a quarter of their walk and up to
// 2.4 tiles (3.6: 64 KB of O a CTA; less where most walks are shorter), and beyond twice that (33 of 8) a cluster waits
// for another.  Taken where it saves a tenth; two CTAs may also share a walk where the longest is about twice the mean
// load.  us at 1 / 2 / 4 / 8 CTAs, bf16:
//   H=32 Hk=8 M=512 N=7300 D=128 (128 query tiles of 107..115 key tiles)   83.4 / 62.2 / 70.6 / 86.6
//   H=32 Hk=8 M=64 N=7300 D=128 (32 of 115)    82.1 / 47.7 / 28.4 / 25.4
//   H=8 M=1024 N=16384 D=128 (64 of 256)       185 / 99 / 69 / 79
//   H=4 L=1024 D=128 causal (32 of 2..16)      16.1 / 13.7 / 11.2 / 14.4
//   H=4 L=512 D=64 causal (16 of 2..8)          9.9 /  9.6 /  8.3 /  9.6
//   B=2 H=4 L=256 D=64 causal (16 of 2..4)      7.1 /  8.2 /  7.5 /  9.6
//   H=32 Hk=8 M=1024 N=4096 D=128 (256 of 50..64)  59.0 / 69.4 / 85.0 / 118
//   H=4 L=8192 D=128 causal (256 of 2..128)    96.4 / 78.8 / 91.0 / 125
//   H=12 L=4096 D=128 causal (384 of 2..64)    56.6 / 69.5 / 90.6 / 145
// and where clusters are too many to run at once or CTAs share SMs for short walks (1 / 2 / 4 / 8):
//   H=8 Hk=1 L=1152 D=128 causal (72 of 2..18)     16.8 / 14.1 / 19.0
//   H=3 B=2 L=1536 D=64 not causal (72 of 24)      19.0 / 14.3 / 20.3
//   H=3 M=3072 N=3170 D=128 causal (72 of 4..50)   37.2 / 24.5 / 23.0
//   H=3 L=1536 D=64 not causal (36 of 24)          19.2 / 13.9 / 13.0 / 16.6
//   B=2 H=8 L=1115 D=128 not causal (144 of 18)    17.4 / 19.1
struct KeySplit {
  int ctas;
  double tiles;
};
static KeySplit key_split(const fa_flash_shape *s, int sms) {
  const int64_t blocks = (s->M + 127) / 128, ctas = blocks * s->B * s->H;
  const int64_t longest = (s->N + 63) / 64;
  // key tiles of the last query tile and, roughly, of the first
  const int64_t shortest = s->causal ? std::max<int64_t>(0, ((int64_t)s->N - s->M + 128 + 63) / 64) : longest;
  const double mean = 0.5 * (double)(longest + std::min(shortest, longest)), pair = 1.0 + 0.25 * mean / (double)longest;
  KeySplit best{1, (double)longest * (ctas > sms ? pair : 1.0)};
  if (sms <= 0 || ctas > 2ll * sms) return best;
  const bool wide = s->D == 128;
  const int64_t alone[3] = {sms / 2, sms * 33 / 148, sms * 15 / 148};   // clusters of 2, 4 and 8 on SMs of their own
  double least = 0.9 * best.tiles;
  for (int i = 0, c = 2; c <= 8 && ctas * c <= 2ll * sms; ++i, c *= 2) {
    const bool share = ctas > alone[i];
    double tiles = (double)longest / c * (share ? pair : 1.0) + (wide ? 4.25 : 3.75) + (share ? (wide ? 3.6 : 2.4) * mean / (double)longest : 0.0);
    if (c == 8 && ctas > alone[1]) break;                       // (two an SM: a cluster of 8 takes four SMs)
    if (c < 8 && ctas > 2 * alone[i]) tiles += mean / c + 0.5;   // the last clusters follow others
    if (tiles < least) best = KeySplit{c, tiles}, least = tiles;
  }
  const double load = (double)ctas * mean / (2.0 * sms);
  if (best.ctas == 1 && longest >= 64 && load <= 0.55 * (double)longest) best.ctas = 2;
  return best;
}

template <typename T, int D, bool PW, bool DROP = false, bool PAD = false>
static int launch_fwd_tc(const fa_flash_shape *s, int w, const fa_tensor4 *q, const fa_tensor4 *k,
                         const fa_tensor4 *q2, const fa_tensor4 *k2, const fa_tensor4 *v,
                         const fa_tensor4 *o, float *lse, cudaStream_t stream, void *bits = nullptr) {
  using C = FwdTcCfg<D>;
  CUtensorMap mq, mk, mv, mq2, mk2;
  if (!make_map_bhld(&mq, q, s->dtype, s->B, s->H, s->M, s->D, C::BM) ||
      !make_map_bhld(&mk, k, s->dtype, s->B, s->Hk, s->N, s->D, C::BN) ||
      !make_map_bhld(&mv, v, s->dtype, s->B, s->Hk, s->N, s->D, C::BN))
    return 1;  // layout not expressible as a tensor map: caller falls back to the generic kernel
  mq2 = mq, mk2 = mk;
  if (PW && (!make_map_bhld(&mq2, q2, s->dtype, s->B, s->H, s->M, s->D, C::BM) ||
             !make_map_bhld(&mk2, k2, s->dtype, s->B, s->Hk, s->N, s->D, C::BN)))
    return 1;
  FwdTcParams p{};
  p.o = o->ptr, p.lse = lse, p.so = strides_of(o);
  p.B = s->B, p.H = s->H, p.Hk = s->Hk, p.M = s->M, p.N = s->N;
  p.causal = s->causal, p.sm_scale = s->sm_scale, p.w = w;
  p.status = device_status_word();
  p.d = s->D;
  if (DROP) {
    p.drop = make_dropout_rule(s->dropout_p, s->philox_seed, s->philox_offset);
    if (bits) keep_bits_in(p.drop, s, bits);
  }
  // the CTAs of a (batch, head) pair share its K and V (and K2 under piecewise), with those of its group's heads
  p.num_m_blocks = (s->M + C::BM - 1) / C::BM;
  p.group_size = forward_group_size((int64_t)s->N * D * 2 * (PW ? 3 : 2) * s->Hk / s->H, s->B * s->H, s->causal,
                                    p.num_m_blocks, D == 128);
  const int64_t tiles = (int64_t)p.num_m_blocks * s->B * s->H;
  p.split = DROP || one_cta_per_tile_forced() ? 1 : key_split(s, sm_count_of_device()).ctas;
  if constexpr (!DROP) {
    if (p.split > 1) {
      auto kern = flash_fwd_tc_kernel<T, D, PW, DROP, PAD, true>;
      static unsigned long long done = 0;
      if (int st = ensure_dyn_smem(kern, C::kTotal, &done)) return st;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = (unsigned)p.split, attr.val.clusterDim.y = 1, attr.val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)(tiles * p.split), 1, 1), cfg.blockDim = dim3(C::kThreads, 1, 1);
      cfg.dynamicSmemBytes = C::kTotal, cfg.stream = stream, cfg.attrs = &attr, cfg.numAttrs = 1;
      if (cudaLaunchKernelEx(&cfg, kern, mq, mk, mv, mq2, mk2, p) != cudaSuccess) return FA_ERR_LAUNCH;
      FA_CHECK_LAUNCH();
      return FA_OK;
    }
  }
  auto kern = flash_fwd_tc_kernel<T, D, PW, DROP, PAD>;
  static unsigned long long done = 0;
  if (int st = ensure_dyn_smem(kern, C::kTotal, &done)) return st;
  kern<<<dim3((unsigned)tiles, 1, 1), C::kThreads, C::kTotal, stream>>>(mq, mk, mv, mq2, mk2, p);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

// Work-item counters of the persistent forward.  The forward entry points take no workspace, so
// the counters live in the library: a table of 64 words per device, one word per launch, taken
// round-robin, zeroed by a four-byte stream-ordered memset in front of the launch (a launch also
// puts its word back to zero with its last fetch, but one that gives up on a wait leaves it mid-way).
// A word is only touched while its kernel runs, so two launches collide only if 64 later launches
// start while the first still runs.
static __device__ unsigned g_fwd_sched[64];
static unsigned *fwd_sched_table() {
  static std::atomic<unsigned *> base[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  unsigned *b = base[dev].load(std::memory_order_acquire);
  if (!b) {
    void *ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_fwd_sched) != cudaSuccess) return nullptr;
    b = static_cast<unsigned *>(ptr);
    base[dev].store(b, std::memory_order_release);
  }
  return b;
}
static unsigned *fwd_sched_slot() {
  static std::atomic<unsigned> next{0};
  unsigned *b = fwd_sched_table();
  return b ? b + (next.fetch_add(1u, std::memory_order_relaxed) & 63u) : nullptr;
}
int reset_fwd_sched() {
  unsigned *b = fwd_sched_table();
  if (!b) return FA_ERR_LAUNCH;
  return cudaMemset(b, 0, 64 * sizeof(unsigned)) == cudaSuccess ? FA_OK : FA_ERR_LAUNCH;
}


// The persistent form (flash_fwd_persist_tc.cuh): two CTAs per SM that work through the query tiles.
template <typename T, int D, bool PAD = false>
static int launch_fwd_persist(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                              const fa_tensor4 *v, const fa_tensor4 *o, float *lse, cudaStream_t stream) {
  using C = FwdPersistCfg<D>;
  CUtensorMap mq, mk, mv;
  if (!make_map_bhld(&mq, q, s->dtype, s->B, s->H, s->M, s->D, C::BM) ||
      !make_map_bhld(&mk, k, s->dtype, s->B, s->Hk, s->N, s->D, C::BN) ||
      !make_map_bhld(&mv, v, s->dtype, s->B, s->Hk, s->N, s->D, C::BN))
    return 1;
  auto kern = flash_fwd_persist_tc_kernel<T, D, PAD>;
  static unsigned long long done = 0;
  if (int st = ensure_dyn_smem(kern, C::kTotal, &done)) return st;
  FwdPersistParams fp{};
  FwdTcParams &p = fp.base;
  p.o = o->ptr, p.lse = lse, p.so = strides_of(o);
  p.B = s->B, p.H = s->H, p.Hk = s->Hk, p.M = s->M, p.N = s->N;
  p.causal = s->causal, p.sm_scale = s->sm_scale, p.w = 0;
  p.status = device_status_word();
  p.d = s->D;
  p.num_m_blocks = (s->M + C::BM - 1) / C::BM;
  p.group_size = forward_group_size((int64_t)s->N * D * 2 * 2 * s->Hk / s->H, s->B * s->H, s->causal,
                                    p.num_m_blocks, D == 128);
  const int64_t items = (int64_t)p.num_m_blocks * s->B * s->H;
  const int sms = sm_count_of_device();
  fp.sched = fwd_sched_slot();
  if (items <= 0 || items > (1ll << 30) || sms <= 0 || !fp.sched) return 1;
  fp.num_items = (int)items;
  dim3 grid((unsigned)(items < 2 * sms ? items : 2 * sms), 1, 1);
  if (cudaMemsetAsync(fp.sched, 0, sizeof(unsigned), stream) != cudaSuccess) return FA_ERR_LAUNCH;
  kern<<<grid, C::kThreads, C::kTotal, stream>>>(mq, mk, mv, fp);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

// head_dim 16 and 32 run as 64 with zero columns: the exponentials bound these kernels, not the padded products.
// Short walks do not pay for it.  bf16 causal, shape-generic -> padded, us:
//   32            B=16 H=16 L=160 13.8 -> 16.9, B=2 H=8 L=256 7.1 -> 7.4, B=16 H=16 Hk=4 L=512 43 -> 38, B=4 H=16 L=2048
//                 122 -> 84, B=4 H=16 M=2048 N=64 12.8 -> 17.4
//   32 piecewise  B=2 H=8 L=512 13.8 -> 14.8, B=4 H=16 L=1024 50 -> 42, L=2048 140 -> 95
//   32 dropout    B=2 H=8 L=128 10.5 -> 11.1, B=16 H=16 L=512 140 -> 119
//   16            B=1 H=4 L=1536 20.9 -> 21.6, B=4 H=16 L=1024 31 -> 33, L=2048 86 -> 84, B=1 H=8 L=4096 65 -> 54
//   16 piecewise  B=4 H=16 L=1024 40 -> 42, L=2048 109 -> 95
//   16 dropout    B=4 H=16 L=1024 139 -> 114
static int fewest_keys(const fa_flash_shape *s, bool piecewise) {
  if (s->D > 32) return 0;
  if (s->dropout_p > 0.f) return s->D == 32 ? 160 : 1024;
  if (piecewise) return s->D == 32 ? 640 : 1280;
  return s->D == 32 ? 384 : 2048;
}
static bool covered(const fa_flash_shape *s, bool piecewise = false) {
  return !generic_forced() && s->sm_scale > 0.f && s->N >= fewest_keys(s, piecewise);
}
// Estimated time of flash_fwd_fine_tc(), 0 for a shape that it leaves: a fit of 260 calls (5 % off, standard deviation).
double fine_microseconds(const fa_flash_shape *s, int sms) {
  if (s->N < fewest_keys(s, false)) return 0.0;
  return (s->D == 128 ? 4.8 : 3.95) + 0.725 * key_split(s, sms).tiles;
}

// Calls of few rows, which went to the split-KV kernels: those follow the row maximum exactly, so P goes in with its
// remainder here.  Return values as below.
int flash_fwd_fine_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k, const fa_tensor4 *v,
                      const fa_tensor4 *o, float *lse, cudaStream_t stream) {
  if (!covered(s) || s->dropout_p > 0.f) return 1;
  if (s->dtype == FA_F16)
    return s->D == 128 ? launch_fwd_tc<__half, 128, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream)
                       : launch_fwd_tc<__half, 64, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream);
  return s->D == 128 ? launch_fwd_tc<__nv_bfloat16, 128, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream)
                     : launch_fwd_tc<__nv_bfloat16, 64, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream);
}

// Return FA_OK / a negative status, or 1 when this path does not cover the call.
int flash_fwd_tc(const fa_flash_shape *s, const fa_tensor4 *q, const fa_tensor4 *k,
                 const fa_tensor4 *v, const fa_tensor4 *o, float *lse, cudaStream_t stream, void *bits) {
  if (!covered(s)) return 1;
  // Dropout is bound by its random numbers (see dropout_keep_bits32()): one CTA per tile at every size.
  // Forward, p = 0.1, bf16 causal, mma.sync kernel -> this: B=16 H=16 Hk=4 L=512 D=64 165 -> 119 us, B=4 H=16 L=2048
  // D=64 541 -> 336 us, D=128 731 -> 343 us.
  if (s->dropout_p > 0.f) {
    if (s->dtype == FA_F16)
      return s->D == 128 ? launch_fwd_tc<__half, 128, false, true>(s, 0, q, k, q, k, v, o, lse, stream, bits)
                         : launch_fwd_tc<__half, 64, false, true>(s, 0, q, k, q, k, v, o, lse, stream, bits);
    return s->D == 128 ? launch_fwd_tc<__nv_bfloat16, 128, false, true>(s, 0, q, k, q, k, v, o, lse, stream, bits)
                       : launch_fwd_tc<__nv_bfloat16, 64, false, true>(s, 0, q, k, q, k, v, o, lse, stream, bits);
  }
  // More query tiles than CTA slots and short walks (or head_dim 64): the persistent kernel.  It
  // measured +3..5 % at N <= 1024 and at head_dim 64, but -10 % at head_dim 128 and N = 4096, -17 %
  // at 16384: its steady tile period is 1750-1840 clocks against 1534 of the one-CTA-per-tile
  // kernel (why is not known: starting the second CTA of every SM a fraction of a tile period late,
  // in case the two walked in step, changed nothing).
  const bool short_walks = s->D <= 64 || s->N <= 1536;
  if (!one_cta_per_tile_forced() && short_walks &&
      (int64_t)((s->M + 127) / 128) * s->B * s->H > 2 * (int64_t)sm_count_of_device()) {
    int st;
    if (s->D < 64)
      st = s->dtype == FA_F16 ? launch_fwd_persist<__half, 64, true>(s, q, k, v, o, lse, stream)
                              : launch_fwd_persist<__nv_bfloat16, 64, true>(s, q, k, v, o, lse, stream);
    else if (s->dtype == FA_F16)
      st = s->D == 128 ? launch_fwd_persist<__half, 128>(s, q, k, v, o, lse, stream)
                       : launch_fwd_persist<__half, 64>(s, q, k, v, o, lse, stream);
    else
      st = s->D == 128 ? launch_fwd_persist<__nv_bfloat16, 128>(s, q, k, v, o, lse, stream)
                       : launch_fwd_persist<__nv_bfloat16, 64>(s, q, k, v, o, lse, stream);
    if (st != 1) return st;
  }
  if (s->D < 64)
    return s->dtype == FA_F16
               ? launch_fwd_tc<__half, 64, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream)
               : launch_fwd_tc<__nv_bfloat16, 64, false, false, true>(s, 0, q, k, q, k, v, o, lse, stream);
  if (s->dtype == FA_F16)
    return s->D == 128 ? launch_fwd_tc<__half, 128, false>(s, 0, q, k, q, k, v, o, lse, stream)
                       : launch_fwd_tc<__half, 64, false>(s, 0, q, k, q, k, v, o, lse, stream);
  return s->D == 128 ? launch_fwd_tc<__nv_bfloat16, 128, false>(s, 0, q, k, q, k, v, o, lse, stream)
                     : launch_fwd_tc<__nv_bfloat16, 64, false>(s, 0, q, k, q, k, v, o, lse, stream);
}

int piecewise_fwd_tc(const fa_flash_shape *s, int w, const fa_tensor4 *q1, const fa_tensor4 *k1,
                     const fa_tensor4 *q2, const fa_tensor4 *k2, const fa_tensor4 *v,
                     const fa_tensor4 *o, float *lse, cudaStream_t stream) {
  if (!covered(s, true) || s->dropout_p > 0.f || w > (1 << 29) || w < -(1 << 29)) return 1;
  if (s->D < 64)
    return s->dtype == FA_F16
               ? launch_fwd_tc<__half, 64, true, false, true>(s, w, q1, k1, q2, k2, v, o, lse, stream)
               : launch_fwd_tc<__nv_bfloat16, 64, true, false, true>(s, w, q1, k1, q2, k2, v, o, lse, stream);
  if (s->dtype == FA_F16)
    return s->D == 128 ? launch_fwd_tc<__half, 128, true>(s, w, q1, k1, q2, k2, v, o, lse, stream)
                       : launch_fwd_tc<__half, 64, true>(s, w, q1, k1, q2, k2, v, o, lse, stream);
  return s->D == 128
             ? launch_fwd_tc<__nv_bfloat16, 128, true>(s, w, q1, k1, q2, k2, v, o, lse, stream)
             : launch_fwd_tc<__nv_bfloat16, 64, true>(s, w, q1, k1, q2, k2, v, o, lse, stream);
}

}  // namespace tc
}  // namespace fa

extern "C" int32_t fa_flash_key_split(const fa_flash_shape *s, int32_t num_sms) {
  if (const int st = fa::validate_shape(s)) return st;
  return s->dropout_p > 0.f ? 1 : fa::tc::key_split(s, num_sms).ctas;
}

extern "C" int32_t fa_set_kernel_family(int32_t family) { return fa::tc::set_kernel_family(family); }
