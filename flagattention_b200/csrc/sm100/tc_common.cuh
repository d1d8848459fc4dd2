// Blackwell (sm_100a) primitives used by the tensor-core kernels: mbarriers with
// time-bounded waits, TMA tiled loads, TMEM allocation, tcgen05 MMA / commit /
// load / store and the shared-memory and instruction descriptors they take.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fa {
namespace tc {

// ---------------------------------------------------------------------------
// error reporting: a wait that runs out of time records where it gave up in a
// device status word and raises a CTA-wide abort flag in shared memory; every
// other wait then returns immediately so the CTA can tear down and exit.
// ---------------------------------------------------------------------------
constexpr long long kWaitCycles = 2000000000ll;  // about one second of SM clocks

struct AbortCtx {
  volatile int *smem_flag;  // CTA-wide abort flag
  int *status;              // device status word (may be null)
};

// One thread of a converged warp, chosen by the hardware (the same one every time).  Code that issues
// tcgen05 / TMA work runs under this and not under `lane == 0`: their operands live in uniform
// registers, and only behind elect.sync does the compiler know that a single thread is active.  The
// issuing thread of the one-pass backward is on its critical path (40 MMAs, 10 waits and 8 commits a
// tile): B=4 H=32 L=4096 D=128 causal bf16 1.573 -> 1.495 ms, B=2 H=16 L=8192 D=64 2.05 -> 1.88 ms.
// In the forward, where two CTAs share an SM and hide each other's issuing, the MMA thread gains 0 to 5 %
// (B=1 H=32 Hk=8 M=512 N=7300 D=128 93.7 -> 91.3 us, B=4 H=16 L=2048 D=64 93 -> 89 us, L=4096 D=128 as before)
// and total_attention 1 % (321 -> 319 us with its forward at L=6144); their producers gain nothing.  A
// whole-warp form of these loops (uniform waits by vote) measured no better than this.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok));
  return ok != 0;
}

// ---------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Returns false when the wait was abandoned (out of time here, or abort raised elsewhere).
__device__ __forceinline__ bool mbar_wait_limit(uint32_t bar, uint32_t parity, const AbortCtx &ctx,
                                                int where, long long limit_cycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (*ctx.smem_flag) return false;
    if (clock64() - t0 > limit_cycles) {
      *ctx.smem_flag = 1;
      if (ctx.status) atomicCAS(ctx.status, 0, where);
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const AbortCtx &ctx,
                                          int where) {
  return mbar_wait_limit(bar, parity, ctx, where, kWaitCycles);
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

// ---------------------------------------------------------------------------
// CTA launch order.  A grid is `nblk` blocks x `npairs` (batch, head) pairs, and under a causal
// mask the cost of a block falls steadily with its index.  Numbering the CTAs pair by pair ends
// the grid with the heavy blocks of the last few pairs running alone (a tail of several per
// cent); numbering them heaviest-first over ALL pairs would have every resident CTA stream a
// different pair's operands, far more than L2 holds.  So the pairs are taken in groups of `gs`
// whose shared operands fit in L2 together, and inside a group all blocks 0 come first, then all
// blocks 1, and so on.  The grid is one-dimensional; every group but the last has `gs` pairs.
// ---------------------------------------------------------------------------
struct CtaCoord {
  int blk, pair;
};
__device__ __forceinline__ CtaCoord grouped_cta(unsigned id, int nblk, int npairs, int gs) {
  const unsigned per_group = (unsigned)gs * nblk;
  const unsigned g = id / per_group, r = id - g * per_group;
  const int n = min(gs, npairs - (int)g * gs);
  return CtaCoord{(int)(r / n), (int)(g * gs + r % n)};
}
// pairs per group: as many as keep `hot_bytes_per_pair` (the bytes the CTAs of one pair share)
// within about a quarter of L2, at most 32
inline int cta_group_size(int64_t hot_bytes_per_pair, int npairs) {
  const int64_t budget = 32ll << 20;
  int64_t gs = budget / (hot_bytes_per_pair > 0 ? hot_bytes_per_pair : 1);
  gs = gs < 1 ? 1 : (gs > 32 ? 32 : gs);
  return (int)(gs < npairs ? gs : (npairs > 0 ? npairs : 1));
}
// The groups cost their own tail: the heavy blocks of the last group start when the grid is nearly through, which
// with a few blocks an SM is up to 48 % of the mean load (list-scheduled).  So ALL pairs form one group, blocks in
// strictly falling order, where L2 can bear it:
//   forward, total attention: what all pairs share fits in L2 together (88 of 126 MB) and blocks differ (causal);
//   one-pass backward: up to 8 blocks an SM and 64 pairs, so that several CTAs walk each pair at any time.
// bf16 causal D=128, in groups -> in one, us: forward H=16 L=6144 175 -> 158 (50 MB), B=2 H=20 L=4096 237 -> 208 (84 MB),
// B=2 H=32 M=1627 N=2855 142 -> 148 (94 MB), B=2 H=32 L=4096 278 -> 311 (134 MB); backward B=3 H=32 Hk=8 L=1867 381 -> 321 (360
// blocks), H=32 Hk=8 L=8192 1871 -> 1383 (512), H=16 L=6144 493 -> 409 (768), B=2 H=32 Hk=16 L=4096 840 -> 762 (1024),
// B=4 H=32 L=1024 197 -> 203 (1024, 128 pairs), H=24 L=8192 1099 -> 1079 (1536), B=2 H=32 L=4096 760 -> 845 (2048).
// At D=64: forward B=2 H=20 L=4096 160 -> 135, B=3 H=32 Hk=8 L=1867 88 -> 82, B=4 H=32 L=1024 46.3 -> 43.5, H=24 L=8192
// 346 -> 307, 500 pairs of 330 39.1 -> 36.9; backward H=16 L=6144 244 -> 218, H=32 Hk=8 L=8192 954 -> 752, B=2 H=32 Hk=16
// L=4096 425 -> 416.
// Walks of a few blocks at head_dim 128 (`wide`) have little tail to gain and bear 64 MB: forward, 250 pairs of 672 63.2 ->
// 65.3, 512 of 300 48.2 -> 50.1, 500 of 330 50.3 -> 51.2; but 192 of 672 (63 MB) 52.1 -> 49.9, 70 of 672 28.1 -> 24.6.
inline bool one_group_in_l2(int64_t hot_bytes_per_pair, int npairs, bool causal) {
  return causal && hot_bytes_per_pair * npairs <= 88ll << 20;
}
inline int forward_group_size(int64_t hot_bytes_per_pair, int npairs, bool causal, int blocks, bool wide) {
  const bool too_much = wide && blocks <= 6 && hot_bytes_per_pair * npairs > 64ll << 20;
  if (!too_much && one_group_in_l2(hot_bytes_per_pair, npairs, causal)) return npairs > 0 ? npairs : 1;
  return cta_group_size(hot_bytes_per_pair, npairs);
}
inline int backward_group_size(int64_t hot_bytes_per_pair, int npairs, int64_t blocks, int sms, bool causal) {
  if (causal && blocks <= 8ll * sms && npairs <= 64) return npairs > 0 ? npairs : 1;
  return cta_group_size(hot_bytes_per_pair, npairs);
}

// ---------------------------------------------------------------------------
// TMA: 4-D tiled load global -> shared of this CTA only, completion on an mbarrier
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap *map,
                                            uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];\n" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// the same box, fetched into L2 only (nothing waits for it)
__device__ __forceinline__ void tma_prefetch_l2_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];\n" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---------------------------------------------------------------------------
// TMEM allocation (one warp, warp-collective)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                   smem_result),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// ---------------------------------------------------------------------------
// descriptors
// ---------------------------------------------------------------------------
// Shared-memory matrix descriptor for a tile stored as rows of 128 bytes with
// the 128-byte swizzle (what a TMA box of 64 16-bit elements x R rows writes).
// `sbo` = bytes between consecutive 8-row groups, `lbo` = bytes between
// consecutive 64-element column blocks (only read for MN-major operands).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr, uint32_t lbo,
                                                    uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of sm_100
  d |= (uint64_t)2 << 61;  // layout type: 128-byte swizzle
  return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16: fp32 accumulate, A and B of
// the same 16-bit type (0 = f16, 1 = bf16), majors 0 = K-major, 1 = MN-major.
__host__ __device__ constexpr uint32_t instr_desc_f16(int m, int n, int ab_format, int a_major,
                                                      int b_major) {
  return (1u << 4)                          // D format: f32
         | ((uint32_t)ab_format << 7)       // A format
         | ((uint32_t)ab_format << 10)      // B format
         | ((uint32_t)a_major << 15) | ((uint32_t)b_major << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// The same descriptor split in two 32-bit words, so that the issuing thread only has to add a
// byte offset (>> 4) to the low word between MMAs: the high word is the same for every operand.
constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version, SW128
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t smem_addr, uint32_t lbo) {
  return ((smem_addr & 0x3FFFF) >> 4) | (((lbo >> 4) & 0x3FFF) << 16);
}
// D[tmem] (+)= A[smem] * B[smem], descriptors given by their low words
__device__ __forceinline__ void mma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate)
      : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrive once every tcgen05 operation issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
      : "memory");
}

// ---------------------------------------------------------------------------
// TMEM <-> registers, 32 lanes x 32-bit, N consecutive columns per thread
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// The same 32 lanes x 32 columns in the fragments of an 8 x 8 matrix product (two 16-lane halves, 16x256b): thread l
// holds rows l / 4 + 8 i (i = 0..3) and columns 8 j + 2 (l % 4) + e (j = 0..3, e = 0, 1) in
// r[(i / 2) * 16 + 4 j + (i % 2) * 2 + e].
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t (&r)[32]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[16 * h]), "=r"(r[16 * h + 1]), "=r"(r[16 * h + 2]), "=r"(r[16 * h + 3]), "=r"(r[16 * h + 4]),
          "=r"(r[16 * h + 5]), "=r"(r[16 * h + 6]), "=r"(r[16 * h + 7]), "=r"(r[16 * h + 8]), "=r"(r[16 * h + 9]),
          "=r"(r[16 * h + 10]), "=r"(r[16 * h + 11]), "=r"(r[16 * h + 12]), "=r"(r[16 * h + 13]),
          "=r"(r[16 * h + 14]), "=r"(r[16 * h + 15])
        : "r"(taddr + ((uint32_t)(16 * h) << 16))
        : "memory");
}
// 32 lanes x 16 columns of packed pairs: pair (row, columns 8 j + 2 (l % 4), + 1) of those fragments, r[k] = the pair
// of elements 2 k, 2 k + 1 above
__device__ __forceinline__ void tmem_st_frag16(uint32_t taddr, const uint32_t (&r)[16]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(
            taddr + ((uint32_t)(16 * h) << 16)),
        "r"(r[8 * h]), "r"(r[8 * h + 1]), "r"(r[8 * h + 2]), "r"(r[8 * h + 3]), "r"(r[8 * h + 4]),
        "r"(r[8 * h + 5]), "r"(r[8 * h + 6]), "r"(r[8 * h + 7])
        : "memory");
}
// four 8 x 8 matrices of 16-bit elements, fragments -> shared memory: lanes 8 m .. 8 m + 7 give the row addresses of
// matrix m
__device__ __forceinline__ void stmatrix4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(r0), "r"(r1),
               "r"(r2), "r"(r3)
               : "memory");
}

template <typename T>
struct TcElem;
template <>
struct TcElem<__half> {
  static constexpr int kFormat = 0;
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2 *>(&u));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
  }
};
template <>
struct TcElem<__nv_bfloat16> {
  static constexpr int kFormat = 1;
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&u));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
  }
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// packed fp32 arithmetic of sm_100: one instruction works on two floats held in a
// 64-bit register pair, which halves the issue slots of the element-wise stages
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

}  // namespace tc
}  // namespace fa
