// paged_attention decode: block-table-indexed gather of the KV cache with
// online softmax, optional split-KV partitions and the partition reducer.
//
// HBM-bound by design: every warp of a CTA streams its own 16-token groups of
// K and V through a private multi-stage cp.async ring (16-byte coalesced
// gathers, swizzled shared memory), so nothing in the main loop needs a
// CTA-wide barrier.  The tiny GEMMs (query group padded to 16 rows) run on
// m16n8k16 tensor-core MMAs so that arithmetic never limits the stream.
#include "common.cuh"

namespace fa {

// IdxT: the table's entry type, or InPlace where there is no table (FA_BLOCK_TABLE_IN_PLACE)
struct InPlace {};
template <typename IdxT>
__device__ __forceinline__ int64_t phys_block(const void *block_tables, int64_t bt_stride_s,
                                              int seq, int logical_block) {
  const int64_t i = (int64_t)seq * bt_stride_s + logical_block;
  if constexpr (std::is_same<IdxT, InPlace>::value) return i;
  else return (int64_t) reinterpret_cast<const IdxT *>(block_tables)[i];
}
__device__ __forceinline__ int context_len(const fa_paged_args &a, int seq) {
  return a.context_lens ? a.context_lens[seq] : a.max_context_len;
}

template <int D>
struct PagedCfg {
  static constexpr int kWarps = D <= 128 ? 4 : 2;
  static constexpr int kStages = D <= 64 ? 4 : 3;
  static constexpr int kGroupBytes = 16 * D * 2;             // one 16-token K or V group
  static constexpr int kStageBytes = 2 * kGroupBytes;        // K + V
  static constexpr int kWarpBytes = kStages * kStageBytes;
  static constexpr int kQBytes = 16 * D * 2;
  static constexpr int kStatBytes = 2 * kWarps * 16 * 4;     // m, l per warp per row
  static constexpr int kRing = kQBytes + kStatBytes;
  static constexpr int kRingBytes = kWarps * kWarpBytes;
  static constexpr int kMergeBytes = kWarps * 16 * D * 4;    // fp32 partial outputs, aliases ring
  static constexpr int kTotal = kRing + (kRingBytes > kMergeBytes ? kRingBytes : kMergeBytes);
};

// How the kernels size the partitions of fa_paged_attention from the lengths themselves; finest == 0: every sequence
// takes a.partition_size.  Sizes are finest * 2^k.
struct Sizing {
  int finest, coarsest;
  int ctas;    // > 0: the largest size, up to `coarsest`, that leaves the whole call this many CTAs
  int parts;   // ctas == 0: the smallest size that cuts a sequence into this many at most
};
// The lengths of the first 64 sequences, two a lane, requested ahead of their use.
struct LaneLens {
  int first, second;
};
__device__ __forceinline__ LaneLens lane_lens(const fa_paged_args &a, const Sizing &z) {
  const int lane = threadIdx.x & 31;
  return LaneLens{z.ctas > 0 && lane < a.num_seqs ? context_len(a, lane) : 0,
                  z.ctas > 0 && lane + 32 < a.num_seqs ? context_len(a, lane + 32) : 0};
}
// Tokens per partition of a sequence of `ctx` tokens, called by whole warps; never more partitions than the P of the
// workspace.
__device__ __forceinline__ int partition_tokens(const fa_paged_args &a, const Sizing &z, LaneLens lens, int ctx, int P) {
  if (z.finest == 0) return a.partition_size;
  int k = 0;
  if (z.ctas > 0) {
    auto count = [&](int len) { return min(((unsigned)max(len, 0) + z.finest - 1) / z.finest, 1u << 20); };
    unsigned lane_n = count(lens.first) + count(lens.second);
    for (int i = (threadIdx.x & 31) + 64; i < a.num_seqs; i += 32) lane_n += count(context_len(a, i));
    // (a sum below 2^32: at most 2048 sequences)
    const unsigned long long n = (unsigned long long)__reduce_add_sync(0xffffffffu, lane_n) *
                                 (a.num_kv_heads * ((a.num_q_heads / a.num_kv_heads + 15) / 16));
    while ((z.finest << k) < z.coarsest && (n >> (k + 1)) >= (unsigned)z.ctas) ++k;
  }
  const int parts = z.ctas > 0 ? P : min(P, z.parts);
  while ((z.finest << k) < a.partition_size && (long long)parts * (z.finest << k) < ctx) ++k;
  return z.finest << k;
}

// HALF: at most 8 query rows, the upper half of the 16-row tile; the lower half serves the remainder of P.
template <typename T, int D, typename IdxT, bool HALF>
__global__ void __launch_bounds__(PagedCfg<D>::kWarps * 32) paged_decode_kernel(
    const fa_paged_args a, const Sizing z) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");   // the reduction waits for all of this grid by itself
  using C = PagedCfg<D>;
  constexpr int NW = C::kWarps, NS = C::kStages, CPR = D / 8;
  constexpr int R = HALF ? 1 : 2;   // accumulator rows of a thread: g and, in a full tile, g + 8
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem = smem_u32(smem_raw);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int seq = blockIdx.x;
  const int G = a.num_q_heads / a.num_kv_heads;
  const int q_tiles = (G + 15) / 16;
  const int hk = blockIdx.y / q_tiles, qt = blockIdx.y % q_tiles;
  const int part = blockIdx.z;
  const int rows = min(16, G - qt * 16);          // valid query rows of this CTA
  const int qh0 = hk * G + qt * 16;               // first query head

  const int ctx = context_len(a, seq);
  int t_begin = 0, t_end = ctx;
  if (a.partition_size > 0) {
    const LaneLens lens = lane_lens(a, z);   // in flight together with ctx
    if ((long long)part * (z.finest ? z.finest : a.partition_size) >= ctx) return;
    const int size = partition_tokens(a, z, lens, ctx, gridDim.z);
    if ((long long)part * size >= ctx) return;
    t_begin = part * size;
    t_end = (int)min((long long)ctx, (long long)t_begin + size);
  }
  const int BS = a.block_size;
  const bool group_in_block = (BS % 16 == 0) && (t_begin % 16 == 0);
  // Several queries per head (a.causal_rows = Mq > 0): query head index = head * Mq + m, and query
  // m of a head is the (Mq - 1 - m)-th from the end of the sequence, so it sees the tokens below
  // ctx - (Mq - 1 - m).  This thread's two accumulator rows are g and g + 8 of the tile.
  int row_end[2] = {t_end, t_end};
  if (a.causal_rows > 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int m = (qt * 16 + g + 8 * r) % a.causal_rows;
      row_end[r] = min(t_end, ctx - (a.causal_rows - 1 - m));
    }
  }

  // ---- query group -> shared (rows >= `rows` are zero) ---------------------
  {
    const T *qg = reinterpret_cast<const T *>(a.query) + (int64_t)seq * a.q_stride_s;
    for (int idx = tid; idx < 16 * CPR; idx += NW * 32) {
      const int r = idx / CPR, ch = idx % CPR;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < rows)
        v = *reinterpret_cast<const uint4 *>(qg + (int64_t)(qh0 + r) * a.q_stride_h + ch * 8);
      *reinterpret_cast<uint4 *>(smem_raw + Tile<D>::offset(r, ch)) = v;
    }
  }
  __syncthreads();

  constexpr bool kQInRegs = D <= 128;
  uint32_t qf[kQInRegs ? D / 16 : 1][4];
  if (kQInRegs) {
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) load_A<D>(qf[kk], smem, 0, kk, lane);
  }

  // ---- this warp's token groups ---------------------------------------------
  const int n_groups = (t_end - t_begin + 15) / 16;           // groups of the CTA
  const int my_groups = n_groups > warp ? (n_groups - warp + NW - 1) / NW : 0;
  const uint32_t ring = smem + C::kRing + warp * C::kWarpBytes;
  const T *kc = reinterpret_cast<const T *>(a.key_cache) + (int64_t)hk * a.kv_stride_h;
  const T *vc = reinterpret_cast<const T *>(a.value_cache) + (int64_t)hk * a.kv_stride_h;

  // Per-lane constants of the gather.  In every 16-token group this lane copies the 16-byte
  // chunk `ch` of rows c * RPC + lane_r (c = 0..NC-1), for K and for V, so the shared-memory
  // offsets are fixed and the global address only advances by RPC rows per step.
  constexpr int NC = 16 * CPR / 32;  // copy steps per lane per group
  constexpr int RPC = 16 / NC;       // rows covered per step
  const int lane_r = lane / CPR, ch = lane % CPR;
  uint32_t dst_off[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) dst_off[c] = Tile<D>::offset(c * RPC + lane_r, ch);
  const int64_t lane_src = (int64_t)lane_r * a.kv_stride_t + ch * 8;
  const int64_t c_step = (int64_t)RPC * a.kv_stride_t;
  const int64_t v_minus_k = vc - kc;
  const int bs_shift = (BS & (BS - 1)) == 0 ? 31 - __clz(BS) : -1;

  auto issue = [&](int i) {  // i-th group of this warp -> stage i % NS
    const int tok0 = t_begin + (warp + i * NW) * 16;
    const uint32_t st = ring + (i % NS) * C::kStageBytes;
    if (group_in_block) {
      // the whole group lies in one physical block: one table lookup, then pointer increments
      const int lb = bs_shift >= 0 ? tok0 >> bs_shift : tok0 / BS;
      const int in_blk = tok0 - lb * BS;
      const int64_t pb = phys_block<IdxT>(a.block_tables, a.bt_stride_s, seq, lb);
      const T *src = kc + pb * a.kv_stride_b + (int64_t)in_blk * a.kv_stride_t + lane_src;
      const int rows_left = t_end - tok0 - lane_r;  // row c*RPC + lane_r exists iff c*RPC < rows_left
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const bool ok = c * RPC < rows_left;
        const T *sk = ok ? src : kc;
        cp_async16(st + dst_off[c], sk, ok);
        cp_async16(st + C::kGroupBytes + dst_off[c], sk + v_minus_k, ok);
        src += c_step;
      }
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int tok = tok0 + c * RPC + lane_r;
        const bool ok = tok < t_end;
        int64_t off = 0;
        if (ok) {
          const int64_t pb = phys_block<IdxT>(a.block_tables, a.bt_stride_s, seq, tok / BS);
          off = pb * a.kv_stride_b + (int64_t)(tok % BS) * a.kv_stride_t + ch * 8;
        }
        cp_async16(st + dst_off[c], kc + off, ok);
        cp_async16(st + C::kGroupBytes + dst_off[c], vc + off, ok);
      }
    }
  };

#pragma unroll
  for (int i = 0; i < NS - 1; ++i) {
    if (i < my_groups) issue(i);
    cp_async_commit();
  }

  float acc[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  float m_i[2] = {-INFINITY, -INFINITY};
  float l_i[2] = {0.f, 0.f};
  const float qk_scale = a.attn_scale * kLog2e;

#pragma unroll 1
  for (int i = 0; i < my_groups; ++i) {
    if (i + NS - 1 < my_groups) issue(i + NS - 1);
    cp_async_commit();
    cp_async_wait<NS - 1>();
    __syncwarp();

    const int tok0 = t_begin + (warp + i * NW) * 16;
    const uint32_t st = ring + (i % NS) * C::kStageBytes;

    float s[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t bb[4];
      load_B_nk<D>(bb, st, 0, kk, lane);
      if (kQInRegs) {
        Elem<T>::mma(s[0], qf[kk], bb[0], bb[1]);
        Elem<T>::mma(s[1], qf[kk], bb[2], bb[3]);
      } else {
        uint32_t qa[4];
        load_A<D>(qa, smem, 0, kk, lane);
        Elem<T>::mma(s[0], qa, bb[0], bb[1]);
        Elem<T>::mma(s[1], qa, bb[2], bb[3]);
      }
    }
    const bool tail = tok0 + 16 > min(row_end[0], row_end[R - 1]);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2 * R; ++e) {
        const int tok = tok0 + j * 8 + 2 * t4 + (e & 1);
        s[j][e] = (tail && tok >= row_end[e >> 1]) ? -INFINITY : s[j][e] * qk_scale;
      }
    // Running maximum with lazy rescaling: the accumulators are only rescaled when some row's
    // maximum grew by more than 2^8 (scores are already in the base-2 domain); otherwise the
    // stale maximum stays the reference point and P simply ranges up to 2^8.
    float m_new[2];
    bool need = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float mx = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
      mx = quad_max(mx);
      m_new[r] = fmaxf(m_i[r], mx);  // -inf only while a row has not seen a token it may see
      need = need || (m_new[r] - m_i[r] > 8.f);
    }
    if (__any_sync(0xffffffffu, need)) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float alpha = (m_new[r] == -INFINITY) ? 1.f : fast_exp2(m_i[r] - m_new[r]);
        l_i[r] *= alpha;
        m_i[r] = m_new[r];
#pragma unroll
        for (int j = 0; j < D / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4 / R; ++e) acc[j][2 * r + e] *= alpha;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float rs = 0.f;
      const float m_ref = (m_i[r] == -INFINITY) ? 0.f : m_i[r];   // all scores -inf: P = 0
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[j][2 * r] = fast_exp2(s[j][2 * r] - m_ref);
        s[j][2 * r + 1] = fast_exp2(s[j][2 * r + 1] - m_ref);
        rs += s[j][2 * r] + s[j][2 * r + 1];
      }
      l_i[r] += rs;
    }
    // P goes in as a 16-bit value and a 16-bit remainder.  Rounded once, its error depends on the run of tokens a
    // warp takes: the one that sets the run's reference maximum has weight 1 and no error, so shorter runs have
    // less of it (fp16, 64 sequences to 32768: 2.79e-4 with partitions of 256, 2.90e-4 of 2048; with the remainder
    // 2.07e-4, the rounding of the output alone).
    uint32_t pa[4], pr[4];
    if (HALF) {
      split_weights<T>(s[0][0], s[0][1], pa[0], pa[1]);
      split_weights<T>(s[1][0], s[1][1], pa[2], pa[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) split_weights<T>(s[i >> 1][2 * (i & 1)], s[i >> 1][2 * (i & 1) + 1], pa[i], pr[i]);
    }
    constexpr int U = HALF ? 1 : D / 16 < 4 ? D / 16 : 4;   // chunks whose two products are kept apart
#pragma unroll
    for (int d0 = 0; d0 < D / 16; d0 += U) {
      uint32_t bb[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        load_B_kn<D>(bb[u], st + C::kGroupBytes, 0, (d0 + u) * 2, lane);
        Elem<T>::mma(acc[2 * (d0 + u)], pa, bb[u][0], bb[u][1]);
        Elem<T>::mma(acc[2 * (d0 + u) + 1], pa, bb[u][2], bb[u][3]);
      }
      if (!HALF) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          Elem<T>::mma(acc[2 * (d0 + u)], pr, bb[u][0], bb[u][1]);
          Elem<T>::mma(acc[2 * (d0 + u) + 1], pr, bb[u][2], bb[u][3]);
        }
      }
    }
    __syncwarp();  // stage may be refilled by the next iteration's issue
  }
  cp_async_wait<0>();

  if (HALF) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) acc[j][0] += acc[j][2], acc[j][1] += acc[j][3];
  }

  // ---- merge the warps' partial states --------------------------------------
  float *stat_m = reinterpret_cast<float *>(smem_raw + C::kQBytes);
  float *stat_l = stat_m + NW * 16;
  float *merge = reinterpret_cast<float *>(smem_raw + C::kRing);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float l = quad_sum(l_i[r]);
    if (t4 == 0) {
      stat_m[warp * 16 + g + 8 * r] = m_i[r];
      stat_l[warp * 16 + g + 8 * r] = l;
    }
  }
  __syncthreads();  // stats visible; every warp has drained its ring
  float scale_w[2];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = g + 8 * r;
    float mm = -INFINITY;
#pragma unroll
    for (int w2 = 0; w2 < NW; ++w2) mm = fmaxf(mm, stat_m[w2 * 16 + row]);
    scale_w[r] = (m_i[r] == -INFINITY) ? 0.f : fast_exp2(m_i[r] - mm);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = g + 8 * r;
    if (row < rows) {
      float *dst = merge + ((int64_t)warp * 16 + row) * D;
#pragma unroll
      for (int j = 0; j < D / 8; ++j)
        *reinterpret_cast<float2 *>(dst + j * 8 + 2 * t4) =
            make_float2(acc[j][2 * r] * scale_w[r], acc[j][2 * r + 1] * scale_w[r]);
    }
  }
  __syncthreads();

  for (int idx = tid; idx < rows * (D / 4); idx += NW * 32) {
    const int row = idx / (D / 4), c4 = idx % (D / 4);
    float mm = -INFINITY;
#pragma unroll
    for (int w2 = 0; w2 < NW; ++w2) mm = fmaxf(mm, stat_m[w2 * 16 + row]);
    float l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w2 = 0; w2 < NW; ++w2) {
      const float mw = stat_m[w2 * 16 + row];
      if (mw != -INFINITY) l += stat_l[w2 * 16 + row] * fast_exp2(mw - mm);
      const float4 v = *reinterpret_cast<const float4 *>(merge + ((int64_t)w2 * 16 + row) * D + c4 * 4);
      o.x += v.x, o.y += v.y, o.z += v.z, o.w += v.w;
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    o.x *= inv, o.y *= inv, o.z *= inv, o.w *= inv;
    const int qh = qh0 + row;
    if (a.partition_size > 0) {
      const int P = (a.max_context_len + a.partition_size - 1) / a.partition_size;
      const int64_t pi = ((int64_t)seq * a.num_q_heads + qh) * P + part;
      *reinterpret_cast<float4 *>(a.part_out + pi * D + c4 * 4) = o;
      if (c4 == 0) {
        a.part_max[pi] = mm;
        a.part_sum[pi] = l;
      }
    } else {
      T *dst = reinterpret_cast<T *>(a.out) + (int64_t)seq * a.o_stride_s +
               (int64_t)qh * a.o_stride_h + c4 * 4;
      uint2 pk;
      pk.x = Elem<T>::pack(o.x, o.y);
      pk.y = Elem<T>::pack(o.z, o.w);
      *reinterpret_cast<uint2 *>(dst) = pk;
    }
  }
}

// One CTA per (seq, query head): its threads are 4 blockDim / D groups of D / 4, a thread owning 4 output columns of every
// so many partitions.  What bounds it is latency, two round trips to L2 (statistics, then rows): a CTA that went
// through the partitions one after another with the threads of one row took 13.4 us for 32 partitions of 32 rows (dense
// decoding, B=2 H=16 N=131072, beside 299 us of decoding) and 8.9 us for 64 sequences of 32 heads up to 32768 tokens:
// the first of these calls 317 -> 307 us.  It is launched while the decode kernel's last CTAs run (programmatic stream
// serialization) and waits for that grid: 307 -> 305 us, H=16 N=512 7.9 -> 6.8 us, 4 sequences up to 1500 10.0 -> 8.4.
//
// Threads a row: up to 256 while all rows find room beside the decode kernel's CTAs, which still hold about half of every
// SM (1024 threads); more rows with fewer threads run at once.  fp16, rows and us at 32 / 64 / 128 / 256 threads a row:
//   128 sequences up to 1562 tokens, 16 heads over 2, D=128 (2048)   27.9 / 28.0 / 30.3 / 33.6
//   64 up to 3029, 16 over 2, D=64 (1024)    26.7 / 26.7 / 27.0 / 29.7      64 up to 3125, D=128 24.4 / 23.9 / 23.9 / 26.1
//   128 up to 1488, 8 over 1, D=256 (1024)     -  / 40.5 / 40.2 / 42.7      100 up to 2000, 8 over 1, D=128 (800)
//   12 up to 13860, 32 over 8, D=128 (384)   75.6 / 74.8 / 73.8 / 74.1      19.5 / 19.2 / 19.5 / 20.0
//   10 up to 19849, 32 over 8, D=128 (320)   89.3 / 85.5 / 83.8 / 83.1      1 up to 28326, 8 over 8, D=256 (8)
//   7 up to 19563, 8 over 1, D=128 (56)      23.3 / 18.1 / 15.6 / 14.4        -  / 47.3 / 44.1 / 42.5
constexpr int kReduceThreads = 256;
static int reduce_threads(int64_t rows, int head_size, int sms) {
  int threads = kReduceThreads;
  while (threads > 32 && threads > head_size / 4 && rows * threads > 1024ll * sms) threads /= 2;
  return threads;
}
template <typename T>
__global__ void __launch_bounds__(kReduceThreads) paged_reduce_kernel(const fa_paged_args a, const Sizing z) {
  __shared__ float4 part_o[kReduceThreads];
  __shared__ float part_den[kReduceThreads];
  const int seq = blockIdx.x, qh = blockIdx.y;
  const int D = a.head_size, cols = D / 4, groups = blockDim.x / cols;
  const int g = threadIdx.x / cols, c4 = threadIdx.x % cols;
  const int P = (a.max_context_len + a.partition_size - 1) / a.partition_size;
  const int ctx = context_len(a, seq);
  const int size = partition_tokens(a, z, lane_lens(a, z), ctx, P);
  const int np = min(P, (ctx + size - 1) / size);
  // launched beside the decode kernel's last CTAs (reduce()): its results are there from here on
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int64_t base = ((int64_t)seq * a.num_q_heads + qh) * P;
  float mm = -INFINITY;
  for (int p = threadIdx.x & 31; p < np; p += 32) mm = fmaxf(mm, a.part_max[base + p]);
#pragma unroll
  for (int off = 16; off; off >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, off));
  float den = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int p = g; p < np; p += groups) {
    const float wgt = a.part_sum[base + p] * fast_exp2(a.part_max[base + p] - mm);
    den += wgt;
    const float4 v = *reinterpret_cast<const float4 *>(a.part_out + (base + p) * D + c4 * 4);
    o.x += wgt * v.x, o.y += wgt * v.y, o.z += wgt * v.z, o.w += wgt * v.w;
  }
  part_o[threadIdx.x] = o, part_den[threadIdx.x] = den;
  __syncthreads();
  if (g > 0) return;
  for (int i = 1; i < min(groups, np); ++i) {
    const float4 v = part_o[i * cols + c4];
    den += part_den[i * cols + c4];
    o.x += v.x, o.y += v.y, o.z += v.z, o.w += v.w;
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  T *dst = reinterpret_cast<T *>(a.out) + (int64_t)seq * a.o_stride_s + (int64_t)qh * a.o_stride_h + c4 * 4;
  uint2 pk;
  pk.x = Elem<T>::pack(o.x * inv, o.y * inv);
  pk.y = Elem<T>::pack(o.z * inv, o.w * inv);
  *reinterpret_cast<uint2 *>(dst) = pk;
}

template <typename IdxT>
__global__ void paged_trace_kernel(const fa_paged_args a, int64_t *visited, int max_blocks) {
  const int seq = blockIdx.x;
  const int ctx = a.context_lens[seq];
  const int used = (ctx + a.block_size - 1) / a.block_size;
  for (int blk = threadIdx.x; blk < max_blocks; blk += blockDim.x)
    visited[(int64_t)seq * max_blocks + blk] =
        blk < used ? phys_block<IdxT>(a.block_tables, a.bt_stride_s, seq, blk) : -1;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// no table and no lengths: the blocks of a sequence follow one another in memory
static bool in_place(const fa_paged_args *a) {
  return a->block_table_is_i64 == FA_BLOCK_TABLE_IN_PLACE && !a->block_tables && !a->context_lens;
}

static int validate_paged(const fa_paged_args *a, bool need_ws) {
  if (!a || !a->query || !a->key_cache || !a->value_cache || !a->out) return FA_ERR_BAD_ARG;
  if ((!a->context_lens || !a->block_tables) && !in_place(a)) return FA_ERR_BAD_ARG;
  if (a->dtype != FA_F16 && a->dtype != FA_BF16) return FA_ERR_BAD_ARG;
  if (a->num_seqs <= 0 || a->num_q_heads <= 0 || a->num_kv_heads <= 0 || a->block_size <= 0 ||
      a->max_context_len <= 0 || a->partition_size < 0)
    return FA_ERR_BAD_ARG;
  if (a->num_q_heads % a->num_kv_heads != 0) return FA_ERR_BAD_ARG;
  if (a->partition_size % 16 != 0) return FA_ERR_BAD_ARG;
  if (a->causal_rows < 0 || (a->causal_rows > 0 && (a->num_q_heads / a->num_kv_heads) % a->causal_rows != 0))
    return FA_ERR_BAD_ARG;
  const int D = a->head_size;
  if (!(D == 16 || D == 32 || D == 64 || D == 128 || D == 256)) return FA_ERR_UNSUPPORTED;
  if (!aligned16(a->query) || !aligned16(a->key_cache) || !aligned16(a->value_cache) ||
      !aligned16(a->out))
    return FA_ERR_ALIGNMENT;
  if (a->q_stride_s % 8 || a->q_stride_h % 8 || a->kv_stride_b % 8 || a->kv_stride_h % 8 ||
      a->kv_stride_t % 8 || a->o_stride_s % 4 || a->o_stride_h % 4)
    return FA_ERR_ALIGNMENT;
  if (need_ws && a->partition_size > 0 && (!a->part_out || !a->part_max || !a->part_sum))
    return FA_ERR_WORKSPACE;
  return FA_OK;
}

template <typename T, int D, typename IdxT, bool HALF>
static int launch_paged(const fa_paged_args *a, const Sizing &z, cudaStream_t stream) {
  using C = PagedCfg<D>;
  auto kern = paged_decode_kernel<T, D, IdxT, HALF>;
  static unsigned long long attr_done = 0;  // per instantiation, one bit per device
  if (int st = ensure_dyn_smem(kern, C::kTotal, &attr_done)) return st;
  const int G = a->num_q_heads / a->num_kv_heads;
  const int q_tiles = (G + 15) / 16;
  const int P = a->partition_size > 0
                    ? (a->max_context_len + a->partition_size - 1) / a->partition_size
                    : 1;
  dim3 grid(a->num_seqs, a->num_kv_heads * q_tiles, P);
  kern<<<grid, C::kWarps * 32, C::kTotal, stream>>>(*a, z);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

template <typename T, typename IdxT>
static int dispatch_paged_d(const fa_paged_args *a, const Sizing &z, cudaStream_t stream) {
  const bool half = a->num_q_heads / a->num_kv_heads <= 8;
  switch (a->head_size) {
    case 16:
      return half ? launch_paged<T, 16, IdxT, true>(a, z, stream) : launch_paged<T, 16, IdxT, false>(a, z, stream);
    case 32:
      return half ? launch_paged<T, 32, IdxT, true>(a, z, stream) : launch_paged<T, 32, IdxT, false>(a, z, stream);
    case 64:
      return half ? launch_paged<T, 64, IdxT, true>(a, z, stream) : launch_paged<T, 64, IdxT, false>(a, z, stream);
    case 128:
      return half ? launch_paged<T, 128, IdxT, true>(a, z, stream) : launch_paged<T, 128, IdxT, false>(a, z, stream);
    case 256:
      return half ? launch_paged<T, 256, IdxT, true>(a, z, stream) : launch_paged<T, 256, IdxT, false>(a, z, stream);
  }
  return FA_ERR_UNSUPPORTED;
}

static int decode(const fa_paged_args *a, const Sizing &z, cudaStream_t s) {
  if (in_place(a))
    return a->dtype == FA_F16 ? dispatch_paged_d<__half, InPlace>(a, z, s)
                              : dispatch_paged_d<__nv_bfloat16, InPlace>(a, z, s);
  if (a->dtype == FA_F16)
    return a->block_table_is_i64 ? dispatch_paged_d<__half, int64_t>(a, z, s)
                                 : dispatch_paged_d<__half, int32_t>(a, z, s);
  return a->block_table_is_i64 ? dispatch_paged_d<__nv_bfloat16, int64_t>(a, z, s)
                               : dispatch_paged_d<__nv_bfloat16, int32_t>(a, z, s);
}

static int reduce(const fa_paged_args *a, const Sizing &z, cudaStream_t s) {
  dim3 grid(a->num_seqs, a->num_q_heads);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid, cfg.stream = s, cfg.attrs = &attr, cfg.numAttrs = 1;
  cfg.blockDim = dim3(reduce_threads((int64_t)a->num_seqs * a->num_q_heads, a->head_size, sm_count_of_device()));
  const cudaError_t st = a->dtype == FA_F16 ? cudaLaunchKernelEx(&cfg, paged_reduce_kernel<__half>, *a, z)
                                            : cudaLaunchKernelEx(&cfg, paged_reduce_kernel<__nv_bfloat16>, *a, z);
  if (st != cudaSuccess) return FA_ERR_LAUNCH;
  FA_CHECK_LAUNCH();
  return FA_OK;
}

// size / finest is a power of two
static bool nests(int size, int finest) {
  return size % finest == 0 && ((size / finest) & (size / finest - 1)) == 0;
}

}  // namespace fa

using namespace fa;

extern "C" int fa_paged_decode(const fa_paged_args *a, void *stream) {
  if (int st = validate_paged(a, true)) return st;
  return decode(a, Sizing{}, static_cast<cudaStream_t>(stream));
}

extern "C" int fa_paged_reduce(const fa_paged_args *a, void *stream) {
  if (int st = validate_paged(a, true)) return st;
  if (a->partition_size <= 0) return FA_ERR_BAD_ARG;
  return reduce(a, Sizing{}, static_cast<cudaStream_t>(stream));
}

extern "C" int fa_paged_attention(const fa_paged_args *a, int32_t finest, int32_t coarsest, int32_t ctas,
                                  int32_t parts, void *stream) {
  if (int st = validate_paged(a, true)) return st;
  if (a->partition_size <= 0 || a->partition_size > (1 << 24) || finest <= 0 || finest % 16 || finest > a->partition_size ||
      coarsest < finest || coarsest > (1 << 24) || !nests(a->partition_size, finest) || !nests(coarsest, finest))
    return FA_ERR_BAD_ARG;
  if (ctas < 0 || (ctas == 0 && parts <= 0) || (ctas > 0 && a->num_seqs > 2048)) return FA_ERR_BAD_ARG;
  const Sizing z{finest, coarsest, ctas, parts};
  if (int st = decode(a, z, static_cast<cudaStream_t>(stream))) return st;
  return reduce(a, z, static_cast<cudaStream_t>(stream));
}

extern "C" int64_t fa_paged_workspace_bytes(const fa_paged_args *a) {
  if (!a || a->partition_size <= 0) return 0;
  const int64_t P = (a->max_context_len + a->partition_size - 1) / a->partition_size;
  const int64_t rows = (int64_t)a->num_seqs * a->num_q_heads * P;
  return rows * a->head_size * 4 + 2 * rows * 4;
}

extern "C" int fa_paged_trace_blocks(const fa_paged_args *a, int64_t *visited, int32_t max_blocks,
                                     void *stream) {
  int st = validate_paged(a, false);
  if (st != FA_OK) return st;
  if (!visited || max_blocks <= 0 || in_place(a)) return FA_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (a->block_table_is_i64)
    paged_trace_kernel<int64_t><<<a->num_seqs, 256, 0, s>>>(*a, visited, max_blocks);
  else
    paged_trace_kernel<int32_t><<<a->num_seqs, 256, 0, s>>>(*a, visited, max_blocks);
  FA_CHECK_LAUNCH();
  return FA_OK;
}

// ---------------------------------------------------------------------------
// Partitioned decode for callers that have no memory to hand us.
//
// Some hosts of this library cannot supply the split-KV workspace: a serving
// process that gave every spare byte of HBM to its KV-cache pool at start-up
// has nothing left to carve a workspace from, and a decode loop that is
// forbidden from entering the CUDA allocator (it would stall on the allocator
// lock or break its latency budget) cannot create one per call either.  For
// them the partial outputs and softmax statistics live in the fixed array
// below, which is part of the library image: every GPU that loads the library
// carries these FA_PAGED_NOALLOC_SCRATCH_BYTES until the process exits.
//
// `g_paged_scratch` names a device object.  Host code must not treat that name
// as a pointer: it is only a handle from which the real device address is
// looked up, once per device, with cudaGetSymbolAddress while that device is
// current; the address is then what the kernels receive.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_paged_scratch[FA_PAGED_NOALLOC_SCRATCH_BYTES];

namespace fa {

static constexpr int kMaxDevices = 64;
static unsigned char *g_paged_scratch_addr[kMaxDevices];  // resolved device addresses, per device

// Looks up (first call on a device) or returns (later calls) the device address of the scratch
// array for the current device.  No allocation happens here or anywhere below.
static int paged_scratch_base(unsigned char **base) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return FA_ERR_LAUNCH;
  if (dev < 0 || dev >= kMaxDevices) return FA_ERR_TOO_LARGE;
  if (!g_paged_scratch_addr[dev]) {
    unsigned char *ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_paged_scratch) != cudaSuccess ||
        !ptr)
      return FA_ERR_LAUNCH;
    g_paged_scratch_addr[dev] = ptr;
  }
  *base = g_paged_scratch_addr[dev];
  return FA_OK;
}

}  // namespace fa

extern "C" int fa_paged_attention_noalloc(const fa_paged_args *a, void *stream) {
  if (!a) return FA_ERR_BAD_ARG;
  if (a->partition_size <= 0) return FA_ERR_BAD_ARG;  // the one-pass mode needs no scratch at all
  fa_paged_args local = *a;
  local.part_out = nullptr, local.part_max = nullptr, local.part_sum = nullptr;
  int st = validate_paged(&local, false);
  if (st != FA_OK) return st;
  const int64_t need = fa_paged_workspace_bytes(&local);
  if (need > (int64_t)FA_PAGED_NOALLOC_SCRATCH_BYTES) return FA_ERR_TOO_LARGE;

  unsigned char *base = nullptr;
  st = paged_scratch_base(&base);
  if (st != FA_OK) return st;
  const int64_t P = (local.max_context_len + local.partition_size - 1) / local.partition_size;
  const int64_t rows = (int64_t)local.num_seqs * local.num_q_heads * P;
  // layout inside the array: partial outputs, then running maxima, then running sums.  Nothing
  // has to be zeroed: the decode kernel writes every (row, partition) slot the reducer later reads.
  local.part_out = reinterpret_cast<float *>(base);
  local.part_max = local.part_out + rows * local.head_size;
  local.part_sum = local.part_max + rows;
  st = fa_paged_decode(&local, stream);
  if (st != FA_OK) return st;
  return fa_paged_reduce(&local, stream);
}
