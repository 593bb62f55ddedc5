// Glue kernels of one decode step, all fp32 like the reference: embedding-row dequantisation
// (src/model.cpp:58-252), RMSNorm with fused residual add (src/layers/norm.cpp:18-34,
// model.cpp:385-399), GQA decode attention with bias + RoPE + KV-cache write folded in
// (model.cpp:312-372, src/layers/embedding.cpp:36-75, src/layers/attention.cpp:23-42) and SiLU(gate)*up (model.cpp:36,414-416).
#include "decode_device.cuh"
#include "device_utils.cuh"

#include <algorithm>
#include <cstdlib>

namespace lmb {

namespace {

__global__ void k_embed_rows(const int *tokens, int kind, const uint8_t *tiles, size_t bpr, size_t vocab, size_t h,
                             float scale, float *hidden) {
  asm volatile("griddepcontrol.launch_dependents;");  // a following GEMV may prefetch its weights
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= h) return;
  const int tok = tokens[blockIdx.y];
  // rows beyond the table read as zero (model.cpp:95-104)
  // gemma-type models scale the row by sqrt(hidden size) (model.cpp:255-260); scale = 1 otherwise
  hidden[size_t(blockIdx.y) * h + i] = (tok >= 0 && size_t(tok) < vocab) ? tile_elem(kind, tiles, bpr, size_t(tok), i) * scale : 0.0f;
}

// hidden += add (if given); out = hidden * rsqrt(mean(hidden^2) + eps) * w.  One CTA per sequence.
__global__ void __launch_bounds__(1024) k_add_rmsnorm(float *hidden, const float *add, const float *w, float *out,
                                                      size_t h, float eps) {
  asm volatile("griddepcontrol.launch_dependents;");  // a following GEMV may prefetch its weights
  __shared__ float red[32];
  float *x = hidden + size_t(blockIdx.x) * h;
  const float *a = add ? add + size_t(blockIdx.x) * h : nullptr;
  float *o = out + size_t(blockIdx.x) * h;
  float ss = 0.0f;
  for (size_t i = threadIdx.x; i < h; i += blockDim.x) {
    float v = x[i];
    if (a) {
      v += a[i];
      x[i] = v;
    }
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float inv = 1.0f / sqrtf(ss / float(h) + eps);
  for (size_t i = threadIdx.x; i < h; i += blockDim.x) o[i] = x[i] * inv * w[i];
}

// Tensor-parallel form of k_add_rmsnorm: the vector to add is the sum over ranks of the partial
// vectors in this rank's exchange block.  Every element is an 8-byte word {value, epoch tag}
// written by its producer with one store; the reader polls the word (bounded) until the tag is
// the expected one, adds the partials in rank order (so that every rank computes the same bits),
// then normalises.  One CTA per sequence; the last CTA to finish advances the epoch.
__device__ __forceinline__ unsigned long long ld_volatile_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__global__ void __launch_bounds__(1024) k_tp_sum_add_rmsnorm(float *hidden, XchgHeader *hdr, const unsigned long long *data, int tp,
                                                             unsigned cap, const float *w, float *out, size_t h, float eps,
                                                             unsigned spin_limit) {
  asm volatile("griddepcontrol.launch_dependents;");
  __shared__ float red[32];
  const unsigned epoch = *reinterpret_cast<volatile unsigned *>(&hdr->epoch);
  const unsigned tag = epoch + 1u;
  const unsigned long long *part = data + size_t(epoch & 1u) * tp * cap + size_t(blockIdx.x) * h;
  float *x = hidden + size_t(blockIdx.x) * h;
  float *o = out + size_t(blockIdx.x) * h;
  float ss = 0.0f;
  bool gave_up = *reinterpret_cast<volatile unsigned *>(&hdr->timed_out) != 0u;
  for (size_t i = threadIdx.x; i < h; i += blockDim.x) {
    float add = 0.0f;
    for (int r = 0; r < tp; ++r) {
      const unsigned long long *src = part + size_t(r) * cap + i;
      unsigned long long word = ld_volatile_u64(src);
      unsigned spins = 0;
      while (unsigned(word >> 32) != tag && !gave_up) {
        if (++spins > spin_limit) {  // give up, report, carry on with what is there
          hdr->timed_out = 1u;
          gave_up = true;
          break;
        }
        __nanosleep(40);
        word = ld_volatile_u64(src);
      }
      add += __uint_as_float(unsigned(word));
    }
    const float v = x[i] + add;
    x[i] = v;
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float inv = 1.0f / sqrtf(ss / float(h) + eps);
  for (size_t i = threadIdx.x; i < h; i += blockDim.x) o[i] = x[i] * inv * w[i];
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&hdr->done, 1u) == gridDim.x - 1u) {
    hdr->done = 0u;
    *reinterpret_cast<volatile unsigned *>(&hdr->epoch) = tag;  // read by the next producer, a later kernel
  }
}

__global__ void __launch_bounds__(ATT_THREADS) k_decode_attn(const AttnArgs a, const RopeDims d) {
  asm volatile("griddepcontrol.launch_dependents;");  // a following GEMV may prefetch its weights
  extern __shared__ float sm[];
  __shared__ int is_last;
  attn_item<false>(a, d, blockIdx.x, blockIdx.y, blockIdx.z, sm, &is_last);
}

// Group attention of one sequence as a kernel of its own: grid = (KV heads x splits, 1).
template <int PER>
__global__ void __launch_bounds__(ATT_THREADS) k_decode_attn_group(const AttnArgs a, const RopeDims d, unsigned spin_limit,
                                                                    unsigned *timed_out, unsigned long long *tl) {
  asm volatile("griddepcontrol.launch_dependents;");
  if (threadIdx.x == 0) tl_min(tl, 0);
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int flag;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  unsigned parity = 0;
  const size_t kvh = blockIdx.x % d.nkv, split = blockIdx.x / d.nkv;
  if (!attn_group_item<false, PER, true>(a, d, kvh, split, blockIdx.y, sm, &bar, parity, spin_limit, &flag, nullptr, tl) && threadIdx.x == 0 &&
      timed_out)
    *timed_out = 1u;
}

// Streaming group attention for several sequences.  One CTA per (KV head, split, sequence) walks its
// positions in chunks through a ring of bulk copies; every warp takes G x T = 32 (query head, position)
// pairs of a chunk at a time and keeps its own running maximum, sum and weighted values (online softmax),
// so no barrier separates scores from values and copies overlap arithmetic.
// What bounds it: the cache is read once, so HBM; the form for one sequence (attn_group_item) re-read
// queries and values from shared memory per head -- 76 cycles of shared-memory bandwidth per position --
// and with many waves of short slices paid its set-up and merge 37 times per KV head.  Here queries and
// sums live in registers, a key or value row is read once for all heads, and the 32 partial dot products
// of a lane are reduced together (31 shuffles for 32 sums).
// Measured, 16 sequences at 2040 positions, 8 KV heads of 8 queries x 128: 130 us before; the 4-layer step it is part of went from
// 1.35 to 1.02 ms a token (41 us of HBM time a layer).
constexpr int STREAM_STAGES = 3;
constexpr int STREAM_THREADS = 256;
constexpr int STREAM_WARPS = STREAM_THREADS / 32;
template <int PER> __host__ __device__ constexpr int stream_chunk() { return PER == 4 ? 32 : 64; }  // positions: 32 KiB of keys and values
template <int PER> __host__ __device__ constexpr size_t stream_smem_floats() {
  return size_t(STREAM_STAGES) * 2 * stream_chunk<PER>() * 32 * PER + size_t(ATT_MAX_GROUP) * 32 * PER + 2 * 32 * PER + STREAM_WARPS * 32 +
         2 * STREAM_WARPS * ATT_MAX_GROUP + ATT_MAX_GROUP * ATT_MAX_SPLITS;
}

template <int PER, int G>
__global__ void __launch_bounds__(STREAM_THREADS, 2) k_decode_attn_stream(const AttnArgs a, const RopeDims d, unsigned spin_limit, int extra_arrivals,
                                                                          unsigned *timed_out, unsigned long long *tl) {
  constexpr int T = 32 / G, HD = 32 * PER, CH = stream_chunk<PER>(), ST = STREAM_STAGES;
  static_assert(CH % (STREAM_WARPS * T) == 0, "whole rounds");
  extern __shared__ __align__(128) float sm[];
  float *ring = sm;                                   // [stage][K|V][CH][HD]
  float *qs = ring + ST * 2 * CH * HD;                // [G][HD] rotated queries
  float *kn = qs + ATT_MAX_GROUP * HD, *vn = kn + HD;  // the new position
  float *pbuf = vn + HD;                              // [warp][head][T]
  float *stat = pbuf + STREAM_WARPS * 32;             // [warp][head]{max, sum}
  float *wk = stat + 2 * STREAM_WARPS * ATT_MAX_GROUP;
  __shared__ __align__(8) uint64_t full[ST], empty[ST];
  __shared__ int flag;
  __shared__ volatile int gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t kvh = blockIdx.x % d.nkv, split = blockIdx.x / d.nkv, b = blockIdx.y;
  const int g = int(d.nh / d.nkv), n_splits = a.n_splits;
  const size_t kv_dim = d.nkv * HD;
  asm volatile("griddepcontrol.launch_dependents;");
  if (tid == 0) {
    tl_min(tl, 0);
    gave_up = 0;
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], unsigned(STREAM_WARPS + extra_arrivals));
    }
  }
  __syncthreads();
  const size_t pos = a.positions[b];
  // cached positions 0 .. pos-1 are cut evenly over the splits; split 0 adds the new one
  const size_t len = (pos + n_splits - 1) / n_splits, t0 = min(split * len, pos), t1 = min(t0 + len, pos);
  const int n = int(t1 - t0), n_chunks = (n + CH - 1) / CH;
  float *kc = a.kv + b * d.seq_stride + (a.layer * 2) * d.max_seq * kv_dim + kvh * d.max_seq * HD;
  float *vc = kc + d.max_seq * kv_dim;
  auto fetch = [&](int c) {  // one thread
    const int rows = min(CH, n - c * CH), st = c % ST;
    const size_t t = t0 + size_t(c) * CH;
#ifdef LMB_DEBUG_BOUNDS
    if (!LMB_IN_BOUNDS(size_t(vc - a.kv) + (t + rows) * HD <= a.kv_floats, BOUNDS_KV_SLICE, size_t(vc - a.kv) + (t + rows) * HD)) {
      mbar_arrive_expect_tx(&full[st], 0u);
      return;
    }
#endif
    float *k = ring + st * 2 * CH * HD;
    const unsigned bytes = unsigned(rows) * HD * 4;
    mbar_arrive_expect_tx(&full[st], 2 * bytes);
    bulk_copy_g2s(k, kc + t * HD, bytes, &full[st]);
    bulk_copy_g2s(k + CH * HD, vc + t * HD, bytes, &full[st]);
  };
  if (tid == 0)
    for (int c = 0; c < min(ST, n_chunks); ++c) fetch(c);  // written by earlier steps: not waited for
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid == 0) {
    tl_min(tl, 1);
    tl_max(tl, 2);
  }
  // rotated queries of the group, and the new position (bias, RoPE; pairs (i, i + hd/2))
  constexpr int half = HD / 2;
  const float *cs = a.cs_table + pos * HD;
  for (int i = tid; i < ATT_MAX_GROUP * half; i += STREAM_THREADS) {
    const int h = i / half, j = i - h * half;
    float r0 = 0.0f, r1 = 0.0f;
    if (h < g) {
      const size_t head = kvh * g + h, i0 = (b * d.nh + head) * HD + j;
      const float c = cs[j], sn = cs[half + j];
      float x0 = a.q[i0], x1 = a.q[i0 + half];
      if (a.qb) {
        x0 += a.qb[head * HD + j];
        x1 += a.qb[head * HD + j + half];
      }
      r0 = x0 * c - x1 * sn;
      r1 = x0 * sn + x1 * c;
    }
    qs[h * HD + j] = r0;
    qs[h * HD + j + half] = r1;
  }
  if (split == 0 && tid < half) {
    const int j = tid;
    const float c = cs[j], sn = cs[half + j];
    const size_t k0 = (b * d.nkv + kvh) * HD + j;
    float y0 = a.k[k0], y1 = a.k[k0 + half], v0 = a.v[k0], v1 = a.v[k0 + half];
    if (a.kb) {
      y0 += a.kb[kvh * HD + j];
      y1 += a.kb[kvh * HD + j + half];
    }
    if (a.vb) {
      v0 += a.vb[kvh * HD + j];
      v1 += a.vb[kvh * HD + j + half];
    }
    const float r0 = y0 * c - y1 * sn, r1 = y0 * sn + y1 * c;
    kn[j] = r0; kn[j + half] = r1;
    vn[j] = v0; vn[j + half] = v1;
    kc[pos * HD + j] = r0; kc[pos * HD + j + half] = r1;  // this CTA is the only one that holds the position
    vc[pos * HD + j] = v0; vc[pos * HD + j + half] = v1;
  }
  __syncthreads();
  if (tid == 0) tl_max(tl, 3);
  LaneVec<PER> q[G], acc[G];
#pragma unroll
  for (int h = 0; h < G; ++h) {
    q[h] = ld_lane_vec<PER>(qs + h * HD, lane);
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[h].v[e] = 0.0f;
  }
  const float scale = 1.0f / sqrtf(float(HD));
  const int my_h = lane % G, my_t = lane / G;
  float mrun = -INFINITY, lsum = 0.0f;  // this lane's head; the sum over this lane's positions
  float *pw = pbuf + warp * 32;
  // T positions: rows K[0 .. n_valid-1] and V alike; the rows behind them repeat the last one and weigh nothing
  auto round = [&](const float *K, const float *V, int n_valid) {
    float s[32];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const LaneVec<PER> kk = ld_lane_vec<PER>(K + min(t, n_valid - 1) * HD, lane);
#pragma unroll
      for (int h = 0; h < G; ++h) {
        float x = q[h].v[0] * kk.v[0];
#pragma unroll
        for (int e = 1; e < PER; ++e) x = fmaf(q[h].v[e], kk.v[e], x);
        s[t * G + h] = x;
      }
    }
    // each step a lane keeps half of its sums and hands the other half to its partner: lane l ends with sum l
#pragma unroll
    for (int m = 16; m > 0; m >>= 1)
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const bool up = lane & m;
        const float keep = up ? s[i + m] : s[i], give = up ? s[i] : s[i + m];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
      }
    const bool valid = my_t < n_valid && my_h < g;
    const float x = s[0] * scale;
    float mx = valid ? x : -INFINITY;
#pragma unroll
    for (int m = G; m < 32; m <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
    const float mnew = fmaxf(mrun, mx);
    const float f = mrun == mnew ? 1.0f : expf(mrun - mnew);
    const float p = valid ? expf(x - mnew) : 0.0f;
    lsum = lsum * f + p;
    mrun = mnew;
    __syncwarp();
    pw[my_h * T + my_t] = p;
    __syncwarp();
    if (__any_sync(0xffffffffu, f != 1.0f)) {
#pragma unroll
      for (int h = 0; h < G; ++h) {
        const float fh = __shfl_sync(0xffffffffu, f, h);
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[h].v[e] *= fh;
      }
    }
    LaneVec<PER> vv[T];
#pragma unroll
    for (int t = 0; t < T; ++t) vv[t] = ld_lane_vec<PER>(V + min(t, n_valid - 1) * HD, lane);
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
      for (int t4 = 0; t4 < T; t4 += 4) {
        const float4 pt = *reinterpret_cast<const float4 *>(pw + h * T + t4);
#pragma unroll
        for (int e = 0; e < PER; ++e)
          acc[h].v[e] = fmaf(pt.w, vv[t4 + 3].v[e], fmaf(pt.z, vv[t4 + 2].v[e], fmaf(pt.y, vv[t4 + 1].v[e], fmaf(pt.x, vv[t4].v[e], acc[h].v[e]))));
      }
  };
  auto wait = [&](uint64_t *bar, unsigned parity) {
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
      if (gave_up || ++spins > spin_limit) {
        gave_up = 1;
        return false;
      }
    }
    return true;
  };
  int st = 0, issued = min(ST, n_chunks);
  unsigned par = 0;
  for (int c = 0; c < n_chunks; ++c) {
    // the stage of the chunk before is refilled now: its readers have had this long to finish
    if (tid == 0 && c > 0 && c - 1 + ST < n_chunks) {
      if (wait(&empty[(c - 1) % ST], unsigned((c - 1) / ST) & 1u)) {
        fetch(c - 1 + ST);
        issued = c + ST;
      }
    }
    if (!__all_sync(0xffffffffu, wait(&full[st], par))) break;
    const float *K = ring + st * 2 * CH * HD;
    const int rows = min(CH, n - c * CH);
#pragma unroll 1
    for (int r = warp * T; r < rows; r += STREAM_WARPS * T) round(K + r * HD, K + (CH + r) * HD, min(T, rows - r));
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr_u32(&empty[st])) : "memory");
    if (++st == ST) {
      st = 0;
      par ^= 1u;
    }
  }
  if (split == 0 && warp == 0) round(kn, vn, 1);
  if (tid == 0)  // copies in flight (after a wait that expired) land before the shared memory is used otherwise
    for (int c = max(0, issued - ST); c < issued; ++c)
      for (unsigned s = 0; s < (1u << 20) && !mbar_try_wait(&full[c % ST], unsigned(c / ST) & 1u); ++s) {}
  __syncthreads();
  if (gave_up) {  // uniform: set before the barrier
    if (tid == 0 && timed_out) *timed_out = 1u;
    return;
  }
  // the warps' states meet in the ring
  float *red = ring;  // [warp][head][HD]
#pragma unroll
  for (int m = G; m < 32; m <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, m);
#pragma unroll
  for (int h = 0; h < G; ++h)
    if (h < g) st_lane_vec<PER>(red + (warp * G + h) * HD, lane, acc[h]);
  if (lane < G) {
    stat[2 * (warp * G + lane)] = mrun;
    stat[2 * (warp * G + lane) + 1] = lsum;
  }
  __syncthreads();
  const size_t rec = HD + ATT_REC_PAD;
  if (warp < g) {
    const int h = warp;
    const size_t head = kvh * g + h;
    float gm = -INFINITY, den = 0.0f;
#pragma unroll
    for (int w = 0; w < STREAM_WARPS; ++w) gm = fmaxf(gm, stat[2 * (w * G + h)]);
    LaneVec<PER> tot;
#pragma unroll
    for (int e = 0; e < PER; ++e) tot.v[e] = 0.0f;
#pragma unroll
    for (int w = 0; w < STREAM_WARPS; ++w) {
      const float m = stat[2 * (w * G + h)], l = stat[2 * (w * G + h) + 1];
      const float ws = l == 0.0f ? 0.0f : (m == gm ? 1.0f : expf(m - gm));  // warps without positions weigh nothing
      if (l != 0.0f) {
        const LaneVec<PER> part = ld_lane_vec<PER>(red + (w * G + h) * HD, lane);
        den += ws * l;
#pragma unroll
        for (int e = 0; e < PER; ++e) tot.v[e] += ws * part.v[e];
      }
    }
    if (n_splits == 1) {
      const float inv = 1.0f / den;
#pragma unroll
      for (int e = 0; e < PER; ++e) tot.v[e] *= inv;
      st_lane_vec<PER>(a.out + (b * d.nh + head) * HD, lane, tot);
    } else {
      float *prt = a.partial + ((b * d.nh + head) * n_splits + split) * rec;
      st_lane_vec<PER>(prt, lane, tot);
      if (lane == 0) {
        prt[HD] = gm;
        prt[HD + 1] = den;
      }
    }
  }
  if (tid == 0) {
    tl_max(tl, 4);
    tl_min(tl, 6);
    tl_max(tl, 5);  // of the CTA that merges: again when it has
  }
  if (n_splits == 1) return;
  __syncthreads();
  unsigned *ctr = a.counters + b * d.nkv + kvh;
  if (tid == 0) {
    unsigned before;  // release: this CTA's partial records; acquire: the other splits' records
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(ctr) : "memory");
    flag = (before == unsigned(n_splits - 1));
    if (flag) *ctr = 0u;
  }
  __syncthreads();
  if (!flag || warp >= g) return;
  // last split to arrive: a warp per query head, statistics in one round trip, records in split order
  const size_t head = kvh * g + warp;
  const float *all = a.partial + ((b * d.nh + head) * n_splits) * rec;
  float *w = wk + warp * ATT_MAX_SPLITS;
  const bool h0 = lane < n_splits, h1 = lane + 32 < n_splits;
  const float2 st0 = h0 ? __ldcg(reinterpret_cast<const float2 *>(all + lane * rec + HD)) : make_float2(-INFINITY, 0.0f);
  const float2 st1 = h1 ? __ldcg(reinterpret_cast<const float2 *>(all + (lane + 32) * rec + HD)) : make_float2(-INFINITY, 0.0f);
  float gmx = fmaxf(st0.x, st1.x);
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) gmx = fmaxf(gmx, __shfl_xor_sync(0xffffffffu, gmx, m));
  const float w0 = st0.y == 0.0f ? 0.0f : expf(st0.x - gmx), w1 = st1.y == 0.0f ? 0.0f : expf(st1.x - gmx);  // empty splits weigh nothing
  if (h0) w[lane] = w0;
  if (h1) w[lane + 32] = w1;
  float den = w0 * st0.y + w1 * st1.y;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) den += __shfl_xor_sync(0xffffffffu, den, m);
  __syncwarp();
  LaneVec<PER> tot;
#pragma unroll
  for (int e = 0; e < PER; ++e) tot.v[e] = 0.0f;
  for (int s2 = 0; s2 < n_splits; s2 += 8) {
    LaneVec<PER> pv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (s2 + i < n_splits) pv[i] = ldcg_lane_vec<PER>(all + (s2 + i) * rec, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (s2 + i < n_splits) {
#pragma unroll
        for (int e = 0; e < PER; ++e) tot.v[e] += w[s2 + i] * pv[i].v[e];
      }
  }
  const float inv = 1.0f / den;
#pragma unroll
  for (int e = 0; e < PER; ++e) tot.v[e] *= inv;
  st_lane_vec<PER>(a.out + (b * d.nh + head) * HD, lane, tot);
  if (tid == 0) tl_max(tl, 5);
}

__global__ void k_interleave_rows(const float *src, float *dst, size_t ranks, size_t batch, size_t n) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x, total = ranks * batch * n;
  if (i >= total) return;
  const size_t r = i / (batch * n), b = (i / n) % batch, j = i % n;
  dst[b * ranks * n + r * n + j] = src[i];
}

__global__ void k_silu_mul(const float *gate, const float *up, float *out, size_t n, int gelu) {
  asm volatile("griddepcontrol.launch_dependents;");  // a following GEMV may prefetch its weights
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) {
    const float g = gate[i];
    out[i] = (gelu ? gelu_tanh(g) : g / (1.0f + expf(-g))) * up[i];
  }
}

}  // namespace

int launch_embed_rows(lmb_ctx *ctx, const int *d_tokens, const lmb_weight *embed, size_t vocab, size_t h, size_t batch,
                      float scale, float *d_hidden) {
  dim3 grid(unsigned((h + 255) / 256), unsigned(batch));
  k_embed_rows<<<grid, 256, 0, ctx->stream>>>(d_tokens, embed->kind, embed->d_tiles, embed->bpr, vocab, h, scale, d_hidden);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int launch_add_rmsnorm(lmb_ctx *ctx, float *d_hidden, const float *d_add, const float *d_w, float *d_out, size_t h,
                       size_t batch, float eps) {
  const int threads = h >= 4096 ? 1024 : (h >= 1024 ? 512 : 256);
  k_add_rmsnorm<<<unsigned(batch), threads, 0, ctx->stream>>>(d_hidden, d_add, d_w, d_out, h, eps);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int launch_tp_sum_add_rmsnorm(lmb_ctx *ctx, float *d_hidden, const float *d_w, float *d_out, size_t h, size_t batch, float eps) {
  if (!ctx->xchg.ready || batch * h > ctx->xchg.cap) {
    set_last_error("tensor-parallel sum: exchange block missing or too small");
    return LMB_ERR_STATE;
  }
  const int threads = h >= 4096 ? 1024 : (h >= 1024 ? 512 : 256);
  XchgHeader *hdr = static_cast<XchgHeader *>(ctx->xchg.local);
  const unsigned long long *data =
      reinterpret_cast<const unsigned long long *>(static_cast<const char *>(ctx->xchg.local) + XCHG_HEADER_BYTES);
  k_tp_sum_add_rmsnorm<<<unsigned(batch), threads, 0, ctx->stream>>>(d_hidden, hdr, data, ctx->tp_size, unsigned(ctx->xchg.cap),
                                                                     d_w, d_out, h, eps, ctx->xchg.spin_limit);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int decode_attn_splits(const lmb_ctx *ctx, size_t nh, size_t batch, size_t max_seq) {
  size_t n = (size_t(2) * ctx->sm_count + nh * batch - 1) / (nh * batch);
  const size_t most = (max_seq + 63) / 64;  // no slice shorter than 64 timesteps at full context
  n = n < 1 ? 1 : (n > 32 ? 32 : n);
  return int(n > most ? most : n);
}

// q/k/v are the fresh projections of this step; the kernel applies bias and RoPE, writes the new
// position into the cache and attends over positions 0..pos.
int launch_decode_attn(lmb_ctx *ctx, const float *q, const float *k, const float *v, const float *qb, const float *kb,
                       const float *vb, const float *cs_table, const size_t *positions, float *kv, float *out,
                       float *partial, unsigned *counters, int n_splits, size_t layer, const RopeDims &d0, size_t batch) {
  RopeDims d = d0;
  if (d.hd > ATT_THREADS || d.hd == 0 || ATT_THREADS % d.hd != 0 || d.hd % 2 != 0) {
    set_last_error("decode attention: head_dim must be even and divide 256");
    return LMB_ERR_ARG;
  }
  size_t len = (d.max_seq + n_splits - 1) / n_splits;
  d.split_len = (len + 15) / 16 * 16;
  const size_t smem = (d.split_len + 3 * d.hd + 32 + ATT_THREADS) * sizeof(float);
  AttnArgs a{q, k, v, qb, kb, vb, cs_table, positions, kv, out, partial, counters, n_splits, layer};
  dim3 grid(unsigned(d.nh), unsigned(n_splits), unsigned(batch));
  k_decode_attn<<<grid, ATT_THREADS, smem, ctx->stream>>>(a, d);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

size_t attn_partial_floats(size_t batch, size_t nh, size_t hd) { return batch * nh * ATT_MAX_SPLITS * (hd + ATT_REC_PAD); }

// Splits of the streaming form: two CTAs per SM; a wave lasts as long as a split's positions plus its fixed
// part (set-up, first copies, merging the warps: about 64 positions' worth).
int stream_splits(size_t nkv, size_t batch, size_t max_seq, size_t sm_count) {
  const size_t pairs = nkv * batch, slots = 2 * sm_count;
  size_t best = 1, best_cost = ~size_t(0);
  for (size_t s = 1; s <= size_t(ATT_MAX_SPLITS) && (s == 1 || max_seq / s >= 32); ++s) {
    const size_t cost = (pairs * s + slots - 1) / slots * ((max_seq + s - 1) / s + 64) + (s > 1 ? 16 : 0);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return int(best);
}

AttnGroupPlan plan_attn_group(size_t nh, size_t nkv, size_t hd, size_t max_seq, size_t batch, size_t want_items, size_t smem_bytes) {
  AttnGroupPlan pl{false, 1, 0, 0, 0};
  if (nkv == 0 || nh % nkv != 0) return pl;
  const size_t g = nh / nkv;
  if (g > size_t(ATT_MAX_GROUP) || (hd != 64 && hd != 128)) return pl;
  pl.per = int(hd / 32);
  // longest slice whose rows, queries and scores fit
  const size_t fixed = g * hd + size_t(ATT_MAX_GROUP) * ATT_MAX_SPLITS + 2 * ATT_MAX_GROUP, budget = smem_bytes / sizeof(float);
  if (budget <= fixed + 8 * (2 * hd + g)) return pl;
  const size_t cap = (budget - fixed) / (2 * hd + g) / 8 * 8;
  const size_t min_splits = (max_seq + cap - 1) / cap;
  size_t want = (want_items + nkv * batch - 1) / (nkv * batch);
  size_t n = std::max(min_splits, std::max<size_t>(want, 1));
  n = std::min<size_t>(n, ATT_MAX_SPLITS);
  n = std::min<size_t>(n, std::max<size_t>(1, (max_seq + 7) / 8));  // no slice shorter than 8 positions at full context
  if (n < min_splits) return pl;
  pl.n_splits = int(n);
  pl.split_len = ((max_seq + n - 1) / n + 7) / 8 * 8;
  if (pl.split_len > cap) return pl;
  pl.smem_bytes = attn_group_smem_floats(pl.split_len, hd, g) * sizeof(float);
  pl.ok = true;
  return pl;
}

int launch_decode_attn_group(lmb_ctx *ctx, const float *q, const float *k, const float *v, const float *qb, const float *kb,
                             const float *vb, const float *cs_table, const size_t *positions, float *kv, float *out,
                             float *partial, unsigned *counters, const AttnGroupPlan &plan, size_t layer, const RopeDims &d0,
                             size_t batch) {
  RopeDims d = d0;
  d.split_len = plan.split_len;
  AttnArgs a{q, k, v, qb, kb, vb, cs_table, positions, kv, out, partial, counters, plan.n_splits, layer};
#ifdef LMB_DEBUG_BOUNDS
  a.kv_floats = d.seq_stride * batch;  // the cache holds at least the sequences of this launch
#endif
  dim3 grid(unsigned(d.nkv * size_t(plan.n_splits)), unsigned(batch));
  unsigned *flag = ctx->d_fault;  // set when a bounded wait for the bulk copies runs out
  // programmatic dependent launch: the CTAs start fetching their cache slices while the q/k/v
  // projections finish, and wait for those only before they read the fresh vectors
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(ATT_THREADS);
  cfg.dynamicSmemBytes = plan.smem_bytes;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  static const bool attn_pdl = [] {  // LMB_ATTN_PDL=0: the attention kernel starts only when the q/k/v projections have finished
    const char *e = std::getenv("LMB_ATTN_PDL");
    return !(e && e[0] == '0');
  }();
  cfg.numAttrs = ctx->pdl && attn_pdl ? 1 : 0;
  // one sequence: one wave of CTAs, bound by their latency; several: bound by throughput (the streaming form, which
  // takes nothing of `plan` but the head size: it has splits of its own, of any length)
  if (batch == 1) {
    unsigned long long *tl = timeline_slot(ctx);
    if (plan.per == 4) LMB_CUDA(cudaLaunchKernelEx(&cfg, k_decode_attn_group<4>, a, d, ctx->xchg.spin_limit, flag, tl));
    else LMB_CUDA(cudaLaunchKernelEx(&cfg, k_decode_attn_group<2>, a, d, ctx->xchg.spin_limit, flag, tl));
  } else {
    a.n_splits = ctx->attn_force_splits ? ctx->attn_force_splits : stream_splits(d.nkv, batch, d.max_seq, size_t(ctx->sm_count));
    const unsigned limit = ctx->attn_spin_limit ? ctx->attn_spin_limit : ctx->xchg.spin_limit;
    const int extra = ctx->attn_extra_arrivals;
    cfg.gridDim = dim3(unsigned(d.nkv * size_t(a.n_splits)), unsigned(batch));
    cfg.dynamicSmemBytes = (plan.per == 4 ? stream_smem_floats<4>() : stream_smem_floats<2>()) * sizeof(float);
    // four query heads per KV head or fewer: eight positions per round instead of four
    if (plan.per == 4) LMB_CUDA(cudaLaunchKernelEx(&cfg, k_decode_attn_stream<4, 8>, a, d, limit, extra, flag, timeline_slot(ctx)));
    else if (d.nh / d.nkv > 4) LMB_CUDA(cudaLaunchKernelEx(&cfg, k_decode_attn_stream<2, 8>, a, d, limit, extra, flag, timeline_slot(ctx)));
    else LMB_CUDA(cudaLaunchKernelEx(&cfg, k_decode_attn_stream<2, 4>, a, d, limit, extra, flag, timeline_slot(ctx)));
  }
  ctx->launches++;
  return LMB_OK;
}

int launch_interleave_rows(lmb_ctx *ctx, const float *src, float *dst, size_t ranks, size_t batch, size_t n) {
  const size_t total = ranks * batch * n;
  k_interleave_rows<<<unsigned((total + 255) / 256), 256, 0, ctx->stream>>>(src, dst, ranks, batch, n);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int launch_silu_mul(lmb_ctx *ctx, const float *gate, const float *up, float *out, size_t n, bool gelu) {
  k_silu_mul<<<unsigned((n + 255) / 256), 256, 0, ctx->stream>>>(gate, up, out, n, gelu ? 1 : 0);
  ctx->launches++;
  LMB_CUDA(cudaGetLastError());
  return LMB_OK;
}

int configure_decode_ops(lmb_ctx *ctx) {
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ctx->smem_optin) - 1024));
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn_group<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ATTN_GROUP_SMEM)));
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn_group<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ATTN_GROUP_SMEM)));
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn_stream<4, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(stream_smem_floats<4>() * 4)));
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn_stream<2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(stream_smem_floats<2>() * 4)));
  LMB_CUDA(cudaFuncSetAttribute(k_decode_attn_stream<2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(stream_smem_floats<2>() * 4)));
  return LMB_OK;
}

}  // namespace lmb

extern "C" int lmb_debug_attn_stream(lmb_ctx *ctx, int n_splits, int extra_arrivals, unsigned spin_limit) {
  LMB_REQUIRE(ctx && n_splits >= 0 && n_splits <= lmb::ATT_MAX_SPLITS && extra_arrivals >= 0, "lmb_debug_attn_stream: bad argument");
  ctx->attn_force_splits = n_splits;
  ctx->attn_extra_arrivals = extra_arrivals;
  ctx->attn_spin_limit = spin_limit;
  return LMB_OK;
}
