// Router post-processing and the stable counting sort of routed slots.
//
// No atomics whose order could show, so every integer output is reproducible:
//   a handful of tokens         route_fused_kernel: one CTA does everything (route_fused() says up to where);
//   otherwise                   route_chunk_kernel: one CTA per chunk of slots ((soft-max + top-k + renormalise when fed
//                               logits) and a histogram of the chunk's expert ids), then route_rank_kernel: every CTA adds
//                               up the histograms of all chunks (one chunk per SM up to 4.8 million slots, so that is a few loads
//                               per thread out of L2 and spares a launch for a scan), derives the offsets and ranks its own
//                               slots -> pos / order / padded row / slot-of-row.  A chunk holds at most 32,768 slots, so with
//                               the slots the chunks become more and those loads grow with their square: beyond kScanChunks
//                               of them route_scan_kernel comes in between and leaves every chunk's prefix and the totals.
// The result equals sort_indices() of the reference (modal/moe_permute.py:240-264): a stable sort
// of slots i = t*k + j by expert id, order[p] = slot at sorted position p, pos = inverse of order.
#pragma once

#include "common.cuh"

namespace lewi {

constexpr int kRouteThreads = 512;
constexpr int kRouteWarps = kRouteThreads / kWarp;
constexpr int kMinChunkSlots = 128;     // lewi_route_workspace_bytes counts on it
constexpr int kMaxChunkSlots = 32768;   // a chunk's expert ids and 17 rows of 512 counters fit in 200 KB of shared memory
constexpr int kScanChunks = 512;        // see route_scan_kernel
constexpr int kMaxExperts = 512;
constexpr int kMaxTopK = 32;

__device__ __forceinline__ uint32_t float_order_key(float v) {
  uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float float_of_key(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

// Per-warp histogram of s_e[begin, end) into run[E] (a row private to this warp).
__device__ __forceinline__ void warp_histogram(const int* s_e, int begin, int end, int* run, int lane) {
  for (int base = begin; base < end; base += kWarp) {
    int i = base + lane;
    int e = (i < end) ? s_e[i] : -1;
    unsigned mask = __match_any_sync(0xffffffffu, e);
    int leader = __ffs(mask) - 1;
    if (e >= 0 && lane == leader) run[e] += __popc(mask);
    __syncwarp();
  }
}

// ER = experts held per lane (E <= 32*ER); NT = tokens a warp works on at once.  The soft-max and the k rounds of
// arg-max are chains of dependent shuffles; NT independent chains side by side keep the warp's issue slots busy
// while one of them waits.  Token i of the group is rows[i] (null: no such token); its results are the same bits
// whatever NT is.
template <int ER, int NT>
__device__ __forceinline__ void warp_softmax_topk(const float* const (&rows)[NT], int E, int k, int lane,
                                                  int (&out_idx)[NT], float (&out_w)[NT], float (&p)[NT][ER]) {
  // order-preserving image of the logits; 0: no such expert, or already chosen (the one NaN whose image is 0 takes 1)
  uint32_t key[NT][ER];
  float mx[NT], sum[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    uint32_t best = 0;
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      const int e = lane + r * kWarp;
      const bool in = e < E && rows[i] != nullptr;
      const float l = in ? rows[i][e] : 0.f;
      key[i][r] = in ? max(float_order_key(l), 1u) : 0u;
      best = max(best, key[i][r]);
      p[i][r] = l;
    }
    mx[i] = float_of_key(__reduce_max_sync(0xffffffffu, best));
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    sum[i] = 0.f;
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      p[i][r] = key[i][r] != 0u ? expf(p[i][r] - mx[i]) : 0.f;
      sum[i] += p[i][r];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < NT; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const float inv = 1.0f / sum[i];
#pragma unroll
    for (int r = 0; r < ER; ++r) p[i][r] *= inv;
  }

  // k rounds of warp arg-max on (logit descending, index ascending): one warp reduction finds the largest key, one the
  // lowest expert that holds it (a 64-bit key through five shuffles each took four times as long).
  float vsum[NT], my_v[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    vsum[i] = 0.f;
    my_v[i] = 0.f;
    out_idx[i] = 0;
  }
  for (int j = 0; j < k; ++j) {
    uint32_t best[NT], cand[NT];
    float best_p[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      best[i] = key[i][0];
#pragma unroll
      for (int r = 1; r < ER; ++r) best[i] = max(best[i], key[i][r]);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) best[i] = __reduce_max_sync(0xffffffffu, best[i]);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      cand[i] = 0xFFFFFFFFu;
      best_p[i] = 0.f;
#pragma unroll
      for (int r = ER - 1; r >= 0; --r) {
        if (key[i][r] == best[i]) {
          cand[i] = lane + r * kWarp;
          best_p[i] = p[i][r];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) cand[i] = __reduce_min_sync(0xffffffffu, cand[i]);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int e_win = rows[i] != nullptr ? (int)cand[i] : 0;
      const float v = __shfl_sync(0xffffffffu, best_p[i], e_win & (kWarp - 1));
#pragma unroll
      for (int r = 0; r < ER; ++r) key[i][r] = lane + r * kWarp == e_win ? 0u : key[i][r];
      vsum[i] += v;
      if (lane == j) {
        my_v[i] = v;
        out_idx[i] = e_win;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) out_w[i] = my_v[i] / vsum[i];
}

// tokens a warp works on at once: fewer when a lane holds many experts
template <int ER> struct RouteGroup { static constexpr int NT = ER <= 4 ? 4 : (ER <= 8 ? 2 : 1); };

// Whether one CTA routes the whole call: while its warps take their tokens in one round, or where there is one chunk of slots anyway
// (and its experts do not make the kernel spill).  A second round doubles the time, two launches spread the tokens over the SMs.
// One CTA and two launches, in us: 128 experts top-6 8 tokens 9.1 and 12.1, 64 12.7 and 12.8, 128 20.6 and 13.0; 256 top-8 32 12.8 and
// 13.8, 64 19.4 and 13.5; 512 top-8 16 16.3 and 18.1, 32 23.0 and 15.6; top-1 128 tokens (one chunk): 64 experts 10.6 and
// 13.1, 256 18.3 and 21.5, 512 38.7 and 32.0.
inline bool route_fused(long long tokens, int E, int n_chunks) {
  const int round = kRouteWarps * (E <= 128 ? RouteGroup<4>::NT : (E <= 256 ? RouteGroup<8>::NT : RouteGroup<16>::NT));
  return tokens > 0 && (tokens <= round || (n_chunks == 1 && E <= 256));
}

struct RouteChunkArgs {
  const float* logits;        // [T,E] or null
  const int32_t* flat_in;     // [M] or null (when logits == null)
  int32_t* topk_idx;          // [T,k] (written when logits != null)
  float* topk_w;              // [T,k]
  int32_t* chunk_hist;        // [n_chunks, E]
  float* chunk_probs;         // [n_chunks, E] or null
  int32_t* row_slot;          // [mpad] or null: filled with -1 here
  long long num_slots;        // M
  long long mpad;
  int E, k, chunk_slots;
};

// Routes the tokens of one chunk: top-k of every token to global memory, its experts to s_e, the soft-max column sums of every
// warp to s_prob [kRouteWarps][E] (when wanted).
template <int ER>
__device__ __forceinline__ void route_chunk_tokens(const float* logits, int32_t* topk_idx, float* topk_w, long long tok0, int n_tok, int E,
                                                   int k, int* s_e, float* s_prob, bool want_probs, int lane, int warp) {
  constexpr int NT = RouteGroup<ER>::NT;
  float pacc[ER];
#pragma unroll
  for (int r = 0; r < ER; ++r) pacc[r] = 0.f;
  for (int t0 = warp; t0 < n_tok; t0 += kRouteWarps * NT) {   // tokens t0, t0 + kRouteWarps, ...
    const float* rows[NT];
    float p[NT][ER];
    int idx[NT];
    float w[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = t0 + i * kRouteWarps;
      rows[i] = t < n_tok ? logits + (tok0 + t) * E : nullptr;
    }
    warp_softmax_topk<ER, NT>(rows, E, k, lane, idx, w, p);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = t0 + i * kRouteWarps;
      if (t >= n_tok) continue;
#pragma unroll
      for (int r = 0; r < ER; ++r) pacc[r] += p[i][r];
      if (lane < k) {
        const long long s = (tok0 + t) * k + lane;
        topk_idx[s] = idx[i];
        topk_w[s] = w[i];
        s_e[t * k + lane] = idx[i];
      }
    }
  }
  if (want_probs) {
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      const int e = lane + r * kWarp;
      if (e < E) s_prob[warp * E + e] = pacc[r];
    }
  }
}

template <int ER>
__global__ void __launch_bounds__(kRouteThreads) route_chunk_kernel(RouteChunkArgs a) {
  extern __shared__ int s_mem[];
  int* s_e = s_mem;                                 // [chunk_slots]
  int* s_hist = s_mem + a.chunk_slots;              // [E]
  float* s_prob = reinterpret_cast<float*>(s_hist + a.E);   // [kRouteWarps][E]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long chunk = blockIdx.x;
  const long long slot0 = chunk * a.chunk_slots;
  const int n_slots = (int)min((long long)a.chunk_slots, a.num_slots - slot0);

  for (int i = tid; i < a.E; i += kRouteThreads) s_hist[i] = 0;
  grid_wait();
  grid_launch();
  if (a.row_slot != nullptr) {
    for (long long r = (long long)blockIdx.x * kRouteThreads + tid; r < a.mpad; r += (long long)gridDim.x * kRouteThreads)
      a.row_slot[r] = -1;
  }
  if (a.logits != nullptr) {
    route_chunk_tokens<ER>(a.logits, a.topk_idx, a.topk_w, slot0 / a.k, n_slots / a.k, a.E, a.k, s_e, s_prob, a.chunk_probs != nullptr,
                           lane, warp);
  } else {
    for (int i = tid; i < n_slots; i += kRouteThreads) {
      const int e = a.flat_in[slot0 + i];
      if (e < 0 || e >= a.E) raise_status(LEWI_STATUS_BAD_INDEX);
      s_e[i] = (e < 0 || e >= a.E) ? -1 : e;
    }
  }
  __syncthreads();
  for (int i = tid; i < n_slots; i += kRouteThreads)
    if (s_e[i] >= 0) atomicAdd(&s_hist[s_e[i]], 1);   // counts: the order of the additions does not show
  __syncthreads();
  for (int e = tid; e < a.E; e += kRouteThreads) {
    a.chunk_hist[chunk * a.E + e] = s_hist[e];
    if (a.chunk_probs != nullptr) {
      float ps = 0.f;
#pragma unroll
      for (int w = 0; w < kRouteWarps; ++w) ps += s_prob[w * a.E + e];
      a.chunk_probs[chunk * a.E + e] = ps;
    }
  }
}

struct RouteTables {
  int32_t* counts;       // [E] or null
  int32_t* offsets;      // [E+1] or null
  int32_t* pad_offsets;  // [E+1] or null
  int32_t* block_expert; // [nbmax] or null
  int32_t* n_blocks;     // [1] or null
  float* probs_sum;      // [E] or null
  float* aux_loss;       // [1] or null: E * sum_e (counts_e / num_slots) * (probs_sum_e / num_tokens)
  int32_t* order;        // [M] or null
  int32_t* pos;          // [M] or null
  int32_t* pad_pos;      // [M] or null
  int32_t* row_slot;     // [mpad] or null
  long long num_slots, num_tokens;
  int E, block, nbmax;
};

// s_off[e] / s_pad[e]: exclusive prefix of the counts and of the counts rounded up to `block`, for e in [0, E].  All threads;
// s_tmp holds two values per warp.  Ends with a barrier.
__device__ __forceinline__ void expert_offsets(const int* s_cnt, int E, int block, int* s_off, int* s_pad, int* s_tmp, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  static_assert(kMaxExperts <= kRouteThreads, "one expert per thread");
  const int c = tid < E ? s_cnt[tid] : 0;
  int a = c, b = block > 0 ? (c + block - 1) / block * block : 0;
  const int b0 = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) {
      a += ua;
      b += ub;
    }
  }
  if (lane == 31) {
    s_tmp[2 * warp] = a;
    s_tmp[2 * warp + 1] = b;
  }
  __syncthreads();
  int pa = 0, pb = 0;
  for (int w = 0; w < warp; ++w) {
    pa += s_tmp[2 * w];
    pb += s_tmp[2 * w + 1];
  }
  if (tid < E) {
    s_off[tid] = pa + a - c;
    s_pad[tid] = pb + b - b0;
    if (tid == E - 1) {
      s_off[E] = pa + a;
      s_pad[E] = pb + b;
    }
  }
  __syncthreads();
}

// Tables over experts and blocks.  `part` of `parts` CTAs writes its share of the block table, part 0 everything else.
__device__ __forceinline__ void write_tables(const RouteTables& t, const int* s_cnt, const int* s_off, const int* s_pad, int tid, int part,
                                             int parts) {
  if (part == 0) {
    for (int x = tid; x <= t.E; x += kRouteThreads) {
      if (t.offsets != nullptr) t.offsets[x] = s_off[x];
      if (t.pad_offsets != nullptr) t.pad_offsets[x] = s_pad[x];
      if (x < t.E && t.counts != nullptr) t.counts[x] = s_cnt[x];
    }
    if (tid == 0 && t.n_blocks != nullptr && t.block > 0) t.n_blocks[0] = s_pad[t.E] / t.block;
  }
  if (t.block_expert != nullptr && t.block > 0) {
    const int nb = s_pad[t.E] / t.block;
    for (int b = part * kRouteThreads + tid; b < t.nbmax; b += parts * kRouteThreads) {
      int val = -1;
      if (b < nb) {
        const int row = b * t.block;
        int lo = 0, hi = t.E;  // largest x with s_pad[x] <= row
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (s_pad[mid] <= row) lo = mid; else hi = mid;
        }
        val = lo;
      }
      t.block_expert[b] = val;
    }
  }
}

// Load-balance loss from the counts and the probability sums: fixed order (within a lane, then a butterfly), one warp.
__device__ __forceinline__ void write_aux_loss(const RouteTables& t, const int* s_cnt, const float* s_ps, int lane) {
  float acc = 0.f;
  for (int x = lane; x < t.E; x += 32) acc += (float)s_cnt[x] * s_ps[x];
  acc = warp_sum(acc);
  const float denom = (float)t.num_slots * (float)t.num_tokens;
  if (lane == 0) t.aux_loss[0] = denom > 0.f ? acc * (float)t.E / denom : 0.f;
}

// Stable ranks of the slots s_e[0, n_slots) of one chunk, whose slots are slot0, slot0 + 1, ... and before which s_base[e] slots
// chose expert e.  Warps own consecutive runs of slots; s_run is [kRouteWarps][E].
__device__ __forceinline__ void rank_slots(const RouteTables& t, const int* s_e, int n_slots, long long slot0, const int* s_base, const int* s_off,
                                           const int* s_pad, int* s_run, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kRouteWarps * t.E; i += kRouteThreads) s_run[i] = 0;
  __syncthreads();
  const int spw = ((n_slots + kRouteWarps - 1) / kRouteWarps + kWarp - 1) / kWarp * kWarp;
  const int begin = min(warp * spw, n_slots), end = min(begin + spw, n_slots);
  int* run = s_run + warp * t.E;
  warp_histogram(s_e, begin, end, run, lane);
  __syncthreads();
  // exclusive prefix over warps, seeded with the prefix over earlier chunks
  for (int e = tid; e < t.E; e += kRouteThreads) {
    int c[kRouteWarps], at = s_base != nullptr ? s_base[e] : 0;
#pragma unroll
    for (int w = 0; w < kRouteWarps; ++w) c[w] = s_run[w * t.E + e];
#pragma unroll
    for (int w = 0; w < kRouteWarps; ++w) {
      s_run[w * t.E + e] = at;
      at += c[w];
    }
  }
  __syncthreads();
  for (int base = begin; base < end; base += kWarp) {
    const int i = base + lane;
    const int e = (i < end) ? s_e[i] : -1;
    const unsigned mask = __match_any_sync(0xffffffffu, e);
    const int leader = __ffs(mask) - 1;
    int rank = 0;
    if (e >= 0) rank = run[e] + __popc(mask & ((1u << lane) - 1u));
    __syncwarp();
    if (e >= 0 && lane == leader) run[e] += __popc(mask);
    __syncwarp();
    if (e >= 0) {
      const long long slot = slot0 + i;
      const int p = s_off[e] + rank;
      if (t.pos != nullptr) t.pos[slot] = p;
      if (t.order != nullptr) t.order[p] = (int)slot;
      if (t.pad_offsets != nullptr) {
        const int pp = s_pad[e] + rank;
        if (t.pad_pos != nullptr) t.pad_pos[slot] = pp;
        if (t.row_slot != nullptr) t.row_slot[pp] = (int)slot;
      }
    }
  }
}

// Histograms of all chunks -> what the earlier chunks hold, and the totals as row n_chunks: a CTA per 32 experts, whose warps take a run
// of chunks each, add it up and walk it again.  Sorting over 512 / 128 / 16 experts, without and with it (chunks of 32,768): 306 chunks
// 0.35 and 0.33 / 0.31 and 0.30 / 0.202 and 0.207 ms, 611 chunks 0.71 and 0.61 / 0.58 and 0.56 / 0.398 and 0.399, 300 million slots 35
// and 9.2 / 12.9 and 8.7 / 5.3 and 4.7, 1.5 billion 1007 and 46 / 220 and 42.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) route_scan_kernel(int32_t* chunk_hist, int n_chunks, int E) {
  constexpr int NW = kScanThreads / kWarp;
  __shared__ int s_sum[NW][kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * kWarp + lane;
  const int per = (n_chunks + NW - 1) / NW, c0 = min(warp * per, n_chunks), c1 = min(c0 + per, n_chunks);
  const bool live = e < E;
  int32_t* col = chunk_hist + e;
  int sum = 0;
#pragma unroll 8
  for (int c = c0; c < c1; ++c) sum += live ? col[(long long)c * E] : 0;
  s_sum[warp][lane] = sum;
  __syncthreads();
  int run = 0;
  for (int w = 0; w < warp; ++w) run += s_sum[w][lane];
#pragma unroll 8
  for (int c = c0; c < c1; ++c) {
    const int h = live ? col[(long long)c * E] : 0;
    if (live) col[(long long)c * E] = run;
    run += h;
  }
  if (warp == NW - 1 && live) col[(long long)n_chunks * E] = run;
}

struct RouteRankArgs {
  RouteTables t;
  const int32_t* flat;        // [M] expert id per slot
  const int32_t* chunk_hist;  // [n_chunks, E], or scanned: [n_chunks + 1, E]
  const float* chunk_probs;   // [n_chunks, E] or null
  int n_chunks, chunk_slots;
  bool scanned;
};

__global__ void __launch_bounds__(kRouteThreads) route_rank_kernel(RouteRankArgs a) {
  extern __shared__ int s_mem[];
  __shared__ int s_cnt[kMaxExperts], s_base[kMaxExperts], s_off[kMaxExperts + 1], s_pad[kMaxExperts + 1], s_tmp[2 * kRouteWarps];
  __shared__ float s_ps[kMaxExperts];
  int* s_e = s_mem;                    // [chunk_slots]
  int* s_run = s_mem + a.chunk_slots;  // [kRouteWarps][E], at least kRouteThreads
  const int tid = threadIdx.x, E = a.t.E, chunk = blockIdx.x;
  const long long slot0 = (long long)chunk * a.chunk_slots;
  const int n_slots = (int)max(0LL, min((long long)a.chunk_slots, a.t.num_slots - slot0));
  for (int e = tid; e < E; e += kRouteThreads) {
    s_cnt[e] = 0;
    s_base[e] = 0;
  }
  grid_wait();
  grid_launch();
  for (int i = tid; i < n_slots; i += kRouteThreads) {
    const int e = a.flat[slot0 + i];
    s_e[i] = (e < 0 || e >= E) ? -1 : e;
  }
  __syncthreads();
  // totals of all chunks and of the earlier ones: an expert's chunks are dealt over kRouteThreads / E threads
  const int parts = kRouteThreads / E, e = tid % E, part = tid / E;
  if (a.scanned) {
    if (tid < E) {
      s_base[tid] = a.chunk_hist[(long long)chunk * E + tid];
      s_cnt[tid] = a.chunk_hist[(long long)a.n_chunks * E + tid];
    }
  } else if (part < parts) {
    int tot = 0, before = 0;
#pragma unroll 8
    for (int c = part; c < a.n_chunks; c += parts) {
      const int h = a.chunk_hist[(long long)c * E + e];
      tot += h;
      before += c < chunk ? h : 0;
    }
    if (tot != 0) atomicAdd(&s_cnt[e], tot);
    if (before != 0) atomicAdd(&s_base[e], before);
  }
  __syncthreads();
  expert_offsets(s_cnt, E, a.t.block, s_off, s_pad, s_tmp, tid);
  write_tables(a.t, s_cnt, s_off, s_pad, tid, chunk, gridDim.x);
  rank_slots(a.t, s_e, n_slots, slot0, s_base, s_off, s_pad, s_run, tid);
  if (a.t.probs_sum != nullptr && a.chunk_probs != nullptr && chunk == (int)gridDim.x - 1) {
    // column sums of the soft-max: parts of the chunks, added in a fixed order
    float* s_part = reinterpret_cast<float*>(s_run);
    __syncthreads();
    if (part < parts) {
      float ps = 0.f;
#pragma unroll 8
      for (int c = part; c < a.n_chunks; c += parts) ps += a.chunk_probs[(long long)c * E + e];
      s_part[part * E + e] = ps;
    }
    __syncthreads();
    for (int x = tid; x < E; x += kRouteThreads) {
      float ps = 0.f;
      for (int q = 0; q < parts; ++q) ps += s_part[q * E + x];
      a.t.probs_sum[x] = ps;
      s_ps[x] = ps;
    }
    __syncthreads();
    if (a.t.aux_loss != nullptr && tid < 32) write_aux_loss(a.t, s_cnt, s_ps, tid);
  }
}

struct RouteFusedArgs {
  RouteTables t;
  const float* logits;
  int32_t* topk_idx;
  float* topk_w;
  long long mpad;
  int k;
};

// Everything for a handful of tokens in one CTA: at decode sizes the three steps cost their launches, not their work.
template <int ER>
__global__ void __launch_bounds__(kRouteThreads) route_fused_kernel(RouteFusedArgs a) {
  extern __shared__ int s_mem[];
  __shared__ int s_cnt[kMaxExperts], s_off[kMaxExperts + 1], s_pad[kMaxExperts + 1], s_tmp[2 * kRouteWarps];
  __shared__ float s_ps[kMaxExperts];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, E = a.t.E;
  const int n_slots = (int)a.t.num_slots;
  int* s_e = s_mem;                             // [n_slots]
  int* s_run = s_mem + (n_slots + 3) / 4 * 4;   // [kRouteWarps][E], the column sums of the soft-max before that
  float* s_prob = reinterpret_cast<float*>(s_run);
  for (int e = tid; e < E; e += kRouteThreads) s_cnt[e] = 0;
  grid_wait();
  grid_launch();
  if (a.t.row_slot != nullptr)
    for (long long r = tid; r < a.mpad; r += kRouteThreads) a.t.row_slot[r] = -1;
  route_chunk_tokens<ER>(a.logits, a.topk_idx, a.topk_w, 0, n_slots / a.k, E, a.k, s_e, s_prob, a.t.probs_sum != nullptr, lane, warp);
  __syncthreads();
  for (int i = tid; i < n_slots; i += kRouteThreads) atomicAdd(&s_cnt[s_e[i]], 1);
  if (a.t.probs_sum != nullptr) {
    for (int e = tid; e < E; e += kRouteThreads) {
      float ps = 0.f;
#pragma unroll
      for (int w = 0; w < kRouteWarps; ++w) ps += s_prob[w * E + e];
      a.t.probs_sum[e] = ps;
      s_ps[e] = ps;
    }
  }
  __syncthreads();
  expert_offsets(s_cnt, E, a.t.block, s_off, s_pad, s_tmp, tid);
  if (a.t.aux_loss != nullptr && warp == kRouteWarps - 1) write_aux_loss(a.t, s_cnt, s_ps, lane);
  write_tables(a.t, s_cnt, s_off, s_pad, tid, 0, 1);
  rank_slots(a.t, s_e, n_slots, 0, nullptr, s_off, s_pad, s_run, tid);
}

// ------------------------------------------------------------------------------------------------
// Backward of softmax -> top-k -> renormalise.  One warp per token.
template <int ER>
__global__ void __launch_bounds__(256) router_topk_bwd_kernel(const float* __restrict__ logits,
                                                              const int32_t* __restrict__ topk_idx,
                                                              const float* __restrict__ dw,
                                                              const float* __restrict__ dw_partial, int dw_parts,
                                                              const int32_t* __restrict__ pad_pos,
                                                              float* __restrict__ dw_out,
                                                              float* __restrict__ dlogits,
                                                              __nv_bfloat16* __restrict__ dlogits_bf16, long long T,
                                                              int E, int k, const int32_t* __restrict__ counts,
                                                              float aux_coef, float* __restrict__ bias_partial) {
  __shared__ float s_bias[kMaxExperts];
  const int lane = threadIdx.x & 31;
  const long long warp_global = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  // gradient of the load-balance loss with respect to the soft-max probabilities of any token: the token
  // fractions are constants, so dL/dp[t,e] = aux_coef * counts[e]
  float cvec[ER], bias_acc[ER];
#pragma unroll
  for (int r = 0; r < ER; ++r) {
    const int e = lane + r * kWarp;
    cvec[r] = (counts != nullptr && e < E) ? aux_coef * (float)counts[e] : 0.f;
    bias_acc[r] = 0.f;
  }
  for (long long t = warp_global; t < T; t += n_warps) {
    const float* row = logits + t * E;
    float l[ER], p[ER];
    float mx = -INFINITY;
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      int e = lane + r * kWarp;
      l[r] = (e < E) ? row[e] : -INFINITY;
      mx = fmaxf(mx, l[r]);
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      int e = lane + r * kWarp;
      p[r] = (e < E) ? expf(l[r] - mx) : 0.f;
      sum += p[r];
    }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
#pragma unroll
    for (int r = 0; r < ER; ++r) p[r] *= inv;
    int my_e = 0;
    float my_v = 0.f, my_dw = 0.f;
    if (lane < k) {
      my_e = topk_idx[t * k + lane];
      my_e = min(max(my_e, 0), E - 1);
      my_v = expf(row[my_e] - mx) * inv;
      if (dw != nullptr) {
        my_dw = dw[t * k + lane];
      } else {  // the routing-weight gradient arrives as per-row pieces written by the dH GEMM's epilogue
        const long long pr = pad_pos[t * k + lane];
        for (int p = 0; p < dw_parts; ++p) my_dw += dw_partial[pr * dw_parts + p];
      }
      if (dw_out != nullptr) dw_out[t * k + lane] = my_dw;
    }
    const float S = warp_sum(my_v);
    const float wj = my_v / S;
    const float dot = warp_sum(my_dw * wj);
    const float dv = (lane < k) ? (my_dw - dot) / S : 0.f;
    const float pdp = warp_sum(my_v * dv);
    float dl[ER];
    float pc = 0.f;
    if (counts != nullptr) {
#pragma unroll
      for (int r = 0; r < ER; ++r) pc += p[r] * cvec[r];
      pc = warp_sum(pc);
    }
#pragma unroll
    for (int r = 0; r < ER; ++r) dl[r] = -p[r] * pdp + p[r] * (cvec[r] - pc);
    for (int j = 0; j < k; ++j) {
      int ej = __shfl_sync(0xffffffffu, my_e, j);
      float dvj = __shfl_sync(0xffffffffu, dv, j);
      if ((ej & (kWarp - 1)) == lane) {
#pragma unroll
        for (int r = 0; r < ER; ++r)
          if ((ej >> 5) == r) dl[r] += p[r] * dvj;
      }
    }
#pragma unroll
    for (int r = 0; r < ER; ++r) {
      int e = lane + r * kWarp;
      if (e < E) {
        if (dlogits != nullptr) dlogits[t * E + e] = dl[r];
        if (dlogits_bf16 != nullptr) dlogits_bf16[t * E + e] = __float2bfloat16_rn(dl[r]);
      }
      bias_acc[r] += dl[r];
    }
  }
  if (bias_partial != nullptr) {
    // column sums of dlogits over this CTA's tokens: warps fold in one after the other (fixed order)
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int w = 0; w < nwarps; ++w) {
      if (warp == w) {
#pragma unroll
        for (int r = 0; r < ER; ++r) {
          const int e = lane + r * kWarp;
          if (e < E) s_bias[e] = (w == 0 ? 0.f : s_bias[e]) + bias_acc[r];
        }
      }
      __syncthreads();
    }
    for (int e = threadIdx.x; e < E; e += blockDim.x) bias_partial[(long long)blockIdx.x * E + e] = s_bias[e];
  }
}

// out[c] = sum over parts of partial[part, c]; one CTA per column group, fixed summation order.
__global__ void __launch_bounds__(256) col_sum_reduce_kernel(const float* __restrict__ partial, int n_parts, int n_cols,
                                                             float* __restrict__ out) {
  __shared__ float s_red[256];
  const int c = blockIdx.x;
  float acc = 0.f;
  for (int p = threadIdx.x; p < n_parts; p += blockDim.x) acc += partial[(long long)p * n_cols + c];
  s_red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s_red[threadIdx.x] += s_red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[c] = s_red[0];
}

// ------------------------------------------------------------------------------------------------
// Row tables for a drop-in ragged_dot: rows already sorted by expert, group_sizes given.
__global__ void __launch_bounds__(kRouteThreads) group_tables_kernel(const int32_t* __restrict__ gs, long long M, int E,
                                                           int block, long long mpad, int nbmax,
                                                           int32_t* pad_offsets, int32_t* block_expert,
                                                           int32_t* n_blocks, int32_t* row_of_padded,
                                                           int32_t* padded_of_row) {
  __shared__ int s_cnt[kMaxExperts], s_off[kMaxExperts + 1], s_pad[kMaxExperts + 1], s_tmp[2 * kRouteWarps];
  if (threadIdx.x < E) s_cnt[threadIdx.x] = max(gs[threadIdx.x], 0);
  __syncthreads();
  expert_offsets(s_cnt, E, block, s_off, s_pad, s_tmp, threadIdx.x);
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  if (blockIdx.x == 0) {
    for (int x = threadIdx.x; x <= E; x += blockDim.x) pad_offsets[x] = s_pad[x];
    if (threadIdx.x == 0) n_blocks[0] = s_pad[E] / block;
  }
  const int nb = s_pad[E] / block;
  for (long long b = gtid; b < nbmax; b += gstride) {
    int val = -1;
    if (b < nb) {
      int row = (int)b * block, lo = 0, hi = E;
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_pad[mid] <= row) lo = mid; else hi = mid;
      }
      val = lo;
    }
    block_expert[b] = val;
  }
  for (long long r = gtid; r < mpad; r += gstride) {
    int val = -1;
    if (r < s_pad[E]) {
      int lo = 0, hi = E;
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_pad[mid] <= r) lo = mid; else hi = mid;
      }
      int local = (int)r - s_pad[lo];
      int cnt = s_off[lo + 1] - s_off[lo];
      if (local < cnt) val = s_off[lo] + local;
    }
    row_of_padded[r] = val;
  }
  for (long long m = gtid; m < M; m += gstride) {
    int val = -1;
    if (m < s_off[E]) {
      int lo = 0, hi = E;  // largest x with s_off[x] <= m and non-empty group containing m
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_off[mid] <= m) lo = mid; else hi = mid;
      }
      val = s_pad[lo] + ((int)m - s_off[lo]);
    }
    padded_of_row[m] = val;
  }
}

// offsets[e] = sum of the sizes of the groups before e (negative sizes count as none), e in [0, E]; sums beyond 2^31 - 1 stay there, so that
// the offsets never fall.
__global__ void __launch_bounds__(kRouteThreads) group_offsets_kernel(const int32_t* __restrict__ gs, int E, int32_t* __restrict__ offsets) {
  __shared__ int s_sum[kRouteWarps];
  static_assert(kMaxExperts <= kRouteThreads, "one expert per thread");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto add = [](int a, int b) { return (int)min((unsigned)a + (unsigned)b, 0x7fffffffu); };
  int run = tid < E ? max(gs[tid], 0) : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run = add(run, up);
  }
  if (lane == 31) s_sum[warp] = run;
  __syncthreads();
  for (int w = 0; w < warp; ++w) run = add(run, s_sum[w]);
  if (tid < E) offsets[tid + 1] = run;
  if (tid == 0) offsets[0] = 0;
}

// f32 -> bf16 (round to nearest even), grid-stride.
__global__ void __launch_bounds__(256) cast_f32_bf16_kernel(const float* __restrict__ src,
                                                            __nv_bfloat16* __restrict__ dst, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}

// f32 -> three bf16 pieces with hi + mid + lo == w to 24 mantissa bits; dst is [3][n].  `rounded` (optional, [n])
// receives hi alone: the weight rounded to bf16.
__global__ void __launch_bounds__(256) split3_bf16_kernel(const float* __restrict__ src,
                                                          __nv_bfloat16* __restrict__ dst,
                                                          __nv_bfloat16* __restrict__ rounded, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float w = src[i];
    const __nv_bfloat16 hi = __float2bfloat16_rn(w);
    const float r1 = w - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(mid);
    dst[i] = hi;
    if (rounded != nullptr) rounded[i] = hi;
    dst[n + i] = mid;
    dst[2 * n + i] = __float2bfloat16_rn(r2);
  }
}

// ------------------------------------------------------------------------------------------------ host

// Slots per chunk: one chunk per SM (see route_rank_kernel), or as few per SM as fit in shared memory, the same number on each (five
// million slots in chunks of 32,768 are one chunk per SM and five more: over 16 experts 127 us, so 70); whole tokens when fed logits
// (k slots each).
inline int route_chunk_slots(long long M, int k, bool tokens) {
  const long long unit = tokens ? (long long)k * kRouteWarps : 256;   // tokens: whole rounds of the CTA's 16 warps
  const long long most = kMaxChunkSlots / unit * unit;
  const long long per_sm = (M + num_sms() - 1) / num_sms(), rounds = (per_sm + most - 1) / most;
  const long long per = rounds > 1 ? (M + num_sms() * rounds - 1) / (num_sms() * rounds) : per_sm;
  long long s = (per + unit - 1) / unit * unit;
  if (s > most) s = most;
  if (s < unit) s = unit;
  if (tokens && s < kMinChunkSlots) s = (kMinChunkSlots + k - 1) / k * k;
  return (int)s;
}

// Raises the kernel's limit on dynamic shared memory, once per device and whatever the first size is: the 48 KB that need no such
// call are for dynamic and static memory together, and these kernels have 8 to 10 KB of the latter.
template <class Kern>
inline bool route_smem_ok(Kern kern, size_t smem, bool (&done)[64]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (done[dev]) return smem <= 200 * 1024;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  done[dev] = true;
  return smem <= 200 * 1024;
}

template <int ER>
inline int launch_route_chunk(cudaStream_t st, const RouteChunkArgs& a, int n_chunks, bool early) {
  static bool done[64] = {false};
  const size_t smem = ((size_t)a.chunk_slots + (size_t)(kRouteWarps + 1) * a.E) * 4;
  if (!route_smem_ok(route_chunk_kernel<ER>, smem, done)) return LEWI_ERR_LIMIT;
  (void)launch_kernel(route_chunk_kernel<ER>, n_chunks, kRouteThreads, smem, st, early, a);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

template <int ER>
inline int launch_route_fused(cudaStream_t st, const RouteFusedArgs& a, bool early) {
  static bool done[64] = {false};
  const size_t smem = ((size_t)a.t.num_slots + 4 + (size_t)kRouteWarps * a.t.E) * 4;
  if (!route_smem_ok(route_fused_kernel<ER>, smem, done)) return LEWI_ERR_LIMIT;
  (void)launch_kernel(route_fused_kernel<ER>, 1, kRouteThreads, smem, st, early, a);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

inline int route_common(cudaStream_t st, const float* logits, const int32_t* flat_in, long long T, long long M,
                        int E, int k, int block, int32_t* topk_idx, float* topk_w, int32_t* counts,
                        int32_t* offsets, int32_t* pad_offsets, int32_t* block_expert, int32_t* n_blocks,
                        int32_t* order, int32_t* pos, int32_t* pad_pos, int32_t* row_slot, float* probs_sum,
                        void* ws, long long ws_bytes, float* aux_loss = nullptr, bool early = false) {
  if (E <= 0 || E > kMaxExperts) return LEWI_ERR_LIMIT;
  if (M > 0x7fffffffLL) return LEWI_ERR_LIMIT;
  const bool padded = block > 0 && pad_offsets != nullptr;
  const long long mpad = padded ? (M + (long long)E * (block - 1)) / block * block : 0;
  RouteTables t;
  t.counts = counts;
  t.offsets = offsets;
  t.pad_offsets = padded ? pad_offsets : nullptr;
  t.block_expert = padded ? block_expert : nullptr;
  t.n_blocks = padded ? n_blocks : nullptr;
  t.probs_sum = probs_sum;
  t.aux_loss = (logits && probs_sum) ? aux_loss : nullptr;
  t.order = order;
  t.pos = pos;
  t.pad_pos = padded ? pad_pos : nullptr;
  t.row_slot = padded ? row_slot : nullptr;
  t.num_slots = M;
  t.num_tokens = T;
  t.E = E;
  t.block = padded ? block : 0;
  t.nbmax = padded ? (int)(mpad / block) : 0;
#define LEWI_ROUTE_ER(call)                  \
  do {                                       \
    int rc_;                                 \
    if (E <= 64) { constexpr int ER = 2; rc_ = call; }        \
    else if (E <= 128) { constexpr int ER = 4; rc_ = call; }  \
    else if (E <= 256) { constexpr int ER = 8; rc_ = call; }  \
    else { constexpr int ER = 16; rc_ = call; }               \
    if (rc_ != LEWI_OK) return rc_;          \
  } while (0)
  const int chunk_slots = route_chunk_slots(M, k, logits != nullptr);
  const int n_chunks = (int)((M + chunk_slots - 1) / chunk_slots);
  const bool scanned = n_chunks > kScanChunks;
  const long long hist_rows = n_chunks + (scanned ? 1 : 0), need = (hist_rows + n_chunks) * E * 4;
  if (ws == nullptr || ws_bytes < need) return LEWI_ERR_WORKSPACE;   // also where the one-CTA path would not touch it
  if (logits != nullptr && route_fused(T, E, n_chunks)) {
    const RouteFusedArgs fa{t, logits, topk_idx, topk_w, mpad, k};
    LEWI_ROUTE_ER(launch_route_fused<ER>(st, fa, early));
    return LEWI_OK;
  }
  int32_t* chunk_hist = reinterpret_cast<int32_t*>(ws);
  float* chunk_probs = reinterpret_cast<float*>(chunk_hist + hist_rows * E);
  RouteChunkArgs ca;
  ca.logits = logits;
  ca.flat_in = flat_in;
  ca.topk_idx = topk_idx;
  ca.topk_w = topk_w;
  ca.chunk_hist = chunk_hist;
  ca.chunk_probs = (logits && probs_sum) ? chunk_probs : nullptr;
  ca.row_slot = padded ? row_slot : nullptr;
  ca.num_slots = M;
  ca.mpad = mpad;
  ca.E = E;
  ca.k = k;
  ca.chunk_slots = chunk_slots;
  if (n_chunks > 0) {
    if (logits) {
      LEWI_ROUTE_ER(launch_route_chunk<ER>(st, ca, n_chunks, early));
    } else if (int rc = launch_route_chunk<1>(st, ca, n_chunks, early)) {
      return rc;
    }
  } else if (padded && row_slot != nullptr && mpad > 0) {
    cudaMemsetAsync(row_slot, 0xff, (size_t)mpad * 4, st);
  }
#undef LEWI_ROUTE_ER
  if (scanned) {
    route_scan_kernel<<<(E + kWarp - 1) / kWarp, kScanThreads, 0, st>>>(chunk_hist, n_chunks, E);
    LEWI_CHECK_LAUNCH();
  }
  const RouteRankArgs ra{t, logits ? topk_idx : flat_in, chunk_hist, ca.chunk_probs, n_chunks, chunk_slots, scanned};
  static bool done[64] = {false};
  // s_run [kRouteWarps][E] also holds one partial probability sum per thread
  const size_t smem = ((size_t)chunk_slots + (size_t)(kRouteWarps * E > kRouteThreads ? kRouteWarps * E : kRouteThreads)) * 4;
  if (!route_smem_ok(route_rank_kernel, smem, done)) return LEWI_ERR_LIMIT;
  (void)launch_kernel(route_rank_kernel, n_chunks > 0 ? n_chunks : 1, kRouteThreads, smem, st, early && !scanned && n_chunks > 0, ra);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

}  // namespace lewi
