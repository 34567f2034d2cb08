// Label search on a corridor's local graph (corridor.cuh), by one CTA.
//
// Labels are processed in waves of increasing p = pa * d + pb * delay, a
// Dijkstra order on the combined weight.  A label that dominates another has
// no larger p, so with narrow waves a label is final when its wave comes and
// nothing that was kept is ever killed; a label that a later one of the same
// wave dominates is merely superfluous.  Inside a corridor every label at v
// has p within [F(v), F(v) + T - F(sink)], a range of a few arcs, so a wave
// holds labels of few vertices, many of each.
//
// A wave is processed in batches of one candidate a thread:
//   1. candidates are sorted by (vertex, d, delay), one 64-bit key, in
//      registers (shared memory for strides past a warp);
//   2. one is dropped when an earlier one of its vertex has no larger delay
//      (a segmented prefix minimum), or when a kept run of its vertex does
//      (binary search: a batch's kept labels of one vertex lie side by side in
//      the arena, d rising and delay falling);
//   3. the kept ones get consecutive arena slots, become a run of their
//      vertex and are expanded at once; children that pass the bounds join
//      this wave or the far pile.
// There are no locks and no per-label chains.  A batch of up to 32 candidates
// is processed by warp 0 alone without block barriers, as most waves of an
// ordinary query are.  Bound by latency: the measured cost is about 0.5 us a
// narrow wave and 4-6 us a batch of 512.
#pragma once

#include "corridor.cuh"

namespace vine {

constexpr int kWaveGroup = 16;  // waves between two decisions of the bucket policy (a
                                // multiple of 4)


// Everything a wave search reads (the arrays are the worker's).
struct WaveSearch {
  const int4 *line;
  const int32_t *col;
  const float2 *w;
  uint4 *state;        // per vertex: delay, length, combined distance to the sink; Pareto mode:
                       // least delay kept in finished waves (see known_better)
  int n, sink;
  uint32_t *sinks;       // Pareto mode: arena slots of the sink's kept labels
  int sink_cap;
  uint2 *seen;           // Pareto mode, per vertex: wave of its runs, their least delay
  uint32_t B, a, b, bB;  // budget, pruning multiplier, b * B
  uint32_t pa, pb;       // order
  Label *pool;
  uint32_t *next;        // run links: see run_dominates
  uint32_t *head;        // [n] newest run of a vertex (kNone = none)
  // candidates: shared part, then the worker's global memory
  unsigned long long *nkey[2], *fkey[2];
  uint32_t *npar[2], *fpar[2], *fp[2];
  int nb, fb;
  uint4 *novf[2], *fovf[2];
  uint32_t novf_cap, fovf_cap;
};

struct __align__(16) SearchShared {
  WaveSearch s;            // what the search reads (see WaveShared::c on why it lies here)
  unsigned long long inc;  // incumbent (cost, delay)
  unsigned long long xk[512];
  uint32_t xp[512];
  unsigned long long tail[16];  // per warp: vertex and least delay of its last segment
  uint32_t tail_first[16];      // per warp: vertex of its first element
  uint32_t inc_parent;
  uint32_t nn[2], nf[2];  // candidates of this / the next round, far pile
  uint32_t far_min, hi;
  uint32_t done;          // candidates of this round already processed
  uint32_t taken;         // arena slot the batch's first kept label gets
  int cur, stop, overflow;
  int scan[kScanScratch];
};
constexpr size_t kSearchBytes = (sizeof(SearchShared) + 15) & ~(size_t)15;

// A candidate label: key = vertex << 48 | d << 24 | delay, its parent's arena
// index and, in the far pile, its p.
__device__ __forceinline__ unsigned long long label_key(uint32_t v, uint32_t d, uint32_t dl) {
  return (unsigned long long)v << 48 | (unsigned long long)d << 24 | dl;
}
__device__ __forceinline__ uint32_t key_vertex(unsigned long long k) { return (uint32_t)(k >> 48); }
__device__ __forceinline__ uint32_t key_cost(unsigned long long k) { return (uint32_t)(k >> 24) & 0xffffffu; }
__device__ __forceinline__ uint32_t key_delay(unsigned long long k) { return (uint32_t)k & 0xffffffu; }

// True when the bounds rule (v, d, dl) out.
__device__ __forceinline__ bool label_beyond(const WaveSearch &S, const uint4 &h, uint32_t d, uint32_t dl,
                                             unsigned long long inc) {
  if (h.y == kNoKey) return true;  // no way to the sink inside the corridor
  const uint32_t lb = dl + h.x;    // all terms are below 2^24
  if (lb > S.B) return true;
  const unsigned long long f = (unsigned long long)(d + h.y) << 32 | lb;
  if (f >= inc) return true;
  // d <= UB and dl <= B here: the sum stays below 2^32 (corridor.cuh)
  return S.a != 0u && S.a * d + S.b * dl + h.z > S.a * (uint32_t)(inc >> 32) + S.bB;
}

// True when a kept label of v has no larger d and no larger delay.  A run is
// named by its first arena slot i, with the top bit set when it has one
// label; next[i] is v's previous run, next[i + 1] the length of a longer one.
// (Plain loads: runs are written once, by this SM, and the candidates of a
// vertex probe the same few lines, so L1 serves most of them.  Read past L1
// they took half of a Pareto query's time.)
__device__ __forceinline__ bool run_dominates(const WaveSearch &S, uint32_t run, uint32_t d, uint32_t dl) {
  while (run != kNone) {
    const uint32_t i = run & 0x7fffffffu;
    int len = 1;
    const uint32_t before = S.next[i];
    if (!(run & 0x80000000u)) len = (int)S.next[i + 1];
    int lo = 0, hi = len;  // labels [0, lo) have d no larger
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((uint32_t)S.pool[i + mid].d <= d) lo = mid + 1;
      else hi = mid;
    }
    if (lo > 0 && (uint32_t)S.pool[i + lo - 1].dl <= dl) return true;
    run = before;
  }
  return false;
}

// True when a label kept before rules the candidate (v, d, dl) out; h: v's state.
//
// Pareto sets are searched in order of d alone.  What finished waves kept at v
// then has a smaller d than any candidate, so one number a vertex, the least delay among
// it, stands for all of it, and a vertex's runs are those of the wave in
// progress.  (In the order of the optimal mode runs had to be kept for good:
// a vertex of a loose 60 x 60 grid query has some 200 labels in as many runs, which
// every candidate walked: 8 queries 66 ms, in this order 14.6 ms.)  The first
// run that a vertex gets in a wave folds the older ones into h.w; until then
// `seen` holds their least delay.
template <bool kPareto>
__device__ __forceinline__ bool known_better(const WaveSearch &S, uint32_t v, const uint4 &h, uint32_t d, uint32_t dl,
                                             uint32_t wave) {
  if (kPareto) {
    if (dl >= h.w) return true;
    const uint2 s = S.seen[v];
    if (s.x != wave) return dl >= s.y;
  }
  return run_dominates(S, S.head[v], d, dl);
}

// Adds the run of `len` labels from arena slot idx on, the least delay among
// them `least`, to v (one thread a vertex).
template <bool kPareto>
__device__ __forceinline__ void add_run(const WaveSearch &S, uint32_t v, uint32_t idx, uint32_t len, uint32_t least,
                                        uint32_t wave) {
  uint32_t before = S.head[v];
  if (kPareto) {
    uint2 s = S.seen[v];
    if (s.x != wave) {
      // (other threads may read the word meanwhile: both values hold)
      S.state[v].w = min(S.state[v].w, s.y);
      s = make_uint2(wave, kNoKey);
      before = kNone;
    }
    s.y = min(s.y, least);
    S.seen[v] = s;
  }
  S.next[idx] = before;
  if (len > 1) S.next[idx + 1] = len;
  S.head[v] = len > 1 ? idx : idx | 0x80000000u;
}

__device__ __forceinline__ void near_get(const WaveSearch &S, int cur, uint32_t i, unsigned long long *k,
                                         uint32_t *par) {
  if (i < (uint32_t)S.nb) {
    *k = S.nkey[cur][i];
    *par = S.npar[cur][i];
  } else {
    const uint4 x = __ldcg(&S.novf[cur][i - S.nb]);
    *k = (unsigned long long)x.y << 32 | x.x;
    *par = x.z;
  }
}

__device__ __forceinline__ void near_put(SearchShared &Q, const WaveSearch &S, int b, uint32_t i,
                                         unsigned long long k, uint32_t par) {
  if (i < (uint32_t)S.nb) {
    S.nkey[b][i] = k;
    S.npar[b][i] = par;
  } else if (i - S.nb < S.novf_cap) {
    __stcg(&S.novf[b][i - S.nb], make_uint4((uint32_t)k, (uint32_t)(k >> 32), par, 0u));
  } else {
    Q.overflow = 1;
  }
}

__device__ __forceinline__ void far_put(SearchShared &Q, const WaveSearch &S, int b, uint32_t i,
                                        unsigned long long k, uint32_t par, uint32_t p) {
  if (i < (uint32_t)S.fb) {
    S.fkey[b][i] = k;
    S.fpar[b][i] = par;
    S.fp[b][i] = p;
  } else if (i - S.fb < S.fovf_cap) {
    __stcg(&S.fovf[b][i - S.fb], make_uint4((uint32_t)k, (uint32_t)(k >> 32), par, p));
  } else {
    Q.overflow = 2;
  }
}

// Files a warp's children: bit k of near / far (all lanes call).
template <int K>
__device__ __forceinline__ void label_emit(SearchShared &Q, const WaveSearch &S, int nxt, int fbuf,
                                           const unsigned long long (&key)[K], const uint32_t (&p)[K],
                                           uint32_t par, uint32_t near, uint32_t far) {
  const unsigned FULL = 0xffffffffu;
  uint32_t pos[K];
  if (__any_sync(FULL, near)) {
    warp_slots<K>(&Q.nn[nxt], near, pos);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (near >> k & 1u) near_put(Q, S, nxt, pos[k], key[k], par);
  }
  if (__any_sync(FULL, far)) {
    warp_slots<K>(&Q.nf[fbuf], far, pos);
    uint32_t least = kNoKey;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (far >> k & 1u) {
        far_put(Q, S, fbuf, pos[k], key[k], par, p[k]);
        least = min(least, p[k]);
      }
    least = __reduce_min_sync(FULL, least);
    if ((threadIdx.x & 31) == 0) atomicMin(&Q.far_min, least);
  }
}

// Expands the kept labels of a warp, one a lane (all lanes call): arena slot
// idx, key k.  *best / *best_par: the best sink label this lane has seen.
template <bool kPareto>
__device__ __forceinline__ uint32_t expand_kept(SearchShared &Q, const WaveSearch &S, bool kept,
                                                unsigned long long k, uint32_t idx, int nxt, int fbuf,
                                                unsigned long long *best, uint32_t *best_par) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t hi = vol(Q.hi);
  int beg = 0, deg = 0;
  const uint32_t d = key_cost(k), dl = key_delay(k);
  ArcLine line;
  if (kept) {
    line = load_line(S.line, (int)key_vertex(k));
    deg = line.a[0].w;
    beg = line.a[1].w;
  }
  auto go = [&](uint32_t on, const int (&u)[kArcBatch], const int2 (&w)[kArcBatch], uint32_t d0, uint32_t dl0,
                uint32_t par) {
    unsigned long long key[kArcBatch];
    uint32_t p[kArcBatch], near = 0, far = 0;
    uint4 h[kArcBatch];
#pragma unroll
    for (int j = 0; j < kArcBatch; ++j)
      if (on >> j & 1u) h[j] = S.state[u[j]];
#pragma unroll
    for (int j = 0; j < kArcBatch; ++j)
      if (on >> j & 1u) {
        const uint32_t nd = d0 + (uint32_t)w[j].x, nl = dl0 + (uint32_t)w[j].y;
        const unsigned long long inc = vol(Q.inc);
        // (a single arc may be as long as 2^24: sums stay below 2^25)
        if (label_beyond(S, h[j], nd, nl, inc)) continue;
        if (kPareto && nl >= h[j].w) continue;  // a finished wave kept a better one
        if (!kPareto && u[j] == S.sink) {
          const unsigned long long c = (unsigned long long)nd << 32 | nl;
          if (c < *best && c < inc) {
            atomicMin(&Q.inc, c);
            *best = c;
            *best_par = par;
          }
          continue;
        }
        key[j] = label_key((uint32_t)u[j], nd, nl);
        p[j] = S.pa * nd + S.pb * nl;
        if (p[j] < hi) near |= 1u << j;
        else far |= 1u << j;
      }
    label_emit<kArcBatch>(Q, S, nxt, fbuf, key, p, par, near, far);
  };
  int u[kArcBatch];
  int2 w[kArcBatch];
  uint32_t on = 0;
#pragma unroll
  for (int j = 0; j < kArcBatch; ++j)
    if (j < deg) {
      u[j] = line.a[j].x;
      w[j] = make_int2(line.a[j].y, line.a[j].z);
      on |= 1u << j;
    }
  go(on, u, w, d, dl, idx);
  unsigned wide = __ballot_sync(FULL, deg > kArcBatch);
  for (; wide; wide &= wide - 1) {  // the further arcs of one label after the other
    const int l = __ffs(wide) - 1;
    const int b0 = __shfl_sync(FULL, beg, l) + kArcBatch, e0 = b0 - kArcBatch + __shfl_sync(FULL, deg, l);
    const uint32_t od = __shfl_sync(FULL, d, l), ol = __shfl_sync(FULL, dl, l), oi = __shfl_sync(FULL, idx, l);
    for (int j0 = b0; j0 < e0; j0 += 32 * kArcBatch) {
      on = 0;
#pragma unroll
      for (int j = 0; j < kArcBatch; ++j) {
        const int e = j0 + 32 * j + lane;
        if (e < e0) {
          const float2 x = S.w[e];
          u[j] = S.col[e];
          w[j] = make_int2((int)x.x, (int)x.y);
          on |= 1u << j;
        }
      }
      go(on, u, w, od, ol, oi);
    }
  }
  return (uint32_t)deg;
}

// One compare-exchange of a bitonic network within a warp.
__device__ __forceinline__ void sort_step(unsigned long long &k, uint32_t &par, int lane, int stride, bool up) {
  const unsigned long long ok = __shfl_xor_sync(0xffffffffu, k, stride);
  const uint32_t op = __shfl_xor_sync(0xffffffffu, par, stride);
  const bool lower = (lane & stride) == 0;
  if ((ok < k) == (lower == up) && ok != k) {
    k = ok;
    par = op;
  }
}

// Exclusive least delay of the elements before this one with its vertex
// (0xffffffff: none) within the warp; *incl: including this one.
__device__ __forceinline__ uint32_t segment_min(uint32_t v, uint32_t dl, uint32_t *incl) {
  const int lane = threadIdx.x & 31;
  uint32_t m = dl;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t ov = __shfl_up_sync(0xffffffffu, v, o), om = __shfl_up_sync(0xffffffffu, m, o);
    if (lane >= o && ov == v) m = min(m, om);  // sorted: equal vertices are side by side
  }
  *incl = m;
  const uint32_t pv = __shfl_up_sync(0xffffffffu, v, 1), pm = __shfl_up_sync(0xffffffffu, m, 1);
  return lane > 0 && pv == v ? pm : 0xffffffffu;
}

// Pareto mode: a kept label of the sink is listed and not expanded.
template <bool kPareto>
__device__ __forceinline__ bool list_sink(QueryState &st, const WaveSearch &S, bool kept, uint32_t v, uint32_t idx) {
  if (!kPareto || !kept || v != (uint32_t)S.sink) return false;
  const uint32_t k = atomicAdd(&st.sink_n, 1u);
  if (k < (uint32_t)S.sink_cap) S.sinks[k] = idx;
  else fail_query(st, VINE_ERR_CAPACITY, kSiteSink);
  return true;
}

struct RunCounters {
  uint32_t kept, dominated, relaxed;
};

// A batch of n <= 32 candidates [i0, i0 + n) by the calling warp alone.
template <bool kPareto>
__device__ __forceinline__ void batch_warp(const SearchParams &P, QueryState &st, SearchShared &Q,
                                           const WaveSearch &S, int cur, int fbuf, uint32_t i0, uint32_t n,
                                           uint32_t wave, RunCounters &C) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned long long k = kUnset;
  uint32_t par = 0;
  if ((uint32_t)lane < n) {
    near_get(S, cur, i0 + (uint32_t)lane, &k, &par);
    const uint32_t v = key_vertex(k);
    const uint4 h = S.state[v];
    if (label_beyond(S, h, key_cost(k), key_delay(k), vol(Q.inc))) {
      k = kUnset;
    } else if (known_better<kPareto>(S, v, h, key_cost(k), key_delay(k), wave)) {
      k = kUnset;
      C.dominated++;
    }
  }
  const unsigned live = __ballot_sync(FULL, k != kUnset);
  if (live == 0) return;
  if (live & (live - 1)) {
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
      for (int stride = size >> 1; stride >= 1; stride >>= 1)
        sort_step(k, par, lane, stride, (lane & size) == 0 || size == 32);
  } else if (live != 1u) {  // a single one goes to lane 0
    const int l = __ffs(live) - 1;
    const unsigned long long k0 = __shfl_sync(FULL, k, l);
    const uint32_t p0 = __shfl_sync(FULL, par, l);
    k = lane == 0 ? k0 : kUnset;
    par = p0;
  }
  const bool in = k != kUnset;
  const uint32_t v = in ? key_vertex(k) : 0xffffffffu;
  uint32_t mi;
  const uint32_t before = segment_min(v, key_delay(k), &mi);
  const bool kept = in && !(before <= key_delay(k));
  C.dominated += in && !kept;
  const unsigned km = __ballot_sync(FULL, kept);
  const uint32_t cnt = (uint32_t)__popc(km);
  if (lane == 0) {
    pool_reserve(P, st, cnt);
    Q.taken = st.chunk_fill;
    if (st.abort) Q.stop = 1;
    else st.chunk_fill += cnt;
  }
  __syncwarp();
  if (vol(*reinterpret_cast<const uint32_t *>(&Q.stop))) return;
  const uint32_t idx = vol(Q.taken) + (uint32_t)__popc(km & ((1u << lane) - 1u));
  if (kept) {
    S.pool[idx] = Label{(int32_t)v, (float)key_cost(k), (float)key_delay(k), (int32_t)par};
    C.kept++;
  }
  // the first kept lane of a vertex writes its run
  const unsigned same = __match_any_sync(FULL, v) & km;
  // along a run delays fall: the last label has the least
  const uint32_t least = kPareto ? __shfl_sync(FULL, key_delay(k), 31 - __clz((int)(same | 1u))) : 0u;
  if (kept && (int)__ffs(same) - 1 == lane) add_run<kPareto>(S, v, idx, (uint32_t)__popc(same), least, wave);
  __syncwarp();
  unsigned long long best = kUnset;
  uint32_t best_par = 0;
  const bool listed = list_sink<kPareto>(st, S, kept, v, idx);
  C.relaxed += expand_kept<kPareto>(Q, S, kept && !listed, k, idx, cur ^ 1, fbuf, &best, &best_par);
  __syncwarp();
  if (best != kUnset && best == vol(Q.inc)) Q.inc_parent = best_par;
  __syncwarp();
}

// Candidates of one batch: the largest power of two of threads.
__device__ __forceinline__ uint32_t batch_size() { return 1u << (31 - __clz((int)blockDim.x)); }

// A batch of n <= batch_size() candidates by the whole block.
template <bool kPareto>
__device__ __forceinline__ void batch_block(const SearchParams &P, QueryState &st, SearchShared &Q,
                                            const WaveSearch &S, int cur, int fbuf, uint32_t i0, uint32_t n,
                                            uint32_t wave, RunCounters &C) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long k = kUnset;
  uint32_t par = 0;
  if ((uint32_t)tid < n) {
    near_get(S, cur, i0 + (uint32_t)tid, &k, &par);
    const uint32_t v = key_vertex(k);
    const uint4 h = S.state[v];
    if (label_beyond(S, h, key_cost(k), key_delay(k), vol(Q.inc))) {
      k = kUnset;
    } else if (known_better<kPareto>(S, v, h, key_cost(k), key_delay(k), wave)) {
      k = kUnset;
      C.dominated++;
    }
  }
  // bitonic sort over the power of two that holds n (rounded up to a warp)
  int size_max = 32;  // at most batch_size(), so partners are threads of the block
  while (size_max < (int)n) size_max <<= 1;
  for (int size = 2; size <= size_max; size <<= 1) {
    const bool up = (tid & size) == 0 || size == size_max;
    int stride = size >> 1;
    for (; stride >= 32; stride >>= 1) {
      __syncthreads();
      Q.xk[tid] = k;
      Q.xp[tid] = par;
      __syncthreads();
      if (tid >= size_max) continue;
      const unsigned long long ok = Q.xk[tid ^ stride];
      const uint32_t op = Q.xp[tid ^ stride];
      const bool lower = (tid & stride) == 0;
      if ((ok < k) == (lower == up) && ok != k) {
        k = ok;
        par = op;
      }
    }
    for (; stride >= 1; stride >>= 1) sort_step(k, par, lane, stride, up);
  }
  const bool in = k != kUnset;
  const uint32_t v = in ? key_vertex(k) : 0xffffffffu;
  uint32_t mi;
  uint32_t before = segment_min(v, key_delay(k), &mi);
  __syncthreads();
  if (lane == 31) Q.tail[warp] = (unsigned long long)v << 32 | mi;
  if (lane == 0) Q.tail_first[warp] = v;
  __syncthreads();
  // a segment that started in earlier warps
  const uint32_t first = Q.tail_first[warp];
  uint32_t carry = 0xffffffffu;
  for (int q = warp - 1; q >= 0 && first != 0xffffffffu; --q) {
    const unsigned long long t = Q.tail[q];
    if ((uint32_t)(t >> 32) != first) break;
    carry = min(carry, (uint32_t)t);
    if (Q.tail_first[q] != first) break;
  }
  if (v == first) before = min(before, carry);
  const bool kept = in && !(before <= key_delay(k));
  C.dominated += in && !kept;
  int total;
  const int rank = block_scan_one(kept ? 1 : 0, Q.scan, &total);
  if (tid == 0) {
    pool_reserve(P, st, (uint32_t)total);
    Q.taken = st.chunk_fill;
    if (st.abort) Q.stop = 1;
    else st.chunk_fill += (uint32_t)total;
  }
  __syncthreads();
  if (Q.stop) return;
  const uint32_t idx = Q.taken + (uint32_t)rank;
  if (kept) {
    S.pool[idx] = Label{(int32_t)v, (float)key_cost(k), (float)key_delay(k), (int32_t)par};
    C.kept++;
  }
  // a vertex's first candidate in the batch is always kept (least d, nothing
  // before it); the last one knows the run's length
  Q.xp[tid] = (uint32_t)rank;
  Q.xk[tid] = (unsigned long long)v;
  __syncthreads();
  if (in) {
    const bool seg_first = tid == 0 || (uint32_t)Q.xk[tid - 1] != v;
    if (seg_first) {
      // length: kept labels up to the next vertex
      int hi = tid + 1;  // galloping, then binary search for the segment's end
      int step = 1;
      const int lim = size_max;
      while (hi < lim && (uint32_t)Q.xk[hi] == v) {
        hi += step;
        step <<= 1;
      }
      int lo = max(tid, hi - step);
      hi = min(hi, lim);
      while (lo + 1 < hi) {  // xk[lo] == v, xk[hi] != v or hi == lim
        const int mid = (lo + hi) >> 1;
        if ((uint32_t)Q.xk[mid] == v) lo = mid;
        else hi = mid;
      }
      const uint32_t end = hi < lim ? Q.xp[hi] : (uint32_t)total;
      const uint32_t len = end - (uint32_t)rank;
      add_run<kPareto>(S, v, idx, len, kPareto ? (uint32_t)S.pool[idx + len - 1].dl : 0u, wave);
    }
  }
  unsigned long long best = kUnset;
  uint32_t best_par = 0;
  const bool listed = list_sink<kPareto>(st, S, kept, v, idx);
  if (warp * 32 < (int)n)
    C.relaxed += expand_kept<kPareto>(Q, S, kept && !listed, k, idx, cur ^ 1, fbuf, &best, &best_par);
  __syncthreads();
  if (best != kUnset && best == vol(Q.inc)) Q.inc_parent = best_par;
  __syncthreads();
}

// Runs the search set up in SearchShared::s (all threads).  On return st.inc_key / st.inc_idx hold the answer.
template <bool kPareto>
static __device__ __noinline__ void wave_search(const SearchParams &P, QueryState &st) {
  extern __shared__ __align__(16) unsigned char smem[];
  SearchShared &Q = *reinterpret_cast<SearchShared *>(smem);
  WaveSearch &S = Q.s;
  const unsigned FULL = 0xffffffffu;
  const int G = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // shared memory behind the state: near and far buffers, then the run heads
  // where they fit
  if (tid == 0) {
    const size_t region = table_region_bytes(P.table_log2, P.lock_log2) - kSearchBytes;
    S.nb = S.fb = region >= 72 * 1024 ? 1024 : region >= 29 * 1024 ? 512 : 128;
    unsigned char *p = smem + kSearchBytes;
    for (int b = 0; b < 2; ++b) {
      S.nkey[b] = reinterpret_cast<unsigned long long *>(p);
      p += S.nb * 8;
      S.fkey[b] = reinterpret_cast<unsigned long long *>(p);
      p += S.fb * 8;
    }
    for (int b = 0; b < 2; ++b) {
      S.npar[b] = reinterpret_cast<uint32_t *>(p);
      p += S.nb * 4;
      S.fpar[b] = reinterpret_cast<uint32_t *>(p);
      p += S.fb * 4;
      S.fp[b] = reinterpret_cast<uint32_t *>(p);
      p += S.fb * 4;
    }
    if ((size_t)(p - smem) + (size_t)S.n * 4 <= kSearchBytes + region) S.head = reinterpret_cast<uint32_t *>(p);
  }
  __syncthreads();
  for (int i = tid; i < S.n; i += G) {
    S.head[i] = kNone;
    if (kPareto) S.seen[i] = make_uint2(kNone, kNoKey);
  }
  // wave width: the policy's bucket width, from cost units to p units (the
  // p of a mean arc for a mean length)
  const float unit = ((float)S.pa * P.mean_len + (float)S.pb * P.mean_delay) / fmaxf(P.mean_len, 1e-3f);
  auto width_of = [&](float w) { return (uint32_t)fminf(fmaxf(w * unit, 1.0f), 536870912.0f); };
  if (tid == 0) {
    Q.inc = (unsigned long long)(uint32_t)key_d(st.inc_key) << 32 | 0xffffffffu;
    Q.inc_parent = kNone;
    Q.nn[0] = 1;
    Q.nn[1] = 0;
    Q.nf[0] = Q.nf[1] = 0;
    Q.far_min = kNoKey;
    Q.hi = width_of(st.width);
    Q.stop = Q.overflow = 0;
    S.nkey[0][0] = label_key((uint32_t)st.src, 0u, 0u);
    S.npar[0][0] = 0xffffffffu;
    st.far_n = 0;
    st.b_labels = st.b_expanded = st.b_rounds = st.b_dominated = 0;
    st.b_candidates = st.b_spilled = st.b_relaxed = 0;
  }
  RunCounters C{0u, 0u, 0u};
  int cur = 0, fbuf = 0;
  uint32_t waves = 0, turn = 0;
  for (;;) {
    __syncthreads();
    const uint32_t nc = min(Q.nn[cur], (uint32_t)S.nb + S.novf_cap);
    if (Q.stop) break;  // changes only between the barriers below, or with the whole block
    if (nc == 0) {
      // ---- the wave is done: the next one starts at the least p left
      const uint32_t fm = Q.far_min, fn = min(Q.nf[fbuf], (uint32_t)S.fb + S.fovf_cap);
      if (fm == kNoKey) break;
      __syncthreads();
      ++waves;
      const bool decide = waves % kWaveGroup == 0;
      if (decide) {  // counters of the group, for the policy and the statistics
        const uint32_t kept = __reduce_add_sync(FULL, C.kept), dom = __reduce_add_sync(FULL, C.dominated),
                       rel = __reduce_add_sync(FULL, C.relaxed);
        C = RunCounters{0u, 0u, 0u};
        if (lane == 0) {
          atomicAdd(&st.b_labels, kept);
          atomicAdd(&st.b_expanded, kept);
          atomicAdd(&st.b_dominated, dom);
          atomicAdd(&st.b_candidates, kept + dom);
          atomicAdd(&st.b_relaxed, rel);
        }
        __syncthreads();
      }
      if (warp == 0) {
        if (decide) {
          if (lane == 0) {
            st.n_expanded += st.b_expanded;
            st.n_inserted += st.b_labels;
            // what the policy sees as one bucket's size is four waves' labels:
            // its target, a quarter of the table, then fills a batch a wave
            st.b_labels /= kWaveGroup / 4;
            st.n_dominated += st.b_dominated;
            st.n_relaxed += st.b_relaxed;
            st.n_buckets++;
            st.far_n = fn;
            st.hi_bits = __float_as_uint((float)Q.hi / unit);
            st.far_min_bits = __float_as_uint((float)fm / unit);
            over_time(P, st);
          }
          __syncwarp();
          const long long t0 = clock64();
          policy_step(P, st);
          if (lane == 0) {
            st.b_labels = st.b_expanded = st.b_rounds = st.b_dominated = 0;
            st.b_candidates = st.b_spilled = st.b_relaxed = 0;
            st.policy_cycles += clock64() - t0;
          }
        }
        if (lane == 0) {
          const uint32_t wd = width_of(st.width);
          Q.hi = min(fm, 0x7fffffffu - wd) + wd;
          Q.far_min = kNoKey;
          Q.nf[fbuf ^ 1] = 0;
          if (Q.overflow || st.abort) Q.stop = 1;
        }
      }
      __syncthreads();
      const uint32_t hi = Q.hi;
      for (uint32_t base = 0; base < fn; base += (uint32_t)G) {
        const uint32_t i = base + (uint32_t)tid;
        if (base + (uint32_t)(warp * 32) >= fn) break;  // whole warps only
        unsigned long long key[1] = {0};
        uint32_t p[1] = {0}, par = 0, near = 0, far = 0;
        if (i < fn) {
          if (i < (uint32_t)S.fb) {
            key[0] = S.fkey[fbuf][i];
            par = S.fpar[fbuf][i];
            p[0] = S.fp[fbuf][i];
          } else {
            const uint4 x = __ldcg(&S.fovf[fbuf][i - S.fb]);
            key[0] = (unsigned long long)x.y << 32 | x.x;
            par = x.z;
            p[0] = x.w;
          }
          if (p[0] < hi) near = 1;
          else far = 1;
        }
        label_emit<1>(Q, S, cur, fbuf ^ 1, key, p, par, near, far);
      }
      fbuf ^= 1;
      continue;
    }
    if (nc <= 32u) {
      __syncthreads();  // every warp has read the count
      if (warp == 0) {
        uint32_t n = nc, run = 0;
        do {
          batch_warp<kPareto>(P, st, Q, S, cur, fbuf, 0, n, waves, C);
          if (lane == 0) {
            Q.nn[cur] = 0;
            st.n_rounds++;
            st.b_rounds++;
          }
          cur ^= 1;
          __syncwarp();
          n = vol(Q.nn[cur]);
        } while (n != 0 && n <= 32u && !vol(*reinterpret_cast<const uint32_t *>(&Q.stop)) && ++run != kNarrowRun);
        if (lane == 0) Q.cur = cur;
      }
    } else {
      for (uint32_t i0 = 0; i0 < nc && !Q.stop; i0 += batch_size()) {
        // (sets st.abort, at which the batch stops the search)
        if (tid == 0 && i0 / batch_size() % kLookAt == kLookAt - 1) look_at_limits(P, st);
        batch_block<kPareto>(P, st, Q, S, cur, fbuf, i0, min(batch_size(), nc - i0), waves, C);
      }
      __syncthreads();
      if (tid == 0) {
        Q.nn[cur] = 0;
        Q.cur = cur ^ 1;
        st.n_rounds++;
        st.b_rounds++;
      }
    }
    if (tid == 0) {
      if (++turn % kLookAt == 0) look_at_limits(P, st);
      if (Q.overflow || st.abort) Q.stop = 1;
    }
    __syncthreads();
    cur = Q.cur;
  }
  __syncthreads();
  const uint32_t kept = __reduce_add_sync(FULL, C.kept), dom = __reduce_add_sync(FULL, C.dominated),
                 rel = __reduce_add_sync(FULL, C.relaxed);
  if (lane == 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&st.n_expanded), (unsigned long long)kept);
    atomicAdd(reinterpret_cast<unsigned long long *>(&st.n_inserted), (unsigned long long)kept);
    atomicAdd(reinterpret_cast<unsigned long long *>(&st.n_dominated), (unsigned long long)dom);
    atomicAdd(reinterpret_cast<unsigned long long *>(&st.n_relaxed), (unsigned long long)rel);
  }
  if (tid == 0) {
    st.n_buckets++;
    if (Q.overflow && !st.abort) fail_query(st, VINE_ERR_CAPACITY, Q.overflow == 1 ? kSiteNear : kSiteBand);
    st.inc_idx = 0xffffffffu;
    if (kPareto) st.inc_key = ~0ull;  // the cost bound is no answer
    if (!st.abort && Q.inc_parent != kNone) {
      pool_reserve(P, st, 1);
      if (!st.abort) {
        const uint32_t idx = st.chunk_fill++;
        const uint32_t cost = (uint32_t)(Q.inc >> 32), dl = (uint32_t)Q.inc;
        S.pool[idx] = Label{S.sink, (float)cost, (float)dl, (int32_t)Q.inc_parent};
        st.inc_idx = idx;
        st.inc_key = pack_key((float)cost, (float)dl);
      }
    }
    st.done = 1;
  }
  __syncthreads();
}

}  // namespace vine
