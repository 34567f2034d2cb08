// Corridor of a query: the part of the graph that can still hold its answer.
//
// A query asks for the cheapest path with delay <= B.  For a multiplier
// lambda = b / a the combined weight a * len + b * delay gives every feasible
// path p (delay(p) <= B) the bound a * cost(p) + b * delay(p) <=
// a * cost(p) + b * B, so with any feasible path of cost UB in hand
//
//     T = a * UB + b * B
//
// only vertices v with F(v) + H(v) <= T matter, F / H being the combined
// distances source -> v and v -> sink (Lagrangian relaxation of the budget;
// Handler and Zang, "A dual algorithm for the constrained shortest path
// problem", Networks 10, 1980).  The same bound prunes single labels during
// the search: a * d + b * delay + H(v) > T.  Equal cost never prunes, so the
// (cost, delay) answer is untouched.
//
// Everything here is integer arithmetic: weights are integers below 2^24,
// keys are kept below 2^31 by the choice of (a, b), and a key that would pass
// that limit is larger than any T, hence prunable.
//
// Per query, by one CTA:
//   1. bi_run: both ends grow at once in the combined weight until their
//      radii cover the best meeting key (the two-sided Dijkstra test), every
//      vertex touched from both ends offering a real path (its delay is
//      carried beside the key) as UB; then on under F + H <= T.  That touches
//      two half-radius balls instead of the full balls around the sink that
//      two reverse searches over the graph need.
//   2. the vertices with F + H <= T are copied out with the arcs between
//      them, renumbered, into a small CSR of the worker (build_local); while
//      it is large, a better multiplier shrinks it again the same way.
//   3. on that CSR: delay and length distances to the sink and the
//      multiplier that maximises the lower bound (a few one-sided passes).
// The label search then runs on the small CSR with all three bounds.
#pragma once

#include "search.cuh"

namespace vine {

constexpr unsigned long long kUnset = ~0ull;
constexpr uint32_t kKeyMax = 0x7ffffffeu;      // largest path key that is kept
constexpr uint32_t kNoKey = 0xffffffffu;
constexpr uint32_t kMemberTag = 0xfffffffeu;   // rf[v].y high word: v has a local id
constexpr float kIntLimit = 16777216.0f;       // 2^24: budgets and costs handled here
constexpr int kWaveQ = 2048;                   // queue entries kept in shared memory
constexpr int kCorridorVertices = 1 << 16;     // largest local graph
constexpr double kFirstLambda = 0.5;           // first multiplier, in mean lengths per mean delay
constexpr double kWideGap = 0.3;               // (T - meeting key) / meeting key worth another multiplier
// A bucket of the two-sided search is no wider than half of what the budget
// suggests of a path (two arcs at least): wider ones flood a graph of small
// diameter before the sides can meet.  64 queries on a random graph of 50,000
// vertices and three arcs each, budget of 3 / 8 mean arcs: 24 arcs wide 4.8 / 10.3 ms,
// by this rule 1.7 / 2.7 ms (reverse searches 0.5 / 2.3 ms); with a quarter in
// place of the half 1.7 / 1.8 ms.  Road, grid and power-law cases do not change.
constexpr float kBudgetShare = 0.5f;
constexpr int kShrinkTo = 1024;                // local graphs up to this size are not shrunk further
constexpr int kHubs = 32;                      // see WaveShared::hub
constexpr int kHubDegree = 256;
// A vertex's arc line: 64 bytes with its first four arcs as {head, length,
// delay, x}, x = the degree in the first and the index of its first arc in
// (col, w) in the second; heads past the degree are -1.  One read instead of
// row, then heads and weights: a round of a wave search is a chain of
// dependent reads, and this takes one of its four out; road vertices
// seldom have more arcs.
struct ArcLine {
  int4 a[4];
};
__device__ __forceinline__ ArcLine load_line(const int4 *line, int v) {
  ArcLine l;
#pragma unroll
  for (int k = 0; k < 4; ++k) l.a[k] = line[4 * (size_t)v + k];  // (plain: local lines are written here)
  return l;
}

constexpr int kArcBatch = 4;                   // arcs of a vertex whose loads go out together

// A worker's local graph: lines and arcs in both directions (row is not used)
// and the original ids.
struct LocalGraph {
  DevGraph g;
  int32_t *gid;
};

// Where a worker's corridor arrays lie (set up once per kernel).
struct CorridorMem {
  ulonglong2 *rf;      // [n] (F, H) of the global search, all ones when unused
  uint32_t *touch[2];  // [n] vertices first reached by each side
  uint32_t *ovf[2];    // queue entries past kWaveQ
  uint32_t ovf_cap;
  unsigned long long *far[2];
  uint32_t far_cap;
  LocalGraph loc[2];
  int lv, la;          // capacity of a local graph: vertices, arcs
  uint32_t *map;       // [lv] old local id -> new local id
  unsigned long long *dist[4];  // [lv] distances on the local graph
  uint4 *state;        // [lv] delay, length and combined distance to the sink (and see WaveSearch)
};

// Weights of one search.  pure: key = delay, the second value is the length;
// otherwise key = a * len + b * delay and the second value is the delay.
struct Combo {
  uint32_t a, b;
  bool pure;
  uint32_t B;
};

// What a local pass computes: distances from `root` along (row, col, w) under
// c; keys above `limit` are dropped.
struct PassArgs {
  const int4 *line;
  const int32_t *col;
  const float2 *w;
  int n, root;
  uint32_t limit;
  uint32_t delta;
  // whole-graph passes (kWhole): arcs longer than max_len or with less delay
  // than min_delay are left out, every arc adds `hop` to the key, and with
  // target >= 0 nothing farther than that vertex is wanted
  float max_len = INFINITY, min_delay = -INFINITY;
  uint32_t hop = 0;
  int target = -1;
};

// Shared-memory state of the wave searches.  It lies over the bucket table,
// which is not in use before the label search starts.
struct __align__(16) WaveShared {
  uint32_t q[2][kWaveQ];
  unsigned long long mu;    // best meeting: (key, delay), pure mode (delay, length)
  unsigned long long best;  // best feasible: (a * cost + b * B, delay), pure mode (cost, delay)
  uint32_t nq[2], nfar[2], ntouch[2];
  uint32_t far_min, hi, rdone;
  uint32_t cnt;
  int cur;
  CorridorMem m;  // the worker's arrays
  // What the search in progress works on.  Kept here and not passed by value:
  // by-value structs of called functions live in local memory, whose lines
  // the waves' gathers push out of L1 (7.0e6 of 9.8e6 loads of a profile).
  Combo c;
  PassArgs a;
  DevGraph g;
  uint32_t delta;
  int fb;
  uint32_t sides;  // two-sided search: bit s: side s still has vertices to go on from
  uint32_t hub[kHubs], nhub;  // vertices of this round whose arcs the block shares
  // clipped: something was left out because its key, with what the other side
  // needs at least, passes kKeyMax; until a path is known that is no bound, so
  // a search that ends without a meeting has then not shown that there is none
  int clipped, overflow, stop;
  int scan[kScanScratch];
};

// 32-bit words of a worker's two local graphs (heads, ids) and the renumbering.
__host__ __device__ constexpr size_t corridor_ints(int lv, int la) {
  return 2 * (2 * (size_t)la + (size_t)lv) + (size_t)lv;
}

constexpr size_t kWaveBytes = (sizeof(WaveShared) + 15) & ~(size_t)15;

// Shared memory of the bucket table and its locks, or of the wave state that
// lies over them when that needs more.
__host__ __device__ constexpr size_t table_region_bytes(int table_log2, int lock_log2) {
  const size_t t = ((sizeof(int32_t) + sizeof(float2) + sizeof(uint32_t)) << table_log2) +
                   (sizeof(int) << lock_log2);
  return ((t > kWaveBytes ? t : kWaveBytes) + 15) & ~(size_t)15;
}

__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2 *p) {
  ulonglong2 r;
  asm volatile("ld.global.cg.v2.u64 {%0,%1}, [%2];" : "=l"(r.x), "=l"(r.y) : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ uint32_t key_hi(unsigned long long x) { return (uint32_t)(x >> 32); }
__device__ __forceinline__ uint32_t vol(const uint32_t &x) {
  return *reinterpret_cast<const volatile uint32_t *>(&x);
}
__device__ __forceinline__ unsigned long long vol(const unsigned long long &x) {
  return *reinterpret_cast<const volatile unsigned long long *>(&x);
}

// Exclusive prefix sum of one value per thread; *total gets the sum.  All
// threads must call.
__device__ __forceinline__ int block_scan_one(int x, int *scratch, int *total) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = (blockDim.x + 31) >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int v = lane < nw ? scratch[lane] : 0;
    int vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += y;
    }
    if (lane < nw) scratch[lane] = vi - v;
    if (lane == nw - 1) scratch[32] = vi;
  }
  __syncthreads();
  const int r = scratch[warp] + incl - x;
  *total = scratch[32];
  __syncthreads();
  return r;
}

__device__ __forceinline__ uint32_t wave_get(const WaveShared &W, const CorridorMem &M, int cur,
                                             uint32_t i) {
  return i < (uint32_t)kWaveQ ? W.q[cur][i] : __ldcg(&M.ovf[cur][i - kWaveQ]);
}

__device__ __forceinline__ void wave_put(WaveShared &W, const CorridorMem &M, int nxt, uint32_t pos,
                                         uint32_t e) {
  if (pos < (uint32_t)kWaveQ) W.q[nxt][pos] = e;
  else if (pos - kWaveQ < M.ovf_cap) M.ovf[nxt][pos - kWaveQ] = e;
  else W.overflow = 1;
}

__device__ __forceinline__ void wave_push(WaveShared &W, const CorridorMem &M, int nxt, uint32_t e) {
  wave_put(W, M, nxt, warp_agg_inc(&W.nq[nxt]), e);
}

__device__ __forceinline__ void far_push(WaveShared &W, const CorridorMem &M, int fb, uint32_t key,
                                         uint32_t e) {
  const uint32_t pos = warp_agg_inc(&W.nfar[fb]);
  if (pos >= M.far_cap) {
    W.overflow = 1;
    return;
  }
  M.far[fb][pos] = ((unsigned long long)key << 32) | e;
  atomicMin(&W.far_min, key);
}

// Slots of the calling warp's flagged entries (bit k of `bits`) in the list
// behind *ctr: one shared atomic for the warp; pos[k] of a flagged entry.
template <int K>
__device__ __forceinline__ void warp_slots(uint32_t *ctr, uint32_t bits, uint32_t (&pos)[K]) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  uint32_t total = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const unsigned b = __ballot_sync(FULL, bits >> k & 1u);
    pos[k] = total + (uint32_t)__popc(b & below);
    total += (uint32_t)__popc(b);
  }
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(ctr, total);
  base = __shfl_sync(FULL, base, 0);
#pragma unroll
  for (int k = 0; k < K; ++k) pos[k] += base;
}

// Queues what a warp's relaxations improved: entry e[k] with key[k] goes to
// the next round (bit k of near) or to the far pile (bit k of far); vertices first reached (bit k of first) are
// listed for their side (bit 0 of e[k]) when `sides`.  All lanes call.
template <int K>
__device__ __forceinline__ void wave_emit(WaveShared &W, const CorridorMem &M, int nxt, int fb,
                                          const uint32_t (&e)[K], const uint32_t (&key)[K],
                                          uint32_t near, uint32_t far, uint32_t first, bool sides) {
  const unsigned FULL = 0xffffffffu;
  uint32_t pos[K];
  if (__any_sync(FULL, near)) {
    warp_slots<K>(&W.nq[nxt], near, pos);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (near >> k & 1u) wave_put(W, M, nxt, pos[k], e[k]);
  }
  if (__any_sync(FULL, far)) {
    warp_slots<K>(&W.nfar[fb], far, pos);
    uint32_t least = kNoKey;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (far >> k & 1u) {
        if (pos[k] < M.far_cap) M.far[fb][pos[k]] = ((unsigned long long)key[k] << 32) | e[k];
        else W.overflow = 1;
        least = min(least, key[k]);
      }
    least = __reduce_min_sync(FULL, least);
    if ((threadIdx.x & 31) == 0) atomicMin(&W.far_min, least);
  }
  if (sides && __any_sync(FULL, first)) {
    uint32_t f1 = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) f1 |= (first >> k & 1u & e[k]) << k;
    if (__any_sync(FULL, first & ~f1)) {
      warp_slots<K>(&W.ntouch[0], first & ~f1, pos);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if ((first & ~f1) >> k & 1u) M.touch[0][pos[k]] = e[k] >> 1;
    }
    if (__any_sync(FULL, f1)) {
      warp_slots<K>(&W.ntouch[1], f1, pos);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (f1 >> k & 1u) M.touch[1][pos[k]] = e[k] >> 1;
    }
  }
}

// ------------------------------------------------------- two-sided search

__device__ __forceinline__ uint32_t combo_limit(const WaveShared &W, const Combo &k) {
  if (k.pure) return k.B;
  const unsigned long long t = vol(W.best) >> 32;
  return t < kKeyMax ? (uint32_t)t : kKeyMax;
}

// A vertex reached from both ends: (k, s) is a real source -> sink path.
__device__ __forceinline__ void meet(WaveShared &W, const Combo &c, unsigned long long x,
                                     unsigned long long y) {
  const uint32_t k = key_hi(x) + key_hi(y);  // both at most kKeyMax
  const unsigned long long s64 = (x & 0xffffffffull) + (y & 0xffffffffull);
  const uint32_t s = s64 > 0xfffffffeull ? 0xfffffffeu : (uint32_t)s64;
  const unsigned long long m = ((unsigned long long)k << 32) | s;
  if (m < vol(W.mu)) atomicMin(&W.mu, m);
  unsigned long long f = kUnset;
  if (c.pure) {
    if (k <= c.B) f = ((unsigned long long)s << 32) | k;
  } else if (s <= c.B) {
    const unsigned long long t = (unsigned long long)k + (unsigned long long)c.b * (c.B - s);
    if (t <= kKeyMax) f = (t << 32) | s;
  }
  if (f < vol(W.best)) atomicMin(&W.best, f);
}

// Relaxes up to K arcs a lane: vertex u[k], reached with (nk[k], ns[k]) on
// side side[k] (0 from the source, 1 from the sink) where bit k of `on` is set.  The
// pair reads go out together, then the atomics.  All lanes call.
template <int K>
__device__ __forceinline__ void bi_relax(WaveShared &W, const CorridorMem &M,
                                         const Combo &c, uint32_t on, const int (&u)[K],
                                         const unsigned long long (&nk)[K], const uint32_t (&ns)[K],
                                         uint32_t side, uint32_t hi, uint32_t rdone, uint32_t limit,
                                         int nxt, int fb) {
  ulonglong2 pu[K];
  unsigned long long old[K];
  uint32_t e[K], key[K];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (on >> k & 1u) {
      if (nk[k] > limit) {
        if (nk[k] > kKeyMax) W.clipped = 1;
        on &= ~(1u << k);
      } else {
        pu[k] = ld_pair(&M.rf[u[k]]);
      }
    }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (on >> k & 1u) {
      const bool back = side >> k & 1u;
      const unsigned long long cand = (nk[k] << 32) | ns[k];
      const unsigned long long mine = back ? pu[k].y : pu[k].x, other = back ? pu[k].x : pu[k].y;
      // What the other side still needs from u, at least: its own distance
      // where that is final, else the radius up to which it is complete.
      const unsigned long long sum = nk[k] + (unsigned long long)min(key_hi(other), rdone);
      if (cand < mine && sum <= limit) {
        old[k] = atomicMin(reinterpret_cast<unsigned long long *>(&M.rf[u[k]]) + (back ? 1 : 0), cand);
      } else {
        if (cand < mine && sum > kKeyMax) W.clipped = 1;
        on &= ~(1u << k);
      }
    }
  uint32_t near = 0, far = 0, first = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    e[k] = ((uint32_t)u[k] << 1) | (side >> k & 1u);
    key[k] = (uint32_t)nk[k];
    if (on >> k & 1u) {
      const unsigned long long cand = (nk[k] << 32) | ns[k];
      if (cand < old[k]) {
        const unsigned long long other = side >> k & 1u ? pu[k].x : pu[k].y;
        if (other != kUnset) meet(W, c, cand, other);
        if (old[k] == kUnset) first |= 1u << k;
        if (key[k] < hi) near |= 1u << k;
        else far |= 1u << k;
      }
    }
  }
  wave_emit<K>(W, M, nxt, fb, e, key, near, far, first, true);
}

// The second value of a path past an arc, kept below the all-ones word.
__device__ __forceinline__ uint32_t add_second(uint32_t s, uint32_t x) {
  return s > 0xfffffffeu - x ? 0xfffffffeu : s + x;
}

// Clears the pairs that the last search wrote.
__device__ __forceinline__ void bi_reset(WaveShared &W, const CorridorMem &M) {
  __syncthreads();
  for (int s = 0; s < 2; ++s)
    for (uint32_t i = threadIdx.x; i < W.ntouch[s]; i += blockDim.x)
      __stcg(&M.rf[M.touch[s][i]], make_ulonglong2(kUnset, kUnset));
  __syncthreads();
  if (threadIdx.x == 0) W.ntouch[0] = W.ntouch[1] = 0;
  __syncthreads();
}

// One warp's share of a round: entries [i0, i0 + take) of the current queue.
__device__ __forceinline__ uint32_t bi_chunk(const DevGraph &g, WaveShared &W, const CorridorMem &M,
                                             const Combo &c, int cur, int fb, uint32_t i0,
                                             uint32_t take) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, nxt = cur ^ 1;
  const uint32_t hi = vol(W.hi), rdone = vol(W.rdone), limit = combo_limit(W, c);
  int beg = 0, deg = 0;
  uint32_t key = 0, sec = 0, side = 0;
  ArcLine line;
  if ((uint32_t)lane < take) {
    const uint32_t e = wave_get(W, M, cur, i0 + (uint32_t)lane);
    const int v = (int)(e >> 1);
    side = e & 1u;
    const ulonglong2 pv = ld_pair(&M.rf[v]);
    line = load_line(side ? g.rline : g.line, v);
    deg = line.a[0].w;
    beg = line.a[1].w;
    const unsigned long long mine = side ? pv.y : pv.x, other = side ? pv.x : pv.y;
    if (other != kUnset) meet(W, c, mine, other);
    key = key_hi(mine);
    sec = (uint32_t)mine;
    if (deg > kHubDegree) {
      const uint32_t h = atomicAdd(&W.nhub, 1u);
      if (h < (uint32_t)kHubs) {
        W.hub[h] = e;
        deg = 0;
      }
    }
  }
  int u[kArcBatch];
  unsigned long long nk[kArcBatch];
  uint32_t ns[kArcBatch];
  {
    uint32_t on = 0;
#pragma unroll
    for (int k = 0; k < kArcBatch; ++k)
      if (k < deg) {
        const uint32_t ln = (uint32_t)line.a[k].y, dl = (uint32_t)line.a[k].z;
        u[k] = line.a[k].x;
        nk[k] = key + (unsigned long long)c.a * ln + (unsigned long long)c.b * dl;
        ns[k] = add_second(sec, c.pure ? ln : dl);
        on |= 1u << k;
      }
    bi_relax<kArcBatch>(W, M, c, on, u, nk, ns, side ? 0xfu : 0u, hi, rdone, limit, nxt, fb);
  }
  // arcs past the first few, dealt to the lanes of the warp
  const int rem = max(0, deg - kArcBatch);
  if (__any_sync(FULL, rem > 0)) {
    int incl = rem;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(FULL, incl, 31), excl = incl - rem;
    for (int e0 = 0; e0 < total; e0 += 32 * kArcBatch) {
      uint32_t on = 0, sides = 0;
#pragma unroll
      for (int b = 0; b < kArcBatch; ++b) {
        const int e = e0 + 32 * b + lane;
        int k = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
          const int ex = __shfl_sync(FULL, excl, (k + step) & 31);
          if (k + step < 32 && ex <= e) k += step;
        }
        const int obeg = __shfl_sync(FULL, beg, k), oex = __shfl_sync(FULL, excl, k);
        const uint32_t oside = __shfl_sync(FULL, side, k);
        const uint32_t okey = __shfl_sync(FULL, key, k), osec = __shfl_sync(FULL, sec, k);
        if (e < total) {
          const int j = obeg + kArcBatch + (e - oex);
          u[b] = (oside ? g.rcol : g.col)[j];
          const float2 w = (oside ? g.rw : g.w)[j];
          const uint32_t ln = (uint32_t)w.x, dl = (uint32_t)w.y;
          nk[b] = okey + (unsigned long long)c.a * ln + (unsigned long long)c.b * dl;
          ns[b] = add_second(osec, c.pure ? ln : dl);
          on |= 1u << b;
          sides |= oside << b;
        }
      }
      bi_relax<kArcBatch>(W, M, c, on, u, nk, ns, sides, hi, rdone, limit, nxt, fb);
    }
  }
  return (uint32_t)deg;
}

// The arcs of the round's hubs, dealt to the whole block.
__device__ __forceinline__ uint32_t bi_hubs(const DevGraph &g, WaveShared &W, const CorridorMem &M,
                                            const Combo &c, int cur, int fb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t hi = vol(W.hi), rdone = vol(W.rdone), limit = combo_limit(W, c);
  const int nh = (int)min(W.nhub, (uint32_t)kHubs);
  uint32_t relaxed = 0;
  for (int h = 0; h < nh; ++h) {
    const uint32_t e = W.hub[h], side = e & 1u;
    const int v = (int)(e >> 1);
    const ulonglong2 pv = ld_pair(&M.rf[v]);
    const int4 *line = (side ? g.rline : g.line) + 4 * (size_t)v;
    const int32_t *col = side ? g.rcol : g.col;
    const float2 *wt = side ? g.rw : g.w;
    const unsigned long long mine = side ? pv.y : pv.x;
    const uint32_t key = key_hi(mine), sec = (uint32_t)mine;
    const int first = line[1].w, end = first + line[0].w;
    for (int j0 = first + warp * 32 * kArcBatch; j0 < end; j0 += nw * 32 * kArcBatch) {
      int u[kArcBatch];
      unsigned long long nk[kArcBatch];
      uint32_t ns[kArcBatch], on = 0;
#pragma unroll
      for (int k = 0; k < kArcBatch; ++k) {
        const int j = j0 + 32 * k + lane;
        if (j < end) {
          u[k] = col[j];
          const float2 w = wt[j];
          const uint32_t ln = (uint32_t)w.x, dl = (uint32_t)w.y;
          nk[k] = key + (unsigned long long)c.a * ln + (unsigned long long)c.b * dl;
          ns[k] = add_second(sec, c.pure ? ln : dl);
          on |= 1u << k;
        }
      }
      relaxed += (uint32_t)__popc(on);
      bi_relax<kArcBatch>(W, M, c, on, u, nk, ns, side ? 0xfu : 0u, hi, rdone, limit, cur ^ 1, fb);
    }
  }
  return relaxed;
}

// A bucket or a wave may take any number of rounds, so the query's limits are
// looked at between them too: warp 0 leaves a run of narrow rounds (about 1 us
// each) after kNarrowRun, and the block looks at every kLookAt-th turn.  That
// costs 1 to 3 % of a call's cycles (96 road pairs 2,017 -> 2,037 M, 64 queries
// on a power-law graph 1,993 -> 2,037 M), 8 and 512 in place of 32 and 128 as much.
constexpr uint32_t kNarrowRun = 128, kLookAt = 32;
static __device__ __noinline__ void look_at_limits(const SearchParams &P, QueryState &st) {
  if (st.n_rounds > kMaxRounds) fail_query(st, VINE_ERR_TIMEOUT, kSiteRounds);
  over_time(P, st);
}

// Runs rounds until the queue is empty or kLookAt turns are over (all threads).
// Returns arcs relaxed by the calling thread.
//
// Bound by latency: a round is a chain of dependent reads (queue, row and
// pair, arcs, their pairs), one atomic and the push.  A lane takes a whole
// vertex of a road graph (at most kArcBatch arcs, the loads and then the
// atomics of all of them in flight together); arcs past that are dealt to the
// lanes of the warp and those of hubs to the block, so hubs do not serialise.
// While a round fits one warp, warp 0 runs on alone without block barriers.
__device__ __forceinline__ uint32_t bi_rounds(QueryState &st, WaveShared &W, int &cur, int fb) {
  const DevGraph &g = W.g;
  const CorridorMem &M = W.m;
  const Combo &c = W.c;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  uint32_t relaxed = 0;
  for (uint32_t turn = 0;; ++turn) {
    __syncthreads();
    const uint32_t nc = min(W.nq[cur], (uint32_t)kWaveQ + M.ovf_cap);
    if (nc == 0 || W.stop || turn == kLookAt) break;  // W.stop changes only between the barriers below
    if (nc <= 32u) __syncthreads();  // every warp has read the count
    const bool narrow = nc <= 32u;
    const uint32_t take = narrow ? 32u : min(32u, (nc + (uint32_t)nw - 1u) / (uint32_t)nw);
    uint32_t n = nc;
    if (!narrow || warp == 0) {
      for (uint32_t run = 1;; ++run) {
        for (uint32_t base = (uint32_t)warp * take; base < n; base += (uint32_t)nw * take)
          relaxed += bi_chunk(g, W, M, c, cur, fb, base, min(take, n - base));
        if (!narrow) break;
        __syncwarp();
        if (lane == 0) {
          W.nq[cur] = 0;
          st.n_rounds++;
        }
        cur ^= 1;
        __syncwarp();
        n = vol(W.nq[cur]);
        // (a vote: a lane that went on may list a hub before another one has looked)
        if (__any_sync(0xffffffffu, n == 0 || n > 32u || vol(W.nhub) != 0 || run == kNarrowRun)) break;
      }
    }
    if (!narrow) __syncthreads();
    if (tid == 0) {
      if (!narrow) {
        W.nq[cur] = 0;
        cur ^= 1;
        st.n_rounds++;
      }
      W.cur = cur;
      if (W.overflow || st.abort) W.stop = 1;
    }
    __syncthreads();
    cur = W.cur;
    if (W.nhub != 0) {
      relaxed += bi_hubs(g, W, M, c, cur ^ 1, fb);
      __syncthreads();
      if (tid == 0) W.nhub = 0;
    }
  }
  return relaxed;
}

// Starts a two-sided search: both ends queued, `best0` what W.best starts from.
__device__ __forceinline__ void bi_start(WaveShared &W, const DevGraph &g, const Combo &c, int s, int t,
                                         unsigned long long best0, uint32_t delta) {
  const CorridorMem &M = W.m;
  __syncthreads();
  if (threadIdx.x == 0) {
    W.g = g;
    W.c = c;
    W.delta = delta;
    W.cur = 0;
    W.fb = 0;
    W.mu = kUnset;
    W.best = best0;
    W.nq[0] = 2;
    W.nq[1] = 0;
    W.nhub = 0;
    W.nfar[0] = W.nfar[1] = 0;
    W.far_min = kNoKey;
    W.hi = delta;
    W.rdone = 0;
    W.sides = 3;
    W.clipped = 0;
    W.stop = 0;
    W.ntouch[0] = W.ntouch[1] = 1;
    M.touch[0][0] = (uint32_t)s;
    M.touch[1][0] = (uint32_t)t;
    __stcg(&M.rf[s], make_ulonglong2(0ull, kUnset));
    __stcg(&M.rf[t], make_ulonglong2(kUnset, 0ull));
    W.q[0][0] = (uint32_t)s << 1;
    W.q[0][1] = ((uint32_t)t << 1) | 1u;
  }
}

// Grows both sides, bucket after bucket of width `delta`: to_meeting: until
// the radii cover the best meeting key (W.mu is then the combined distance);
// else until nothing is left below the limit, when every vertex with
// F + H <= T has both its distances: on a shortest way to such a vertex no
// vertex is pruned, since what it is charged for the other side, its distance
// there or the radius of that side, is never more than the truth.
// W.cur / W.fb: queue and far pile in use.
static __device__ __noinline__ uint32_t bi_run(const SearchParams &P, QueryState &st, bool to_meeting) {
  extern __shared__ __align__(16) unsigned char smem[];
  WaveShared &W = *reinterpret_cast<WaveShared *>(smem);
  const CorridorMem &M = W.m;
  const Combo &c = W.c;
  __syncthreads();
  int cur = W.cur, fb = W.fb;
  uint32_t relaxed = 0;
  for (;;) {
    relaxed += bi_rounds(st, W, cur, fb);
    if (W.nq[cur] != 0 && !W.stop) {  // (the same for every thread: nothing changes until the barrier)
      __syncthreads();
      if (threadIdx.x == 0) {
        look_at_limits(P, st);
        if (st.abort) W.stop = 1;
      }
      continue;
    }
    // nothing unsettled lies below far_min on either side
    const uint32_t fm = W.far_min, lo = max(W.hi, fm);
    // Once one side has no vertex left, it has reached all that a path can take:
    // without a meeting, and with nothing left out for its key, there is none.
    const bool apart = W.sides != 3u && vol(W.mu) == kUnset && vol(W.best) == kUnset && !W.clipped;
    const bool stop = fm == kNoKey || W.stop || (to_meeting && (apart || 2ull * lo >= (vol(W.mu) >> 32)));
    __syncthreads();
    if (threadIdx.x == 0) {
      W.rdone = fm == kNoKey ? kKeyMax : lo;
      if (!stop) {
        if (over_time(P, st)) W.stop = 1;
        W.hi = min(lo, kKeyMax + 1u - W.delta) + W.delta;
        W.far_min = kNoKey;
        W.nfar[fb ^ 1] = 0;
        W.sides = 0;
      } else {
        W.cur = cur;
        W.fb = fb;
      }
    }
    __syncthreads();
    if (stop) break;
    // far entries below the new upper key join the queue; one that a shorter
    // way overtook or that the bound rules out is dropped
    const uint32_t fn = min(W.nfar[fb], M.far_cap), hi = W.hi, limit = combo_limit(W, c), rdone = W.rdone;
    uint32_t sides = 0;
    for (uint32_t i = threadIdx.x; i < fn; i += blockDim.x) {
      const unsigned long long x = __ldcg(&M.far[fb][i]);
      const uint32_t key = key_hi(x), e = (uint32_t)x;
      sides |= 1u << (e & 1u);
      if (key < hi) {
        const ulonglong2 pv = ld_pair(&M.rf[e >> 1]);
        const unsigned long long mine = e & 1u ? pv.y : pv.x, other = e & 1u ? pv.x : pv.y;
        const unsigned long long sum = key + (unsigned long long)min(key_hi(other), rdone);
        if (key_hi(mine) == key) {
          if (sum <= limit) wave_push(W, M, cur, e);
          else if (sum > kKeyMax) W.clipped = 1;
        }
      } else if (key <= limit) {
        far_push(W, M, fb ^ 1, key, e);
      }
    }
    if (sides) atomicOr(&W.sides, sides);
    fb ^= 1;
  }
  return relaxed;
}

// ---------------------------------------------------------------- local CSR

// One direction of a renumbered graph: vertex i is old_of(i) of the old graph,
// arcs to vertices without a new id (new_of < 0) are left out.  Arcs of
// vertices with more than a line holds go to (col, w) as well.  False when
// they do not fit (all threads agree).
template <typename OldOf, typename NewOf>
__device__ __forceinline__ bool build_csr(WaveShared &W, const int4 *oline, const int32_t *ocol,
                                          const float2 *ow, int ne, OldOf old_of, NewOf new_of,
                                          int4 *line, int32_t *col, float2 *w, int cap) {
  const unsigned FULL = 0xffffffffu;
  const int G = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  int run = 0;
  for (int base = 0; base < ne; base += G) {
    const int i = base + tid;
    int beg = 0, deg = 0, cnt = 0, large = 0;
    if (i < ne) {
      ArcLine o = load_line(oline, old_of(i));
      deg = o.a[0].w;
      beg = o.a[1].w;
      if (deg <= 4) {
        int nid[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) nid[k] = k < deg ? new_of(o.a[k].x) : -1;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          o.a[k].x = nid[k];
          cnt += nid[k] >= 0;
        }
        // the kept arcs move to the front (four elements: three passes)
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (o.a[k].x < 0) {
              const int4 t = o.a[k];
              o.a[k] = o.a[k + 1];
              o.a[k + 1] = t;
            }
        o.a[0].w = cnt;
        o.a[1].w = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) line[4 * (size_t)i + k] = o.a[k];
      }
    }
    // wider vertices, one after the other by their warp: count, then write
    const unsigned wm = __ballot_sync(FULL, deg > 4);
    for (unsigned m = wm; m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const int b = __shfl_sync(FULL, beg, l), e = b + __shfl_sync(FULL, deg, l);
      int n = 0;
      for (int j = b + lane; j < e; j += 32) n += new_of(ocol[j]) >= 0;
      n = __reduce_add_sync(FULL, n);
      if (lane == l) cnt = n;
    }
    if (deg > 4 && cnt > 4) large = cnt;
    int at = 0;
    if (__syncthreads_or((int)wm)) {
      int total;
      at = run + block_scan_one(large, W.scan, &total);
      run += total;
      if (run > cap) return false;
    }
    for (unsigned m = wm; m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const int b = __shfl_sync(FULL, beg, l), e = b + __shfl_sync(FULL, deg, l);
      const int to = __shfl_sync(FULL, at, l), n = __shfl_sync(FULL, cnt, l), v = __shfl_sync(FULL, i, l);
      int put = 0;
      for (int j0 = b; j0 < e; j0 += 32) {
        const int j = j0 + lane;
        const int id = j < e ? new_of(ocol[j]) : -1;
        const unsigned hit = __ballot_sync(FULL, id >= 0);
        if (id >= 0) {
          const int p = put + __popc(hit & ((1u << lane) - 1u));
          const float2 x = ow[j];
          if (n > 4) {
            col[to + p] = id;
            w[to + p] = x;
          }
          if (p < 4) line[4 * (size_t)v + p] = make_int4(id, (int)x.x, (int)x.y, p == 0 ? n : p == 1 ? to : 0);
        }
        put += __popc(hit);
      }
      if (lane >= put && lane < 4) line[4 * (size_t)v + lane] = make_int4(-1, 0, 0, 0);
      if (lane == 0 && n == 0) line[4 * (size_t)v].w = 0;
    }
  }
  __syncthreads();
  return true;
}

// Copies the corridor of the finished two-sided search (graph W.g) into L
// (og: original ids of its vertices, null for the whole graph).  The new ids
// of those vertices stay in rf until the next reset.  Returns the vertex count;
// -1 (nothing copied) when it does not fit or exceeds `most`.
static __device__ __noinline__ int build_local(const int32_t *og, LocalGraph &L, int most) {
  extern __shared__ __align__(16) unsigned char smem[];
  WaveShared &W = *reinterpret_cast<WaveShared *>(smem);
  const DevGraph &g = W.g;
  const Combo &c = W.c;
  const CorridorMem &M = W.m;
  const int G = blockDim.x, tid = threadIdx.x;
  __syncthreads();
  if (tid == 0) W.cnt = 0;
  __syncthreads();
  const uint32_t nt = W.ntouch[0], limit = combo_limit(W, c), cap = (uint32_t)min(M.lv, most);
  for (uint32_t i = tid; i < nt; i += G) {
    const uint32_t v = __ldcg(&M.touch[0][i]);
    const ulonglong2 p = ld_pair(&M.rf[v]);
    if (p.y != kUnset && (unsigned long long)key_hi(p.x) + key_hi(p.y) <= limit) {
      const uint32_t id = warp_agg_inc(&W.cnt);
      if (id < cap) {
        M.map[id] = v;
        L.gid[id] = og ? og[v] : (int32_t)v;
        __stcg(reinterpret_cast<unsigned long long *>(&M.rf[v]) + 1,
               ((unsigned long long)kMemberTag << 32) | id);
      }
    }
  }
  __syncthreads();
  if (W.cnt > cap) return -1;
  const int ne = (int)W.cnt;
  const uint32_t *map = M.map;
  auto old_of = [map](int i) { return (int)map[i]; };
  const ulonglong2 *rf = M.rf;
  auto new_of = [rf](int v) {
    const unsigned long long h = __ldcg(reinterpret_cast<const unsigned long long *>(&rf[v]) + 1);
    return key_hi(h) == kMemberTag ? (int)(uint32_t)h : -1;
  };
  if (!build_csr(W, g.line, g.col, g.w, ne, old_of, new_of, const_cast<int4 *>(L.g.line),
                 const_cast<int32_t *>(L.g.col), const_cast<float2 *>(L.g.w), M.la))
    return -1;
  if (!build_csr(W, g.rline, g.rcol, g.rw, ne, old_of, new_of, const_cast<int4 *>(L.g.rline),
                 const_cast<int32_t *>(L.g.rcol), const_cast<float2 *>(L.g.rw), M.la))
    return -1;
  if (tid == 0) L.g.n = ne;
  __syncthreads();
  return ne;
}

// Distances of a local pass: in shared memory (behind the wave state) where
// the graph fits, else in the worker's global array.
template <bool kShared>
struct DistArray {
  unsigned long long *p;
  __device__ __forceinline__ unsigned long long get(int i) const {
    if (kShared) return *reinterpret_cast<const volatile unsigned long long *>(p + i);
    return __ldcg(p + i);
  }
  __device__ __forceinline__ void set(int i, unsigned long long x) const {
    if (kShared) *reinterpret_cast<volatile unsigned long long *>(p + i) = x;
    else __stcg(p + i, x);
  }
};

template <bool kShared, bool kWhole>
__device__ __forceinline__ uint32_t local_chunk(WaveShared &W, const DistArray<kShared> &D, int cur,
                                                int fb, uint32_t i0, uint32_t take) {
  const CorridorMem &M = W.m;
  const PassArgs &A = W.a;
  const Combo &c = W.c;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, nxt = cur ^ 1;
  const uint32_t hi = vol(W.hi), limit = A.limit;
  int beg = 0, deg = 0;
  uint32_t key = 0, sec = 0;
  ArcLine line;
  if ((uint32_t)lane < take) {
    const int v = (int)wave_get(W, M, cur, i0 + (uint32_t)lane);
    const unsigned long long x = D.get(v);
    line = load_line(A.line, v);
    deg = line.a[0].w;
    beg = line.a[1].w;
    key = key_hi(x);
    sec = (uint32_t)x;
  }
  auto relax = [&](uint32_t on, const int (&u)[kArcBatch], const int2 (&w)[kArcBatch],
                   const uint32_t (&k0)[kArcBatch], const uint32_t (&s0)[kArcBatch]) {
    unsigned long long cand[kArcBatch], old[kArcBatch];
    uint32_t e[kArcBatch], nkey[kArcBatch], near = 0, far = 0;
#pragma unroll
    for (int k = 0; k < kArcBatch; ++k) {
      cand[k] = 0;
      if (on >> k & 1u) {
        const uint32_t ln = (uint32_t)w[k].x, dl = (uint32_t)w[k].y;
        unsigned long long nk =
            k0[k] + (unsigned long long)c.a * ln + (unsigned long long)c.b * dl;
        if (kWhole) nk += A.hop;
        if (nk > limit || (kWhole && ((float)w[k].x > A.max_len || (float)w[k].y < A.min_delay))) {
          if (kWhole && nk > kKeyMax) W.clipped = 1;
          on &= ~(1u << k);
        } else {
          cand[k] = (nk << 32) | add_second(s0[k], c.pure ? ln : dl);
          if (cand[k] >= D.get(u[k])) on &= ~(1u << k);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kArcBatch; ++k)
      if (on >> k & 1u) old[k] = atomicMin(&D.p[u[k]], cand[k]);
#pragma unroll
    for (int k = 0; k < kArcBatch; ++k) {
      e[k] = (uint32_t)u[k];
      nkey[k] = key_hi(cand[k]);
      if ((on >> k & 1u) && cand[k] < old[k]) {
        if (nkey[k] < hi) near |= 1u << k;
        else far |= 1u << k;
      }
    }
    wave_emit<kArcBatch>(W, M, nxt, fb, e, nkey, near, far, 0u, false);
  };
  int u[kArcBatch];
  int2 w[kArcBatch];
  uint32_t k0[kArcBatch], s0[kArcBatch], on = 0;
#pragma unroll
  for (int k = 0; k < kArcBatch; ++k) {
    k0[k] = key;
    s0[k] = sec;
    if (k < deg) {
      u[k] = line.a[k].x;
      w[k] = make_int2(line.a[k].y, line.a[k].z);
      on |= 1u << k;
    }
  }
  relax(on, u, w, k0, s0);
  unsigned wide = __ballot_sync(FULL, deg > kArcBatch);
  for (; wide; wide &= wide - 1) {  // the further arcs of one vertex after the other
    const int l = __ffs(wide) - 1;
    const int b0 = __shfl_sync(FULL, beg, l) + kArcBatch, e0 = b0 - kArcBatch + __shfl_sync(FULL, deg, l);
    const uint32_t ok = __shfl_sync(FULL, key, l), os = __shfl_sync(FULL, sec, l);
    for (int j0 = b0; j0 < e0; j0 += 32 * kArcBatch) {
      on = 0;
#pragma unroll
      for (int k = 0; k < kArcBatch; ++k) {
        const int j = j0 + 32 * k + lane;
        k0[k] = ok;
        s0[k] = os;
        if (j < e0) {
          const float2 x = A.w[j];
          u[k] = A.col[j];
          w[k] = make_int2((int)x.x, (int)x.y);
          on |= 1u << k;
        }
      }
      relax(on, u, w, k0, s0);
    }
  }
  return (uint32_t)deg;
}

// Runs a local pass with the whole block; `out` receives the distances.
// Latency-bound like bi_rounds; a corridor is long and narrow, so most rounds
// fit one warp and run without block barriers, on shared-memory distances.
template <bool kShared, bool kWhole = false, typename Params, typename State>
static __device__ __noinline__ uint32_t local_pass_in(const Params &P, State &st, unsigned long long *out) {
  extern __shared__ __align__(16) unsigned char smem[];
  WaveShared &W = *reinterpret_cast<WaveShared *>(smem);
  const CorridorMem &M = W.m;
  const PassArgs &A = W.a;
  const int G = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = G >> 5;
  DistArray<kShared> D;
  D.p = kShared ? reinterpret_cast<unsigned long long *>(smem + kWaveBytes) : out;
  __syncthreads();
  for (int i = tid; i < A.n; i += G) D.set(i, i == A.root ? 0ull : kUnset);
  if (tid == 0) {
    W.nq[0] = 1;
    W.nq[1] = 0;
    W.nfar[0] = W.nfar[1] = 0;
    W.far_min = kNoKey;
    W.hi = A.delta;
    W.stop = 0;
    W.mu = kUnset;
    W.q[0][0] = (uint32_t)A.root;
  }
  uint32_t relaxed = 0, turn = 0;
  int cur = 0, fb = 0;
  for (;;) {
    __syncthreads();
    const uint32_t nc = min(W.nq[cur], (uint32_t)kWaveQ + M.ovf_cap);
    if (W.stop) break;  // changes only between the barriers below
    if (nc == 0) {
      const uint32_t fm = W.far_min, fn = min(W.nfar[fb], M.far_cap);
      if (fm == kNoKey) break;
      __syncthreads();
      if (tid == 0) {
        over_time(P, st);
        if (W.overflow || st.abort) W.stop = 1;
        if (kWhole && A.target >= 0) W.a.limit = min(A.limit, key_hi(D.get(A.target)));
        W.hi = min(max(W.hi, fm), kKeyMax + 1u - A.delta) + A.delta;
        W.far_min = kNoKey;
        W.nfar[fb ^ 1] = 0;
      }
      __syncthreads();
      const uint32_t hi = W.hi;
      for (uint32_t i = tid; i < fn; i += G) {
        const unsigned long long x = __ldcg(&M.far[fb][i]);
        if (key_hi(x) < hi) {
          if (key_hi(D.get((int)(uint32_t)x)) == key_hi(x)) wave_push(W, M, cur, (uint32_t)x);
        } else {
          far_push(W, M, fb ^ 1, key_hi(x), (uint32_t)x);
        }
      }
      fb ^= 1;
      continue;
    }
    if (nc <= 32u) {
      __syncthreads();  // every warp has read the count
      if (warp == 0) {
        uint32_t n = nc, run = 0;
        do {
          relaxed += local_chunk<kShared, kWhole>(W, D, cur, fb, 0, n);
          __syncwarp();
          if (lane == 0) {
            W.nq[cur] = 0;
            st.n_rounds++;
          }
          cur ^= 1;
          __syncwarp();
          n = vol(W.nq[cur]);
        } while (n != 0 && n <= 32u && ++run != kNarrowRun);
        if (lane == 0) W.cur = cur;
      }
    } else {
      const uint32_t take = min(32u, (nc + (uint32_t)nw - 1u) / (uint32_t)nw);
      for (uint32_t base = (uint32_t)warp * take; base < nc; base += (uint32_t)nw * take)
        relaxed += local_chunk<kShared, kWhole>(W, D, cur, fb, base, min(take, nc - base));
      __syncthreads();
      if (tid == 0) {
        W.nq[cur] = 0;
        W.cur = cur ^ 1;
        st.n_rounds++;
      }
    }
    if (tid == 0) {
      if (++turn % kLookAt == 0) look_at_limits(P, st);
      if (W.overflow || st.abort) W.stop = 1;
    }
    __syncthreads();
    cur = W.cur;
  }
  __syncthreads();
  if (kShared) {
    for (int i = tid; i < A.n; i += G) __stcg(&out[i], D.get(i));
    __syncthreads();
  }
  return relaxed;
}

__device__ __forceinline__ uint32_t local_pass(const SearchParams &P, QueryState &st, WaveShared &W,
                                               const PassArgs &A, const Combo &c,
                                               unsigned long long *out) {
  __syncthreads();
  if (threadIdx.x == 0) {
    W.a = A;
    W.c = c;
  }
  __syncthreads();
  const int cap = (int)((table_region_bytes(P.table_log2, P.lock_log2) - kWaveBytes) / sizeof(unsigned long long));
  return A.n <= cap ? local_pass_in<true>(P, st, out) : local_pass_in<false>(P, st, out);
}

// ----------------------------------------------------------------- multipliers

// (a, b) with b / a close to lambda and a * ub + b * B <= kKeyMax.  False when
// one of them would vanish.
__device__ inline bool pick_combo(double lambda, double ub, double B, Combo *c) {
  const double s = (double)(kKeyMax - 1u) / fmax(1.0, ub + lambda * B);
  const double a = floor(fmin(s, 1073741824.0)), b = floor(fmin(lambda * s, 1073741824.0));
  if (!(a >= 1.0) || !(b >= 1.0)) return false;
  c->a = (uint32_t)a;
  c->b = (uint32_t)b;
  c->pure = false;
  return true;
}

// Bucket width of a wave in key units: a few mean arcs.
__device__ __forceinline__ uint32_t combo_delta(const SearchParams &P, const Combo &c, float mult) {
  const double d = (double)mult * ((double)c.a * P.mean_len + (double)c.b * P.mean_delay);
  return (uint32_t)fmin(fmax(d, 1.0), 536870912.0);
}

enum CorridorResult { kCorridorNone = 0, kCorridorReady = 1, kCorridorInfeasible = 2 };

// What is known about a query's paths while its corridor is built.  (len,
// delay) pairs of real paths: p1 the best combined path that is too slow, p2
// the best combined path within the budget; ub the smallest cost of any path
// within the budget.  < 0: none yet.
struct Duals {
  double ub, ub_delay, len1, del1, len2, del2;

  __device__ void feasible(double len, double del) {
    if (ub < 0.0 || len < ub) {
      ub = len;
      ub_delay = del;
    }
  }
  // The best path under (c.a, c.b), as (key, delay).
  __device__ void optimum(const Combo &c, unsigned long long x) {
    const double del = (double)(uint32_t)x;
    const double len = floor(((double)(x >> 32) - (double)c.b * del) / (double)c.a);
    if (del <= (double)c.B) {
      feasible(len, del);
      len2 = len;
      del2 = del;
    } else {
      len1 = len;
      del1 = del;
    }
  }
  // Slope between the best paths on both sides of the budget (Handler and
  // Zang's next multiplier), < 0 while one is missing.
  __device__ double slope() const {
    if (len1 < 0.0) return -1.0;
    const double l2 = len2 >= 0.0 ? len2 : ub, d2 = len2 >= 0.0 ? del2 : ub_delay;
    if (l2 < 0.0 || !(del1 > d2) || !(l2 > len1)) return -1.0;
    return (l2 - len1) / (del1 - d2);
  }
  __device__ uint32_t T(const Combo &c) const {
    return (uint32_t)((unsigned long long)c.a * (unsigned long long)ub + (unsigned long long)c.b * c.B);
  }
};

// Builds the query's corridor (all threads; every thread computes the same
// multipliers).  kCorridorReady: local graph *which holds it, M.state is
// filled, st.src / st.dst are local ids, st.inc_key carries the cost bound,
// st.lam_* the multiplier and st.ord_* the order of the search; kCorridorInfeasible: no path within the
// budget; kCorridorNone: not handled here (costs from 2^24 on, or a corridor
// past the local capacity).
static __device__ __noinline__ int corridor_prepare(const SearchParams &P, QueryState &st, int *which) {
  extern __shared__ __align__(16) unsigned char smem[];
  WaveShared &W = *reinterpret_cast<WaveShared *>(smem);
  CorridorMem &M = W.m;
  const unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, G = blockDim.x;
  const uint32_t B = (uint32_t)floorf(st.budget);
  const int s = st.src, t = st.dst;
  const double unit = fmax((double)P.mean_len, 1e-3) / fmax((double)P.mean_delay, 1e-3);
  if (tid == 0) {
    W.overflow = 0;
    W.stop = 0;
    W.ntouch[0] = W.ntouch[1] = 0;
  }
  uint32_t relaxed = 0;
  Duals k{-1.0, 0.0, -1.0, 0.0, -1.0, 0.0};
  const float mult = fminf(P.wave_mult, fmaxf(2.0f, kBudgetShare * (float)B / fmaxf(P.mean_delay, 1e-3f)));
  double lambda = unit * kFirstLambda;
  int result = kCorridorNone, ne = -1, cl = -1, ls = s, lt = t;  // cl: graph searched (-1: the whole one)
  // the Pareto set takes every vertex on a way within the budget: the pure
  // delay search alone
  const bool pareto = P.mode == VINE_MODE_PARETO;
  bool pure = pareto;
  Combo c;
  c.B = B;
  for (int attempt = 0;; ++attempt) {
    // before a path is known its cost is taken to be at most 16 times what
    // the budget suggests; where that fails the pure delay search answers
    const double guess = k.ub >= 0.0 ? k.ub : fmin((double)kIntLimit, 16.0 * (B + P.mean_delay) * unit);
    if (!pure && !pick_combo(lambda, guess, (double)B, &c)) {
      if (k.ub >= 0.0) break;
      pure = true;
    }
    if (pure) {
      c.a = 0;
      c.b = 1;
    }
    c.pure = pure;
    unsigned long long best0 = kUnset;
    if (k.ub >= 0.0)
      best0 = ((unsigned long long)(pure ? (uint32_t)k.ub : k.T(c)) << 32) | (uint32_t)k.ub_delay;
    const DevGraph &g = cl < 0 ? P.g : M.loc[cl].g;
    const uint32_t delta = combo_delta(P, c, mult);
    bi_start(W, g, c, ls, lt, best0, delta);
    relaxed += bi_run(P, st, true);
    if (W.stop) break;
    const unsigned long long mu = W.mu, best = W.best;
    if (best != kUnset) {
      const double cost = pure ? (double)(best >> 32)
                               : floor((double)((best >> 32) - (unsigned long long)c.b * B) / (double)c.a);
      k.feasible(cost, (double)(uint32_t)best);
    }
    if (mu != kUnset && !pure) {
      if ((mu >> 32) <= kKeyMax) {
        k.optimum(c, mu);
      } else if ((uint32_t)mu <= B) {
        // a path past the keys kept: not known to be the best one, but real
        k.feasible(floor(((double)(mu >> 32) - (double)c.b * (double)(uint32_t)mu) / (double)c.a), (double)(uint32_t)mu);
      }
    }
    if (k.ub < 0.0) {
      // nothing feasible seen: unreachable, or weigh the delay more, at last alone
      if (pure || (mu == kUnset && !W.clipped)) {
        result = kCorridorInfeasible;
        break;
      }
      bi_reset(W, M);
      if (attempt == 0 && mu != kUnset) lambda *= 4.0;
      else pure = true;
      continue;
    }
    if (k.ub >= (double)kIntLimit) break;
    if (best == kUnset) {
      // the weights were made for a cheaper path: a * ub + b * B passes
      // kKeyMax, so no limit holds this one.  Again, with weights for its cost.
      bi_reset(W, M);
      continue;
    }
    // The next multiplier to try: the slope once both sides of the budget
    // are known, else less weight on the delay.
    double next = k.slope();
    if (next < 0.0) {
      // the more of the budget the best combined path leaves, the smaller the
      // multiplier: on the road graphs a path with 0.95 of the budget met
      // multipliers about half as large, 0.92 a quarter (ratio^16)
      const float used = k.len2 >= 0.0 && !pure ? (float)(k.del2 / fmax(1.0, (double)B)) : 0.9f;
      float f = used * used;
      f *= f;
      f *= f;
      f *= f;
      next = (pure ? unit : lambda) * (double)fminf(0.7f, fmaxf(0.1f, f));
    }
    const bool settled = !pure && fabs(next - lambda) <= 0.1 * lambda;
    // A wide gap between T and the meeting key means a poor multiplier:
    // another search now costs less than completing this one.
    const double gap = pure ? 1.0 : ((double)k.T(c) - (double)(mu >> 32)) / fmax(1.0, (double)(mu >> 32));
    if (pareto || attempt >= 4 || settled || cl >= 0 || !(gap > kWideGap)) {
      __syncthreads();
      relaxed += bi_run(P, st, false);
      if (W.stop) break;
      const unsigned long long b2 = W.best;
      k.feasible(pure ? (double)(b2 >> 32)
                      : floor((double)((b2 >> 32) - (unsigned long long)c.b * B) / (double)c.a),
                 (double)(uint32_t)b2);
      const int to = cl < 0 ? 0 : cl ^ 1;
      const int n2 = build_local(cl < 0 ? nullptr : M.loc[cl].gid, M.loc[to],
                                 cl < 0 ? M.lv : ne - ne / 4);
      if (n2 >= 0) {
        const unsigned long long ms = __ldcg(reinterpret_cast<const unsigned long long *>(&M.rf[ls]) + 1);
        const unsigned long long mt = __ldcg(reinterpret_cast<const unsigned long long *>(&M.rf[lt]) + 1);
        if (key_hi(ms) != kMemberTag || key_hi(mt) != kMemberTag) {  // both ends lie in every corridor
          ne = -1;
          break;
        }
        ls = (int)(uint32_t)ms;
        lt = (int)(uint32_t)mt;
        cl = to;
        ne = n2;
      }
      if (pareto || settled || attempt >= 6 || (ne >= 0 && ne <= kShrinkTo)) break;
    }
    bi_reset(W, M);
    lambda = next;
    pure = false;
  }
  const bool stopped = W.stop != 0;
  bi_reset(W, M);
  if (stopped) ne = -1;

  unsigned long long *D0 = M.dist[0], *D1 = M.dist[1], *Hbest = M.dist[2], *Hcur = M.dist[3];
  Combo use;
  use.a = use.b = 0;
  if (ne >= 0) {
    // ---- bounds on the corridor: delay, length, best multiplier
    const DevGraph &g = M.loc[cl].g;
    const bool wide = ne > 4096;  // one bucket on small graphs
    const uint32_t one = 0x40000000u;
    Combo cd{0u, 1u, true, B}, cl_{1u, 0u, false, B};
    PassArgs A{g.rline, g.rcol, g.rw, ne, lt, B, wide ? combo_delta(P, cd, P.wave_mult) : one};
    relaxed += local_pass(P, st, W, A, cd, D0);
    const unsigned long long xd = __ldcg(&D0[ls]);  // the fastest path
    if (pareto) {
      // no sink label longer than the fastest path (the shortest of those)
      // is in the Pareto set
      k.ub = xd != kUnset ? (double)(uint32_t)xd : (double)kIntLimit;
      if (k.ub >= (double)kIntLimit) ne = -1;
    } else if (xd != kUnset) {
      k.feasible((double)(uint32_t)xd, (double)(xd >> 32));
      if (k.len2 < 0.0) {
        k.len2 = (double)(uint32_t)xd;
        k.del2 = (double)(xd >> 32);
      }
    }
    A.limit = ne >= 0 ? (uint32_t)k.ub : 0u;
    A.delta = wide ? combo_delta(P, cl_, P.wave_mult) : one;
    relaxed += local_pass(P, st, W, A, cl_, D1);
    const unsigned long long xl = __ldcg(&D1[ls]);  // the shortest path
    if (xl != kUnset && !pareto) {
      const double l0 = (double)(xl >> 32), d0 = (double)(uint32_t)xl;
      if (d0 <= (double)B) {
        k.feasible(l0, d0);  // the answer's cost
      } else {
        if (k.len1 < 0.0) {
          k.len1 = l0;
          k.del1 = d0;
        }
        double lb = -1.0;
        for (int it = 0; it < 8 && !st.abort && !W.overflow; ++it) {
          const double next = k.slope();
          if (next < 0.0 || !pick_combo(next, k.ub, (double)B, &c)) break;
          const double l2 = k.len2, d2 = k.del2, l1 = k.len1, d1 = k.del1;
          A.limit = k.T(c);
          A.delta = wide ? combo_delta(P, c, P.wave_mult) : one;
          relaxed += local_pass(P, st, W, A, c, Hcur);
          const unsigned long long x = __ldcg(&Hcur[ls]);
          if (x == kUnset) break;
          const double low = ((double)(x >> 32) - (double)c.b * (double)B) / (double)c.a;
          if (use.a == 0 || low > lb) {
            lb = low;
            use = c;
            unsigned long long *h = Hbest;
            Hbest = Hcur;
            Hcur = h;
          }
          k.optimum(c, x);
          // done when no path lies below the line through the two points, or
          // when the bound meets the cost
          const double line = fmin((double)c.a * l1 + (double)c.b * d1, (double)c.a * l2 + (double)c.b * d2);
          if ((double)(x >> 32) >= line || ceil(low) >= k.ub) break;
        }
      }
    }
  }
  __syncthreads();
  relaxed = __reduce_add_sync(FULL, relaxed);
  if ((tid & 31) == 0)
    atomicAdd(reinterpret_cast<unsigned long long *>(&st.n_relaxed), (unsigned long long)relaxed);
  if (W.overflow && tid == 0 && !st.abort) fail_query(st, VINE_ERR_CAPACITY, kSiteBand);
  if (ne >= 0) {
    for (int i = tid; i < ne; i += G) {
      const unsigned long long hd = __ldcg(&D0[i]), hl = __ldcg(&D1[i]);
      const uint32_t hm = use.a ? key_hi(__ldcg(&Hbest[i])) : 0u;
      const bool in = hd != kUnset && hl != kUnset && hm != kNoKey;
      M.state[i] = make_uint4(key_hi(hd), in ? key_hi(hl) : kNoKey, hm, kNoKey);
    }
    if (tid == 0) {
      st.src = ls;
      st.dst = lt;
      st.lam_a = use.a;
      st.lam_b = use.b;
      st.lam_bB = use.b * B;
      st.inc_key = pack_key((float)k.ub, INFINITY);
      Combo o = use;  // the search's order: the same weights, else both criteria alike
      if (use.a == 0 && !pick_combo(unit, k.ub, (double)B, &o)) o.a = o.b = 1;
      if (pareto) {  // by cost alone (see known_better)
        o.a = 1;
        o.b = 0;
      }
      st.ord_a = o.a;
      st.ord_b = o.b;
    }
    *which = cl;
    result = kCorridorReady;
  }
  __syncthreads();
  return result;
}

}  // namespace vine
