// k_link.cu -- tight triplet connectivity, circle fit and the cellular automaton.
//
// Connectivity replaces tripletEtaCalculatorStore / tripletConnectivityTightCount /
// tripletConnectivityTightStore / predicateInversionStore /
// streamCompactionGetValidIndexesStore (TripletConnectivityTight.h:47-346,
// .cpp:5-475).  The reference scans, for every basis triplet, the whole next
// layer-triplet segment; here the followers sharing the basis' two outer hits
// are found by binary search, because inside one segment the triplets are
// ordered by (second hit, first hit) -- the pair order -- and where each
// layer is the second of one layer triplet at most, from the run of triplets
// with that second hit on.  The search range is
// the reference's [offsets[k], offsets[k+1]) (with its quirks: the segment
// skip of :113-115, the event check of :130-132, the monotonized offsets)
// intersected with the true segment k, outside of which no follower can
// share the basis' hits.
//
// The circle fit is trackletCircleFitterStore (TrackletCircleFitter.h:32-97).
//
// The CA replaces the host-driven iteration loop and the backward kernels of
// CellularAutomaton.{h,cpp}.  Its forward phase converges to the length of
// the longest chain of links ending at each triplet (a link only ever raises
// a follower whose state equals its basis', so a basis can never overtake
// its follower, and at the fixed point every follower sits one above its
// highest basis); links always point to a higher layer triplet, so that fixed
// point is computed exactly in one sweep over the layer triplets, with no
// host round trip.  The backward phase keeps the reference's semantics:
// candidate bases with state + 1 == follower state, minimum |pT difference|
// with select-by-multiply, scanned in link order (ascending basis index, one
// of the orders the reference's atomic_inc allows).
#include "trax_kernels.h"

namespace trax {

namespace {

int grid_for(uint64_t items, int threads) {
  uint64_t blocks = (items + threads - 1) / threads;
  uint64_t cap = (uint64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

#define GRID_STRIDE(i, n) for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

// What connectivity starts from (TripletConnectivityTight.h:47-74), in one pass
// over the triplets.
__global__ void __launch_bounds__(256)
    link_start_kernel(Stamp stamp, DevConfig cfg, const float4* __restrict__ hits, const uint32_t* __restrict__ h1,
                      const uint32_t* __restrict__ h2, const uint32_t* __restrict__ h3, const uint32_t* nTDev,
                      LinkStart link) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  GRID_STRIDE(t, nT) {
    const float4 a = hits[trax_hit(h1[t], cfg)], b = hits[trax_hit(h3[t], cfg)];
    const float px = b.x - a.x, py = b.y - a.y, pz = b.z - a.z;
    const float tt = div_(pz, sqrt_(px * px + py * py));
    link.eta[t] = asinh_(tt);
    link.inDeg[t] = 0u;
    link.inCursor[t] = 0u;
    if (link.runs) {
      const uint32_t mid = trax_hit(h2[t], cfg);
      const uint32_t prev = t ? trax_hit(h2[t - 1], cfg) : mid;
      if (t == 0 || prev != mid) {
        link.runs[mid].x = t;
        if (t) link.runs[prev].y = t;
      }
      if (t + 1 == nT) link.runs[mid].y = nT;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) link.inDeg[nT] = 0u;  // the scan's +1 slot
}

// The segments of a caller's triplets: segStart[s] = first triplet of segment s
// or later.  A triplet whose segment differs from its predecessor's starts all
// segments in between; the warp fills a gap of empty ones together.
__global__ void __launch_bounds__(256)
    triplet_segments_kernel(Stamp stamp, DevConfig cfg, const uint32_t* __restrict__ hitEvt,
                            const uint32_t* __restrict__ hitLayer, const uint32_t* __restrict__ h1,
                            const uint32_t* nTDev, uint32_t* segStart, uint32_t* segOf) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  const uint32_t S = cfg.E * cfg.nLT;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < nT; base += gridDim.x * blockDim.x) {
    const uint32_t t = base + lane;
    uint32_t seg = 0;
    if (t < nT) {
      const uint32_t hi = trax_hit(h1[t], cfg);
      seg = hitEvt[hi] * cfg.nLT + (hitLayer[hi] - 1);
      segOf[t] = seg;
    }
    // the first segment this triplet starts: after its predecessor's
    uint32_t from = __shfl_up_sync(0xffffffffu, seg, 1) + 1u;
    if (lane == 0) {
      if (t == 0) {
        from = 0u;
      } else {
        const uint32_t hp = trax_hit(h1[t - 1], cfg);
        from = hitEvt[hp] * cfg.nLT + (hitLayer[hp] - 1) + 1u;
      }
    }
    const bool starts = t < nT && from <= seg;
    if (starts && seg <= S) segStart[seg] = t;
    uint32_t gaps = __ballot_sync(0xffffffffu, starts && from < seg);
    while (gaps) {
      const int l = __ffs(gaps) - 1;
      gaps &= gaps - 1u;
      const uint32_t a = __shfl_sync(0xffffffffu, from, l), b = __shfl_sync(0xffffffffu, seg, l);
      for (uint32_t s = a + lane; s < b && s <= S; s += 32u) segStart[s] = base + l;
    }
    if (base + 32u >= nT) {  // the warp with the last triplet: nothing starts after it
      const uint32_t last = __shfl_sync(0xffffffffu, seg, (nT - 1u) & 31u);
      for (uint32_t s = last + 1u + lane; s <= S; s += 32u) segStart[s] = nT;
    }
  }
}

// trackletOffsets: filterOffsetStore (TripletThetaPhiFilter.h:221-257) writes
// the first triplet of every segment that holds one, and the last triplet
// after the last such segment; the monotonize kernel (:267-280) lets empty
// segments inherit their predecessor's value, a running maximum.  One CTA,
// OFF_ITEMS consecutive segments per thread and step.
constexpr int OFF_THREADS = 1024, OFF_ITEMS = 8;
__global__ void __launch_bounds__(OFF_THREADS)
    triplet_offsets_kernel(Stamp stamp, uint32_t S, const uint32_t* nTDev, uint32_t* segStart, uint32_t* offsets) {
  stamp_begin(stamp);
  __shared__ uint32_t s_warp[OFF_THREADS / 32];
  const uint32_t nT = *nTDev;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t s0 = 0; s0 <= S; s0 += OFF_THREADS * OFF_ITEMS) {
    const uint32_t a = s0 + threadIdx.x * OFF_ITEMS;
    uint32_t v[OFF_ITEMS];
    // start of segment a - 1, a, ...: nT == 0 leaves them unwritten, all 0
    uint32_t prev = nT && a > 0 && a <= S ? segStart[a - 1] : 0u;
    uint32_t cur = nT && a <= S ? segStart[a] : 0u;
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < OFF_ITEMS; ++k) {
      const uint32_t s = a + k;
      const uint32_t next = nT && s < S ? segStart[s + 1] : cur;
      uint32_t x = 0;
      if (s < S && next > cur) x = cur;                                    // holds triplets: its first
      if (s > 0 && s <= S && nT > 1 && cur == nT && prev < nT) x = nT - 1;  // after the last one that does
      m = max(m, x);
      v[k] = m;
      prev = cur;
      cur = next;
    }
    uint32_t incl = m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= (uint32_t)d) incl = max(incl, t);
    }
    if (lane == 31) s_warp[warp] = incl;
    uint32_t before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= (uint32_t)d) w = max(w, t);
      }
      s_warp[lane] = w;  // inclusive over the warps
    }
    __syncthreads();
    before = max(max(before, carry), warp ? s_warp[warp - 1] : 0u);
#pragma unroll
    for (int k = 0; k < OFF_ITEMS; ++k)
      if (a + k <= S) offsets[a + k] = max(before, v[k]);
    carry = max(carry, s_warp[OFF_THREADS / 32 - 1]);
    __syncthreads();
  }
}

// first index in [lo, hi) whose (h2, h1) key is >= (k2, k1)
__device__ __forceinline__ uint32_t key_lower_bound(const uint32_t* h1, const uint32_t* h2, uint32_t lo, uint32_t hi,
                                                    uint32_t k1, uint32_t k2) {
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    uint32_t a2 = h2[mid], a1 = h1[mid];
    if (a2 < k2 || (a2 == k2 && a1 < k1)) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Followers of every basis triplet.  The count pass adds to the followers'
// in-degrees (for the CA and the connectable flags) and leaves where it
// started looking to the store pass.
__global__ void __launch_bounds__(256)
    conn_count_kernel(Stamp stamp, DevConfig cfg, const uint32_t* __restrict__ hitEvt,
                      const uint32_t* __restrict__ hitLayer, const uint32_t* __restrict__ h1,
                      const uint32_t* __restrict__ h2, const uint32_t* __restrict__ h3, const uint32_t* nTDev,
                      const float* __restrict__ eta, const uint32_t* __restrict__ offsets,
                      const uint32_t* __restrict__ segStart, const uint2* __restrict__ runs, uint32_t* linkCount,
                      uint32_t* inDeg, uint32_t* runStart, bool sortedSegments) {
  stamp_begin(stamp);
  const uint32_t S = cfg.E * cfg.nLT;
  const uint32_t nT = S > 0 ? *nTDev : 0u;
  const float dEtaCut = cfg.dEtaCut;
  GRID_STRIDE(t, nT) {
    uint32_t cnt = 0;
    bool ok = !(t >= offsets[S - 1]);  // :113-115 (nOffsets - 2 == S - 1)
    uint32_t begin = 0, end = 0, k = 0;
    const uint32_t inner = h2[t], outer = h3[t];
    if (ok) {
      const uint32_t ev = hitEvt[trax_hit(inner, cfg)];
      k = ev * cfg.nLT + (hitLayer[trax_hit(inner, cfg)] - 1);
      ok = k < S;  // the reference would read past the offsets
      if (ok) {
        begin = offsets[k];
        end = offsets[k + 1];
        // :130-132; an empty range has no follower to compare (the reference
        // reads one past its triplets there) and gives no links either way
        ok = begin < end && ev == hitEvt[trax_hit(h1[begin], cfg)];
      }
    }
    if (ok) {
      uint32_t lo = max(begin, segStart[k]);
      uint32_t hi = min(end, segStart[k + 1]);
      const float localEta = eta[t];
      // sorted segments: binary search to the (h2, h1) run, among the
      // triplets with that second hit where their place is known (`runs`:
      // a few of them instead of the segment's, 1.01 -> 0.50 ms for the 29 M
      // triplets of the pileup batch); otherwise scan the whole range like
      // the reference (caller-provided triplets)
      if (runs) {
        const uint2 run = runs[trax_hit(outer, cfg)];
        if (run.x < nT && h2[run.x] == outer) {
          lo = max(lo, run.x);
          hi = min(hi, run.y);
        } else {
          hi = lo;  // no triplet has that second hit
        }
      }
      const uint32_t first = sortedSegments ? key_lower_bound(h1, h2, lo, hi, inner, outer) : lo;
      runStart[t] = first;
      for (uint32_t i = first; i < hi; ++i) {
        if (h2[i] != outer || h1[i] != inner) {
          if (sortedSegments) break;
          continue;
        }
        if (fabs_(localEta - eta[i]) < dEtaCut) {
          atomicAdd(&inDeg[i], 1u);
          ++cnt;
        }
      }
    }
    linkCount[t] = cnt;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) linkCount[nT] = 0u;
}

// The links of the bases that have some, in basis order; every link also
// takes a place in its follower's list of incoming bases.  The Q9 predicate
// streams over the first nT-1 triplets come out on the way as words of 32
// flags (connectable: a basis or a follower of some link) with the number set
// per word, so that the compaction scans one value per 32 triplets.
__global__ void __launch_bounds__(256)
    conn_store_kernel(Stamp stamp, DevConfig cfg, const uint32_t* __restrict__ h1, const uint32_t* __restrict__ h2,
                      const uint32_t* __restrict__ h3, const uint32_t* nTDev, const float* __restrict__ eta,
                      LinkStore ls) {
  stamp_begin(stamp);
  const uint32_t nT = cfg.E * cfg.nLT > 0 ? *nTDev : 0u;
  const float dEtaCut = cfg.dEtaCut;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < nT; base += gridDim.x * blockDim.x) {
    const uint32_t t = base + lane;
    uint32_t pos = 0, limit = 0;
    bool connectable = false;
    if (t < nT) {
      pos = ls.linkStart[t];
      limit = ls.linkStart[t + 1] - pos;
      connectable = t + 1 < nT && (limit != 0u || ls.inStart[t] != ls.inStart[t + 1]);
    }
    const uint32_t word = __ballot_sync(0xffffffffu, connectable);
    if (lane == 0) {
      ls.connWords[base >> 5] = word;
      ls.connSums[base >> 5] = (uint32_t)__popc(word);
    }
    if (limit == 0u) continue;
    if (pos >= ls.capLinks) limit = 0;
    else if (limit > ls.capLinks - pos) limit = ls.capLinks - pos;
    const uint32_t inner = h2[t], outer = h3[t];
    const float localEta = eta[t];
    // the count pass found exactly `limit` followers from runStart on
    for (uint32_t i = ls.runStart[t], cnt = 0; cnt < limit && i < nT; ++i) {
      if (h2[i] != outer || h1[i] != inner) {
        if (ls.sortedSegments) break;
        continue;
      }
      if (!(fabs_(localEta - eta[i]) < dEtaCut)) continue;
      ls.basis[pos + cnt] = t;
      ls.follower[pos + cnt] = i;
      const uint32_t p = ls.inStart[i] + atomicAdd(&ls.inCursor[i], 1u);
      if (p < ls.capLinks) ls.inList[p] = t;
      ++cnt;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const uint32_t nW = (nT + 31u) >> 5;
    ls.connSums[nW] = 0u;
    *ls.nWordsOut = nW;
  }
}

// TrackletCircleFitter.h:32-97
__device__ __forceinline__ float circle_radius(float4 a, float4 b, float4 c) {
  const f3 pP0 = make_f3(a.x, a.y, a.x * a.x + a.y * a.y);
  const f3 pP1 = make_f3(b.x, b.y, b.x * b.x + b.y * b.y);
  const f3 pP2 = make_f3(c.x, c.y, c.x * c.x + c.y * c.y);
  const f3 n3 = cross3(sub3(pP1, pP0), sub3(pP2, pP0));
  const f3 un = normalize3(n3);
  const float cc = -dot3(un, pP0);
  const float nz2 = un.z * un.z;
  return sqrt_(div_(1 - nz2 - 4 * cc * un.z, 4 * nz2));
}

// Every k < nT - 1 goes to one of the two lists: a connectable one to
// wordStart[k / 32] + (connectable bits below k in its word), a
// non-connectable one to k minus the connectable ones before it.
__device__ __forceinline__ void connectable_entry(uint32_t k, uint32_t nT, uint32_t w, const ConnLists& lists) {
  if (k + 1 >= nT) return;
  const uint32_t bit = k & 31u;
  const uint32_t rank = lists.wordStart[k >> 5] + (uint32_t)__popc(w & ((1u << bit) - 1u));
  if ((w >> bit) & 1u) lists.conn[rank] = k;
  else lists.nonConn[k - rank] = k;
}

__global__ void __launch_bounds__(256)
    connectable_kernel(Stamp stamp, const uint32_t* nTDev, const uint32_t* __restrict__ words, ConnLists lists) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  GRID_STRIDE(k, nT) connectable_entry(k, nT, words[k >> 5], lists);
}

// The circle fit over all triplets with the flags as they are, without the
// list and without clearing pt first: the reads stay in triplet order.
// LISTS: the connectable lists as well, for a captured chain: a launch less
// and the words read once (100 events of 200 tracks: 160.9 -> 157.6 us).
template <bool LISTS>
__global__ void __launch_bounds__(256)
    circle_fit_words_kernel(Stamp stamp, const float4* __restrict__ hits, const uint32_t* __restrict__ h1,
                            const uint32_t* __restrict__ h2, const uint32_t* __restrict__ h3, const uint32_t* nTDev,
                            const uint32_t* __restrict__ words, float* pt, ConnLists lists) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  GRID_STRIDE(k, nT) {
    const uint32_t w = words[k >> 5];
    if (LISTS) connectable_entry(k, nT, w, lists);
    pt[k] = (w >> (k & 31u)) & 1u ? circle_radius(hits[h1[k]], hits[h2[k]], hits[h3[k]]) : 0.0f;
  }
}

__global__ void circle_fit_kernel(Stamp stamp, const float4* __restrict__ hits, const uint32_t* __restrict__ h1,
                                  const uint32_t* __restrict__ h2, const uint32_t* __restrict__ h3,
                                  const uint32_t* __restrict__ conn, const uint32_t* nConnDev, float* pt) {
  stamp_begin(stamp);
  const uint32_t n = *nConnDev;
  GRID_STRIDE(j, n) {
    const uint32_t t = conn[j];
    pt[t] = circle_radius(hits[h1[t]], hits[h2[t]], hits[h3[t]]);
  }
}

__global__ void in_degree_kernel(Stamp stamp, const uint32_t* __restrict__ follower, const uint32_t* nLinksDev,
                                 uint32_t* inDeg) {
  stamp_begin(stamp);
  const uint32_t n = *nLinksDev;
  GRID_STRIDE(p, n) atomicAdd(&inDeg[follower[p]], 1u);
}

// The bases of each follower's incoming links.  Links are stored in basis
// order, so the bases of one follower (all distinct) sort like the link
// indices do.
__global__ void in_fill_kernel(Stamp stamp, const uint32_t* __restrict__ basis, const uint32_t* __restrict__ follower,
                               const uint32_t* nLinksDev, const uint32_t* __restrict__ inStart, uint32_t* cursor,
                               uint32_t* inList) {
  stamp_begin(stamp);
  const uint32_t n = *nLinksDev;
  GRID_STRIDE(p, n) {
    const uint32_t f = follower[p];
    inList[inStart[f] + atomicAdd(&cursor[f], 1u)] = basis[p];
  }
}

// the CA's per-triplet state before a run: states 1, no best basis, and
// (caller links) in-degrees and cursors 0
__global__ void ca_init_kernel(Stamp stamp, CABuffers b, const uint32_t* nTDev, bool degrees) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  GRID_STRIDE(i, nT + 1) {
    if (degrees) b.inStart[i] = 0u;
    if (i < nT) {
      if (degrees) b.inCursor[i] = 0u;
      b.states[i] = 1u;
      b.best[i] = TRAX_SENTINEL;
      b.isBest[i] = 0u;
    }
  }
}

// A run whose links overflowed their capacity or whose scans failed left
// lists half written: the CA does not follow them, and the call fails or
// recalibrates.
__device__ __forceinline__ bool ca_skip(const uint32_t* err) {
  return (*err & (TRAX_EBIT_CAPACITY | TRAX_EBIT_TIMEOUT | TRAX_EBIT_OVERFLOW)) != 0u;
}

// one above the highest incoming basis
__device__ __forceinline__ uint32_t ca_state(const uint32_t* inStart, const uint32_t* inList, const uint32_t* states,
                                             uint32_t t) {
  uint32_t m = 0;
  for (uint32_t j = inStart[t], b = inStart[t + 1]; j < b; ++j) m = max(m, states[inList[j]]);
  return m + 1u;
}

// One layer-triplet level of the forward phase.  SEGMENTS: the triplets of
// the level are the ranges of its segments, bpe blocks per event; otherwise
// (caller triplets, whose hits may mix events) all triplets are looked at.
template <bool SEGMENTS>
__global__ void ca_level_kernel(Stamp stamp, DevConfig cfg, uint32_t level, uint32_t bpe, CABuffers b,
                                const uint32_t* __restrict__ segStart, const uint32_t* nTDev) {
  stamp_begin(stamp);
  if (ca_skip(cfg.err)) return;
  if (SEGMENTS) {
    const uint32_t s = (blockIdx.x / bpe) * cfg.nLT + level, end = *nTDev ? segStart[s + 1] : 0u;
    for (uint32_t t = (end ? segStart[s] : 0u) + (blockIdx.x % bpe) * blockDim.x + threadIdx.x; t < end;
         t += bpe * blockDim.x)
      b.states[t] = ca_state(b.inStart, b.inList, b.states, t);
  } else {
    const uint32_t nT = *nTDev;
    GRID_STRIDE(t, nT) {
      if (b.segOf[t] % cfg.nLT != level || b.inStart[t] == b.inStart[t + 1]) continue;
      b.states[t] = ca_state(b.inStart, b.inList, b.states, t);
    }
  }
}

// The reference's forward iteration over any link set (`iteration`,
// CellularAutomaton.h:52-100): next[f] = max(next[f], cur[f] + (cur[b] ==
// cur[f])) for every link b -> f, and a living flag when a follower's state
// equals its basis's.  The host repeats it, swapping the buffers without
// copying (CellularAutomaton.cpp:52-98), until no cell lives.  Used for
// caller-provided links, which need not go from one layer triplet to the
// next as the chain's own do.
__global__ void ca_iteration_kernel(Stamp stamp, const uint32_t* __restrict__ basis,
                                    const uint32_t* __restrict__ follower, uint32_t nLinks,
                                    const uint32_t* __restrict__ cur, uint32_t* next, uint32_t* living) {
  stamp_begin(stamp);
  GRID_STRIDE(p, nLinks) {
    const uint32_t f = follower[p];
    const uint32_t fs = cur[f];
    const uint32_t same = cur[basis[p]] == fs ? 1u : 0u;
    atomicMax(&next[f], fs + same);
    if (same) *living = 1u;
  }
}

__global__ void fill_u32_kernel(Stamp stamp, uint32_t* p, uint32_t v, uint32_t n) {
  stamp_begin(stamp);
  GRID_STRIDE(i, n) p[i] = v;
}

// followerBestBasisStore semantics (CellularAutomaton.h:212-263) over the
// incoming bases in ascending order, which is the order of their links (an
// insertion sort first; lists are short)
__device__ __forceinline__ void ca_pick_best(const CABuffers& b, const float* pt, uint32_t t, uint32_t sf) {
  const uint32_t first = b.inStart[t], end = b.inStart[t + 1];
  for (uint32_t i = first + 1; i < end; ++i) {
    const uint32_t v = b.inList[i];
    uint32_t j = i;
    while (j > first && b.inList[j - 1] > v) {
      b.inList[j] = b.inList[j - 1];
      --j;
    }
    b.inList[j] = v;
  }
  if (first >= end) return;
  const float ptT = pt[t];
  bool have = false;
  float minPt = 0.0f;
  uint32_t minIdx = 0;
  for (uint32_t j = first; j < end; ++j) {
    const uint32_t bb = b.inList[j];
    if (b.states[bb] + 1 != sf) continue;
    const float d = fabs_(pt[bb] - ptT);
    if (!have) {
      minPt = d;
      minIdx = bb;
      have = true;
    } else {
      const uint32_t test = d < minPt;
      minPt = minPt * (float)(!test) + d * (float)test;
      minIdx = minIdx * (!test) + bb * test;
    }
  }
  if (have) {
    b.best[t] = minIdx;
    b.isBest[minIdx] = 1u;
  }
}

__global__ void ca_best_kernel(Stamp stamp, const float* pt, CABuffers b, const uint32_t* nTDev,
                               const uint32_t* err) {
  stamp_begin(stamp);
  if (ca_skip(err)) return;
  const uint32_t nT = *nTDev;
  GRID_STRIDE(t, nT) ca_pick_best(b, pt, t, b.states[t]);
}

// Both phases and the handlers of one event per CTA: the chain's links stay
// in their event and go to the next layer triplet, so the levels of an event
// need only block barriers between them.  One launch in place of an init, a
// launch per level, the best bases and the handlers.
__global__ void __launch_bounds__(1024)
    ca_event_kernel(Stamp stamp, DevConfig cfg, const float* pt, CABuffers b, const uint32_t* segStart,
                    const uint32_t* nTDev, const uint32_t* nLinksDev) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  if (blockIdx.x == 0 && threadIdx.x == 0) b.handlers[nT] = 0u;  // the scan's +1 slot
  if (nT == 0u || ca_skip(cfg.err)) return;
  const uint32_t s0 = blockIdx.x * cfg.nLT;
  const uint32_t t0 = segStart[s0], t1 = segStart[s0 + cfg.nLT];
  // A triplet's bases lie in earlier levels, so its state and its best basis
  // come out of one visit (the CA stage of 37 ttbar-like events took 39.5 us
  // with a pass of its own for the best bases, 35.0 us so; of 1000, 155 and
  // 146 us).  Taking a single basis without the general case gained nothing.
  for (uint32_t level = 0; level < cfg.nLT; ++level) {
    for (uint32_t t = segStart[s0 + level] + threadIdx.x, end = segStart[s0 + level + 1]; t < end; t += blockDim.x) {
      const uint32_t state = level ? ca_state(b.inStart, b.inList, b.states, t) : 1u;
      b.states[t] = state;
      b.best[t] = TRAX_SENTINEL;
      b.isBest[t] = 0u;
      if (level) ca_pick_best(b, pt, t, state);
    }
    __syncthreads();
  }
  const bool any = *nLinksDev != 0u;
  for (uint32_t t = t0 + threadIdx.x; t < t1; t += blockDim.x)
    b.handlers[t] = any ? (b.isBest[t] == 0u) * b.states[t] : 0u;
}

// handlersStateStore (CellularAutomaton.h:270-288); no tracks at all when
// there are no links (the reference skips the CA, TripletBuilder.cpp:414-421)
__global__ void handlers_kernel(Stamp stamp, const uint32_t* __restrict__ states, const uint32_t* __restrict__ isBest,
                                const uint32_t* nTDev, const uint32_t* nLinksDev, uint32_t* handlers) {
  stamp_begin(stamp);
  const uint32_t nT = *nTDev;
  const bool any = *nLinksDev != 0u;
  GRID_STRIDE(t, nT + 1) handlers[t] = (any && t < nT) ? (isBest[t] == 0u) * states[t] : 0u;
}

__global__ void tracks_kernel(Stamp stamp, const uint32_t* __restrict__ handlers, const uint32_t* __restrict__ best,
                              const uint32_t* nTDev, uint32_t* tracks, uint64_t maxTracks, uint32_t* err) {
  stamp_begin(stamp);
  if (ca_skip(err)) return;
  const uint32_t nT = *nTDev;
  GRID_STRIDE(t, nT) {
    const uint32_t off = handlers[t];
    const uint32_t len = handlers[t + 1] - off;
    uint32_t b = t;
    for (uint32_t i = 0; i < len && b != TRAX_SENTINEL; ++i) {
      if ((uint64_t)off + i >= maxTracks) {
        raise_error(err, TRAX_EBIT_CAPACITY);
        break;
      }
      tracks[off + i] = b;
      b = best[b];
    }
  }
}

}  // namespace

cudaError_t triplet_segments(const DevConfig& cfg, DevHits hits, TripletView t, uint32_t* segStart, uint32_t* segOf,
                             uint32_t* offsets, Queue& q) {
  if (t.maxN > 0)
    launch(q, triplet_segments_kernel, grid_for(t.maxN, 256), 256, 0, cfg, hits.evt, hits.layer, t.h1, t.nDev,
           segStart, segOf);
  launch(q, triplet_offsets_kernel, 1, OFF_THREADS, 0, cfg.E * cfg.nLT, t.nDev, segStart, offsets);
  return cudaGetLastError();
}

cudaError_t triplet_link_start(const DevConfig& cfg, DevHits hits, TripletView t, LinkStart link, Queue& q) {
  launch(q, link_start_kernel, grid_for(t.maxN + 1, 256), 256, 0, cfg, hits.xyzp, t.h1, t.h2, t.h3, t.nDev, link);
  return cudaGetLastError();
}

cudaError_t connectivity_count(const DevConfig& cfg, DevHits hits, TripletView t, const float* eta,
                               const uint32_t* offsets, const uint32_t* segStart, const uint2* runs,
                               uint32_t* linkCount, uint32_t* inDeg, uint32_t* runStart, bool sortedSegments,
                               Queue& q) {
  launch(q, conn_count_kernel, grid_for(t.maxN + 1, 256), 256, 0, cfg, hits.evt, hits.layer, t.h1, t.h2, t.h3, t.nDev,
         eta, offsets, segStart, runs, linkCount, inDeg, runStart, sortedSegments);
  return cudaGetLastError();
}

cudaError_t connectivity_store(const DevConfig& cfg, TripletView t, const float* eta, LinkStore ls, Queue& q) {
  launch(q, conn_store_kernel, grid_for(t.maxN + 1, 256), 256, 0, cfg, t.h1, t.h2, t.h3, t.nDev, eta, ls);
  return cudaGetLastError();
}

cudaError_t connectable_lists(TripletView t, const uint32_t* connWords, ConnLists lists, Queue& q) {
  if (t.maxN == 0) return cudaSuccess;
  launch(q, connectable_kernel, grid_for(t.maxN, 256), 256, 0, t.nDev, connWords, lists);
  return cudaGetLastError();
}

cudaError_t circle_fit_words(DevHits hits, TripletView t, const uint32_t* connWords, float* pt, const ConnLists* lists,
                             Queue& q) {
  if (t.maxN == 0) return cudaSuccess;
  launch(q, lists ? circle_fit_words_kernel<true> : circle_fit_words_kernel<false>, grid_for(t.maxN, 256), 256, 0,
         hits.xyzp, t.h1, t.h2, t.h3, t.nDev, connWords, pt, lists ? *lists : ConnLists{});
  return cudaGetLastError();
}

cudaError_t circle_fit(DevHits hits, TripletView t, const uint32_t* connectable, const uint32_t* nConnDev,
                       uint64_t maxConn, float* pt, Queue& q) {
  if (maxConn == 0) return cudaSuccess;
  launch(q, circle_fit_kernel, grid_for(maxConn, 256), 256, 0, hits.xyzp, t.h1, t.h2, t.h3, connectable, nConnDev,
         pt);
  return cudaGetLastError();
}

cudaError_t ca_in_degree(const uint32_t* follower, const uint32_t* nLinksDev, uint64_t maxLinks, CABuffers b,
                         const uint32_t* nTDev, uint64_t maxT, Queue& q) {
  launch(q, ca_init_kernel, grid_for(maxT + 1, 256), 256, 0, b, nTDev, true);
  if (maxLinks > 0) launch(q, in_degree_kernel, grid_for(maxLinks, 256), 256, 0, follower, nLinksDev, b.inStart);
  return cudaGetLastError();
}

cudaError_t ca_fill(const uint32_t* basis, const uint32_t* follower, const uint32_t* nLinksDev, uint64_t maxLinks,
                    CABuffers b, Queue& q) {
  if (maxLinks > 0)
    launch(q, in_fill_kernel, grid_for(maxLinks, 256), 256, 0, basis, follower, nLinksDev, b.inStart, b.inCursor,
           b.inList);
  return cudaGetLastError();
}

cudaError_t ca_chain(const DevConfig& cfg, const float* pt, CABuffers b, const uint32_t* segStart, bool perEvent,
                     const uint32_t* nTDev, uint64_t maxT, const uint32_t* nLinksDev, Queue& q) {
  if (perEvent) {
    const uint64_t mean = maxT / cfg.E;  // triplets of an event
    const unsigned threads = mean > 4096 ? 1024 : mean > 1024 ? 512 : mean > 256 ? 256 : 128;
    launch(q, ca_event_kernel, cfg.E, threads, 0, cfg, pt, b, segStart, nTDev, nLinksDev);
    return cudaGetLastError();
  }
  launch(q, ca_init_kernel, grid_for(maxT + 1, 256), 256, 0, b, nTDev, false);
  const uint64_t events = cfg.E ? cfg.E : 1;  // (a launch needs a block; without events it has no triplets)
  uint64_t bpe = maxT / (events * cfg.nLT * 256) + 1;
  const uint64_t most = (uint64_t)sm_count() * 16 / events + 1;
  if (bpe > most) bpe = most;
  for (uint32_t level = 1; level < cfg.nLT; ++level) {
    if (segStart)
      launch(q, ca_level_kernel<true>, (unsigned)(events * bpe), 256, 0, cfg, level, (uint32_t)bpe, b, segStart,
             nTDev);
    else
      launch(q, ca_level_kernel<false>, grid_for(maxT, 256), 256, 0, cfg, level, 1u, b, segStart, nTDev);
  }
  return ca_backward(pt, b, nTDev, maxT, nLinksDev, cfg.err, q);
}

cudaError_t ca_iteration(const uint32_t* basis, const uint32_t* follower, uint32_t nLinks, const uint32_t* cur,
                         uint32_t* next, uint32_t* living, Queue& q) {
  if (nLinks == 0) return cudaSuccess;
  launch(q, ca_iteration_kernel, grid_for(nLinks, 256), 256, 0, basis, follower, nLinks, cur, next, living);
  return cudaGetLastError();
}

cudaError_t fill_u32(uint32_t* p, uint32_t v, uint32_t n, Queue& q) {
  if (n == 0) return cudaSuccess;
  launch(q, fill_u32_kernel, grid_for(n, 256), 256, 0, p, v, n);
  return cudaGetLastError();
}

cudaError_t ca_backward(const float* pt, CABuffers b, const uint32_t* nTDev, uint64_t maxT,
                        const uint32_t* nLinksDev, const uint32_t* err, Queue& q) {
  launch(q, ca_best_kernel, grid_for(maxT, 256), 256, 0, pt, b, nTDev, err);
  launch(q, handlers_kernel, grid_for(maxT + 1, 256), 256, 0, b.states, b.isBest, nTDev, nLinksDev, b.handlers);
  return cudaGetLastError();
}

cudaError_t ca_tracks(CABuffers b, const uint32_t* nTDev, uint64_t maxT, uint32_t* tracks, uint64_t maxTracks,
                      uint32_t* err, Queue& q) {
  if (maxT == 0) return cudaSuccess;
  launch(q, tracks_kernel, grid_for(maxT, 256), 256, 0, b.handlers, b.best, nTDev, tracks, maxTracks, err);
  return cudaGetLastError();
}

}  // namespace trax
