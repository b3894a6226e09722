// SITE by locally dominant picks.
//
// Without intervis a candidate's area is its gain, which only falls, and only
// when a candidate within 2*roi of it is picked.  A candidate whose key (area <<
// 32 | ~index) exceeds those of all unused candidates within 2*roi is therefore
// picked by the sequential greedy before any of them, with the gain it has now:
// a neighbour could only be picked first with a larger key, and keys do not
// rise.  So every such candidate can be picked at once.  Keys of successive
// greedy picks fall, so the greedy's order is the picks by falling key; it ends at
// the first pick whose cumulative area passes the 95% stop, and the picks that a
// round took beyond that are dropped at the end.  All true picks are among those
// taken once the areas of the picks with keys above every remaining key reach
// the stop.  (Simulated on terrains of 1000^2 to 2048^2 and run on the GPU against
// the sequential order: 12-25 rounds, where the longest prefix of the global key
// order without a conflict takes 84-190.)
//
// With intervis a touched candidate (one within 2*roi of a pick) has area 0 until a
// pick covers its cell, so it can become eligible late with a large key.  The greedy
// takes it right after the pick that covered it if its key is then the largest.  So
// each candidate has a chain: itself, the pick that covered its cell, the pick that
// covered that one's, and so on.  Its level is the least key of its chain, and the
// greedy takes larger levels first.  Of two with the same level, the one whose least
// key is larger on its part of the chains up to where they meet comes first (the
// common part holds both back alike).  Dominance is by this order, and a dominant
// candidate c is kept only if no touched, uncovered neighbour with a key above
// c's level may be covered before c's turn: B2 searches back from these along "who
// sees whom", and c is put off when it meets an eligible candidate that comes before
// c.  The first candidate of all is always kept, so every round takes the greedy's
// next pick at least.
//
// Candidates are sorted into square bins of a quarter of roi, row-major, so a run of
// bins in a bin row is one range of the sorted arrays.  A round:
//   A. eight lanes a bin find its first candidate;
//   B. of each cell of 4x4 bins (any two of its candidates are within 2*roi) only
//      the first can be dominant: a warp compares it with the first ones of the
//      bins within 2*roi, and with the single candidates of those whose first comes
//      before it but is too far; dominant ones of at least half the largest level's
//      area are this round's picks (below that, a pick may well lie beyond the stop);
//   B2. (intervis) the searches: a warp looks at one candidate of a search's queue at a
//      time.  The CTAs left over share searches of 2 to 16 CTAs through global memory
//      (a single CTA's warps took 0.2 ms a round on the longest searches, 500
//      candidates deep: 1600^2, radius 98, 40 000 candidates 3.8 -> 2.3 ms); with more
//      dominant candidates than half the CTAs each search stays in a CTA's shared memory;
//   C. the rows of the picks' new bits N = placed(shed) & ~coverage, spread over
//      all threads;
//   D. |V_u n N| for each (pick, unused candidate u within 2*roi): the candidates
//      in the picks' bin ranges are split evenly over the CTAs; a CTA lists its
//      pairs, copies the one or two picks' N that it needs to shared memory, and its
//      warps count a pair at a time, consecutive lanes on consecutive words.  Picks
//      are more than 2*roi apart, so their new bits are disjoint and the gains'
//      decreases add up.
// Four group barriers a round, five with intervis.  A round is bound by the latency of
// its dependent L2 reads and of the barriers (4096^2, radius 100, intervis: 120 us, of
// which B2 takes half and D a third; start to end 348 rounds and 6.7 ms in the global
// order, 33 rounds and 4.0 ms here); only at 16384^2 does D's reading of sheds count.
#pragma once

#include "common.cuh"

namespace siting {
namespace {

constexpr int kLocalMaxBins = 256;   // bins a side at most
constexpr int kLocalMaxPicks = 256;  // picks of a round at most
constexpr int kLocalRanges = 20;     // bin rows a pick's candidates can span (4*roi+1 cells and a margin)
constexpr int kLocalCell = 4;        // bins a side of a cell of B
constexpr int kLocalTodo = 128;
// A search of B2 in global memory: a hash table of the candidates met, the queue of
// those to look at, and {tail, CTAs that have queued their starts, done}, {head}.
constexpr int kLocalSeenLog = 11, kLocalProbes = 32;  // places in the table (log2), probes at most
constexpr int kLocalQueue = 1024;
constexpr int kLocalSearch = (1 << kLocalSeenLog) + kLocalQueue + 64;  // words
// CTAs of a search: one, in its shared memory, or from so many to so many.
constexpr int kLocalShareMin = 2, kLocalShare = 16;
constexpr int kLocalStride = 7919;   // order of a pick's candidates
constexpr int kLocalLook = 12;       // 32s of bins within reach: at most 19 a side
// Picks whose order is found by comparing each with all in shared memory, without and with
// intervis, and buckets for more of them (thousand cycles so and by buckets: 4500 picks of
// 2458^2, radius 26, without 76, 180; 2500 of 4096^2, radius 100, with 460, 50; 16384
// buckets 152 and 122, for their sums).
constexpr int kLocalDirect = 8192, kLocalDirectChains = 1024, kLocalBuckets = 4096;

// Bins: side (cells of the DEM) and count a side.
__host__ __device__ __forceinline__ int local_bin_side(int n, int roi) {
  const int least = (n + kLocalMaxBins - 1) / kLocalMaxBins, quarter = (roi + 3) / 4;
  return quarter > least ? quarter : least;
}
__host__ __device__ __forceinline__ int local_bins(int n, int roi) {
  const int s = local_bin_side(n, roi);
  return (n + s - 1) / s;
}
// Cells of B a side.
__host__ __device__ __forceinline__ int local_cells(int n, int roi) {
  return (local_bins(n, roi) + kLocalCell - 1) / kLocalCell;
}
// Whether a placed row of a window has a lane of a warp for each word (radius <= 992).
__host__ __device__ __forceinline__ bool local_width(int roi) { return (2 * roi + 64) / 64 + 1 <= 32; }
// Picks a round takes at most: 256 while their new bits take at most 8 MB (radius 227),
// 128 while these do (radius 340), else 64.
__host__ __device__ __forceinline__ int local_cap(int roi) {
  const size_t nr = 2 * (size_t)roi + 1, one = nr * ((nr + 63) / 64 + 1) * 8;
  return kLocalMaxPicks * one <= (size_t)8 << 20   ? kLocalMaxPicks
         : kLocalMaxPicks / 2 * one <= (size_t)8 << 20 ? kLocalMaxPicks / 2
                                                       : kLocalMaxPicks / 4;
}

// Shared memory of a CTA, sized for the largest job; the picks' new bits follow.
struct LocalShared {
  int at[kLocalMaxPicks], cand[kLocalMaxPicks], pos[kLocalMaxPicks], area[kLocalMaxPicks];
  int parent[kLocalMaxPicks], order[kLocalMaxPicks];
  unsigned long long reach[kLocalMaxPicks];
  int range0[kLocalMaxPicks * kLocalRanges];        // range starts in the sorted arrays
  int prefix[kLocalMaxPicks * kLocalRanges + 4];    // candidates before each range
  int pair_at[1024], pair_cand[1024], pair_pos[1024], pair_pick[1024];
  uint16_t todo[32][kLocalTodo];  // a warp's bins to look into
  unsigned long long red[32];
  unsigned long long total;
  int flag, n, next, first, last;
};

__device__ __forceinline__ unsigned long long local_key(int area, int c) {
  return ((unsigned long long)(unsigned)area << 32) |
         (unsigned long long)(0xFFFFFFFFu - (unsigned)c);
}

__device__ __forceinline__ unsigned long long warp_max64(unsigned long long key) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

__device__ __forceinline__ int row_of(int p) { return (int)((unsigned)p >> 16); }

__device__ __forceinline__ bool within(int p, int q, int lim2) {
  const int dx = row_of(p) - row_of(q), dy = (p & 0xffff) - (q & 0xffff);
  return dx * dx + dy * dy <= lim2;
}

// A sorted candidate: {cell, gain (0: used), index, flags}; flags: 1 touched (a pick
// lies within 2*roi; the area is then 0 unless the cell is covered), 2 covered, and
// from bit 2 on the pick that covered the cell, as its place in the list of picks.
__device__ __forceinline__ bool eligible(const int4 &c) { return c.y > 0 && (c.w & 3) != 1; }

// The level of an eligible candidate: the least key on its chain of picks, each the
// one that covered the next one's cell, and the candidate itself.
__device__ __forceinline__ unsigned long long local_level(const LocalScratch &L, const int4 &c) {
  const unsigned long long key = local_key(c.y, c.z);
  if (!(c.w & 2)) return key;
  const unsigned long long r = __ldcg(L.preach + (c.w >> 2));
  return r < key ? r : key;
}

// Whether the candidate or pick with key ky and last covering pick py comes before
// the one with kx, px in the greedy's order, their levels being equal: the larger of
// the least keys on the two chains up to where they meet.
__device__ __forceinline__ bool chain_before(const unsigned long long *plist, const int *pparent,
                                             unsigned long long ky, int py, unsigned long long kx,
                                             int px) {
  while (px != py) {  // a pick is in the list after the one that covered it
    if (px > py) {
      const unsigned long long q = __ldcg(plist + px);
      kx = q < kx ? q : kx;
      px = __ldcg(pparent + px);
    } else {
      const unsigned long long q = __ldcg(plist + py);
      ky = q < ky ? q : ky;
      py = __ldcg(pparent + py);
    }
  }
  return ky > kx;
}
__device__ __forceinline__ int parent_of(const int4 &c) { return (c.w & 2) ? c.w >> 2 : -1; }
// Whether the eligible candidate y of level ly comes before x of level lx.
__device__ __forceinline__ bool local_before(const LocalScratch &L, const int4 &y,
                                             unsigned long long ly, const int4 &x,
                                             unsigned long long lx) {
  if (ly != lx) return ly > lx;
  if (y.z == x.z) return false;
  return chain_before(L.plist, L.pparent, local_key(y.y, y.z), parent_of(y), local_key(x.y, x.z),
                      parent_of(x));
}

// Sum over the CTA (every thread gets it).
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v,
                                                        unsigned long long *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  unsigned long long s = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w];
  return s;
}

// |placed(shed of u) n N_p| over the rows and words that the two windows share, by
// one warp, consecutive lanes on consecutive words (a lane a row reads each line
// of the shed once a word: 2.8 times the wavefronts); kShared: N_p in shared memory.
// The windows share at most 32 words of a row (local_width).
template <bool kShared>
__device__ __forceinline__ int local_pair(const uint64_t *shed, const uint64_t *nbits, int n, int cw,
                                          int roi, int cpos, int ppos, int lane) {
  const int nr = 2 * roi + 1, nwpr = (nr + 63) / 64, nb2 = nwpr + 1;
  const int cx = row_of(cpos), cy = cpos & 0xffff, px = row_of(ppos), py = ppos & 0xffff;
  // rows of u's shed inside the pick's window and the DEM, words of the row in both
  const int r0 = max(max(0, px - cx), roi - cx);
  const int r1 = min(min(nr - 1, px - cx + 2 * roi), n - 1 - cx + roi);
  const int fwc = (cy - roi) >> 6, fbc = (cy - roi) & 63, fwp = (py - roi) >> 6;
  const int lo = max(max(fwc, fwp), 0), hi = min(min((cy + roi) >> 6, fwp + nwpr), cw - 1);
  const int nw = hi - lo + 1, total = nw > 0 ? max(0, r1 - r0 + 1) * nw : 0;
  if (total == 0) return 0;
  // A lane keeps its word of the row and takes every `rows`-th row.  u's word uq
  // reaches the placed words uq and uq+1.
  const int rows = 32 / nw, lr = lane / nw, q = lane - lr * nw;
  const int uq = lo - fwc + q;
  const bool has_cur = uq < nwpr, has_prev = fbc && uq > 0;
  const uint64_t *crow = shed + (size_t)(r0 + lr) * nwpr + uq;
  const uint64_t *nrow = nbits + (size_t)(cx - px + r0 + lr) * nb2 + (lo - fwp + q);
  const int cstep = rows * nwpr, nstep = rows * nb2;
  int d = 0;
  for (int left = lr < rows ? r1 - r0 - lr : -1; left >= 0; left -= 4 * rows) {
    uint64_t x[4], cur[4], prev[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      x[i] = 0ull;
      if (left >= i * rows) x[i] = kShared ? nrow[i * nstep] : __ldcg(nrow + i * nstep);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {  // nothing of u is read where the pick adds nothing
      cur[i] = x[i] && has_cur ? __ldg(crow + i * cstep) : 0ull;
      prev[i] = x[i] && has_prev ? __ldg(crow + i * cstep - 1) : 0ull;
    }
    crow += 4 * cstep;
    nrow += 4 * nstep;
#pragma unroll
    for (int i = 0; i < 4; i++)
      d += __popcll(((cur[i] >> fbc) | (prev[i] << ((64 - fbc) & 63))) & x[i]);
  }
  return __reduce_add_sync(0xffffffffu, d);
}

// Takes the pairs of the CTA's list, a warp one at a time.
template <bool kShared>
__device__ __forceinline__ void local_pairs(const SiteArgs &a, LocalShared &s, const uint64_t *N,
                                            int first, int cw, int lane) {
  const int nr = 2 * a.roi + 1, nwpr = (nr + 63) / 64;
  const size_t per = (size_t)nr * nwpr, nper = (size_t)nr * (nwpr + 1);
  for (;;) {
    int j = 0;
    if (lane == 0) j = atomicAdd(&s.next, 1);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= s.n) break;
    const int p = s.pair_pick[j];
    const int d = local_pair<kShared>(a.sheds + (size_t)s.pair_cand[j] * per,
                                      N + (size_t)(p - first) * nper, a.n, cw, a.roi,
                                      s.pair_pos[j], s.pos[p], lane);
    if (d && lane == 0) atomicSub(&a.local.rec[s.pair_at[j]].y, d);
  }
}

// The candidates of 32*I bins about (x, y), from the `from`-th of the square on, whose
// bin reaches into radius r and has its largest key at `level` or above: the t-th of
// them is start[q] + t, q the last with before[q] <= t.  By one warp; returns how many.
template <int I>
__device__ __forceinline__ int local_list(const SiteArgs &a, int *start, int *before, int x, int y,
                                          int r, int from, unsigned long long level, int side,
                                          int nbin, int lane) {
  const LocalScratch &L = a.local;
  const int x0 = max(0, x - r) / side, y0 = max(0, y - r) / side;
  const int w = min(a.n - 1, y + r) / side - y0 + 1;
  const int cnt = (min(a.n - 1, x + r) / side - x0 + 1) * w;
  int i0[I], len[I], sum = 0;
  unsigned long long cap[I];
#pragma unroll
  for (int i = 0; i < I; i++) {
    const int j = from + lane * I + i, jx = x0 + j / w, jy = y0 + j % w;
    const int ex = max(0, max(jx * side - x, x - (jx * side + side - 1)));
    const int ey = max(0, max(jy * side - y, y - (jy * side + side - 1)));
    const bool in = j < cnt && ex * ex + ey * ey <= r * r;
    const int o = jx * nbin + jy;
    cap[i] = in ? __ldcg(L.bincap + o) : 0ull;
    i0[i] = in ? (int)__ldcg(L.count + o) : 0;
    len[i] = in ? (int)__ldcg(L.count + o + 1) - i0[i] : 0;
  }
#pragma unroll
  for (int i = 0; i < I; i++) {
    if (cap[i] < level) len[i] = 0;
    sum += len[i];
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int run = incl - sum;
#pragma unroll
  for (int i = 0; i < I; i++) {
    start[lane * I + i] = i0[i] - run;
    before[lane * I + i] = run;
    run += len[i];
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, incl, 31);
}
template <int I>
__device__ __forceinline__ int local_nth(const int *start, const int *before, int t) {
  int lo = 0, hi = 32 * I - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (before[mid] <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  return start[lo] + t;
}

// B2: whether a candidate near the dominant candidate c = {place, index, cell, area}
// may become eligible and be picked before it.  Such a candidate is touched and
// uncovered, its gain key is above c's level, and a pick before c covers it, that is
// a candidate that sees it: one that is eligible now and comes before c, or one of the
// same kind.  The search goes back along such chains from c's neighbours until it
// meets an eligible candidate before c, or ends.  c's neighbours themselves need no
// step among one another: the eligible ones come after c and the others are all
// starts, so a start within roi of c has none to look at.  By `parts` CTAs together:
// this one takes every parts-th start from `part` on and what it meets first; `seen`
// is their table of what was met, *bad their result.
template <bool kShared>
__device__ __noinline__ void local_threat(const SiteArgs &a, LocalShared &s, unsigned *search,
                                          int *bad, int4 c, int side, int nbin, int part,
                                          int parts) {
  const LocalScratch &L = a.local;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int roi = a.roi, nr = 2 * roi + 1, nwpr = (nr + 63) / 64;
  const size_t per = (size_t)nr * nwpr;
  const int4 me = __ldcg(L.rec + c.x);
  const unsigned long long level = local_level(L, me);
  const int lim2 = 4 * roi * roi;
  unsigned *seen = search, *queue = seen + (1 << kLocalSeenLog), *tail = queue + kLocalQueue;
  unsigned *ready = tail + 1, *fin = tail + 2, *head = tail + 32;
  int *start = s.range0 + warp * 128, *before = s.prefix + warp * 128;
  auto get = [&](const unsigned *p) {
    return kShared ? *(const volatile unsigned *)p : ld_acquire_u32(p);
  };
  auto put = [&](unsigned *p, unsigned v) {
    if (kShared)
      *(volatile unsigned *)p = v;
    else
      __stcg(p, v);
  };
  if (kShared) {
    for (int i = tid; i < kLocalSearch; i += blockDim.x) search[i] = 0u;
    __syncthreads();
  }
  auto hash = [&](int i) { return ((unsigned)i * 2654435761u) >> (32 - kLocalSeenLog); };
  auto push = [&](int i) {
    const unsigned j = atomicAdd(tail, 1u);
    if (j < (unsigned)kLocalQueue)
      put(queue + j, (unsigned)i + 1u);
    else
      __stcg(bad, 1);  // too many to search: not this round
  };
  auto first = [&](int i) {  // whether no warp has met i before
    for (unsigned p = 0, h = hash(i); p < (unsigned)kLocalProbes; p++) {
      const unsigned old =
          atomicCAS(seen + ((h + p) & ((1u << kLocalSeenLog) - 1u)), 0u, (unsigned)i + 1u);
      if (old == 0u) return true;
      if (old == (unsigned)i + 1u) return false;
    }
    __stcg(bad, 1);  // nor with a full table
    return false;
  };
  {
    const int x = row_of(c.z), y = c.z & 0xffff;
    for (int from = warp * 32; from < kLocalLook * 32; from += nwarps * 32) {
      const int total = local_list<1>(a, start, before, x, y, 2 * roi, from, level, side, nbin, lane);
      for (int t0 = lane; t0 < total; t0 += 128) {
        int4 u[4];
        int at[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          at[j] = local_nth<1>(start, before, min(t0 + 32 * j, total - 1));
          u[j] = __ldcg(L.rec + at[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (t0 + 32 * j < total && u[j].y > 0 && !eligible(u[j]) &&
              local_key(u[j].y, u[j].z) > level && within(u[j].x, c.z, lim2) &&
              !within(u[j].x, c.z, roi * roi) && at[j] % parts == part)
            push(at[j]);
      }
      __syncwarp();
    }
  }
  if (!kShared) __threadfence();
  __syncthreads();
  if (tid == 0) atomicAdd(ready, 1u);
  for (;;) {
    // the next of the queue; none when every start is queued and all that was queued is done
    int u = -1;
    if (lane == 0) {
      const unsigned h = atomicAdd(head, 1u);
      const long long t0 = clock64();
      while (h < (unsigned)kLocalQueue) {
        const unsigned v = kShared ? get(queue + h) : __ldcg(queue + h);
        if (*(volatile int *)bad) break;
        if (v) {
          u = (int)v - 1;
          break;
        }
        if (get(ready) == (unsigned)parts) {
          const unsigned done = get(fin);
          if (done == get(tail)) break;
        }
        if (clock64() - t0 > kWaitCycles) {
          atomicOr(a.err, kErrBarrierTimeout);
          __stcg(bad, 1);
          break;
        }
      }
    }
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u < 0) break;
    const int upos = __ldcg(&L.rec[u].x);
    const int x = row_of(upos), y = upos & 0xffff;
    // 10 x 10 bins at most
    const int total = local_list<4>(a, start, before, x, y, roi, 0, level, side, nbin, lane);
    bool pushed = false;
    for (int t0 = lane; t0 < total; t0 += 128) {  // four candidates a lane, loads together
      int4 p[4];
      int at[4];
      uint64_t w[4], more[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        at[j] = local_nth<4>(start, before, min(t0 + 32 * j, total - 1));
        p[j] = __ldcg(L.rec + at[j]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        // outside c's neighbourhood, above c's level, sees u
        const bool look = t0 + 32 * j < total && p[j].y > 0 &&
                          local_key(p[j].y, p[j].z) > level && within(p[j].x, upos, roi * roi) &&
                          !within(p[j].x, c.z, lim2);
        const int row = x - row_of(p[j].x) + roi, col = y - (p[j].x & 0xffff) + roi;
        w[j] = 0ull;
        more[j] = ~0ull;
        if (look) {
          w[j] = __ldg(a.sheds + (size_t)p[j].z * per + (size_t)row * nwpr + (col >> 6)) >>
                     (63 - (col & 63)) & 1ull;
          if (!eligible(p[j]))
            more[j] = kShared ? get(seen + hash(at[j])) : __ldcg(seen + hash(at[j]));
          else if (p[j].w & 2)
            more[j] = __ldcg(L.preach + (p[j].w >> 2));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!w[j]) continue;
        if (!eligible(p[j])) {
          if (more[j] != (uint64_t)at[j] + 1ull && first(at[j])) {
            push(at[j]);
            pushed = true;
          }
        } else if (more[j] >= level &&
                   local_before(L, p[j], min((unsigned long long)more[j], local_key(p[j].y, p[j].z)),
                                me, level)) {
          __stcg(bad, 1);
        }
      }
    }
    if (pushed) kShared ? __threadfence_block() : __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(fin, 1u);
  }
  __syncthreads();
}

// The order of many picks: they are sorted into buckets of falling levels, and each is
// compared with its bucket's.  (All with all, 454 712 picks of 12000^2, radius 5, took
// 291 ms of 525 with intervis, 75 of 155 without.)  The bins' and the candidates' scratch
// is free by then.
template <class Place>
__device__ __forceinline__ void local_order(const SiteArgs &a, LocalShared &s, GroupBarrier &gb, int k,
                                            int np, Place place) {
  const LocalScratch &L = a.local;
  const int G = a.G, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
  const int gtid = k * T + tid, gthreads = G * T;
  const bool iv = a.intervis;
  const int nbin = local_bins(a.n, a.roi), B = min(nbin * nbin, kLocalBuckets);
  const unsigned long long *reach = iv ? L.preach : L.plist;
  unsigned long long *sum = L.binkey, *base = reinterpret_cast<unsigned long long *>(L.binat);
  unsigned *fill = L.fill;
  ulonglong2 *sorted = reinterpret_cast<ulonglong2 *>(L.rec);  // {level, key}
  int *which = const_cast<int *>(a.gains);                     // the pick
  // a level's bucket: by area, and by index where there are buckets to spare
  const unsigned span = (unsigned)((2 * a.roi + 1) * (2 * a.roi + 1)) + 1u;
  const unsigned spare = (unsigned)B / span;
  auto bucket = [&](unsigned long long level) {
    const unsigned ar = min((unsigned)(level >> 32), span - 1u), c = 0xFFFFFFFFu - (unsigned)level;
    const unsigned v = spare ? ar * spare + spare - 1u -
                                   (unsigned)((unsigned long long)c * spare / (unsigned)a.nsheds)
                             : (unsigned)((unsigned long long)ar * (unsigned)B / span);
    return B - 1 - (int)v;
  };
  for (int b = gtid; b < B; b += gthreads) {
    __stcg(sum + b, 0ull);
    __stcg(fill + b, 0u);
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
  for (int x = gtid; x < np; x += gthreads)  // picks and their areas
    atomicAdd(sum + bucket(__ldcg(reach + x)), 1ull << 32 | __ldcg(L.plist + x) >> 32);
  if (!group_sync(gb, a.err, &s.flag)) return;
  if (k == 0) {
    const int each = (B + T - 1) / T, b0 = min(tid * each, B), b1 = min(b0 + each, B);
    unsigned long long mine = 0;
    for (int b = b0; b < b1; b++) mine += __ldcg(sum + b);
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s.red[warp] = incl;
    __syncthreads();
    unsigned long long run = incl - mine;
    for (int w = 0; w < warp; w++) run += s.red[w];
    for (int b = b0; b < b1; b++) {
      __stcg(base + b, run);
      run += __ldcg(sum + b);
    }
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
  for (int x = gtid; x < np; x += gthreads) {
    const unsigned long long r = __ldcg(reach + x);
    const int b = bucket(r);
    const unsigned at = (unsigned)(__ldcg(base + b) >> 32) + atomicAdd(fill + b, 1u);
    __stcg(sorted + at, make_ulonglong2(r, __ldcg(L.plist + x)));
    __stcg(which + at, x);
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
  for (int i = gtid; i < np; i += gthreads) {
    const ulonglong2 me = sorted[i];
    const int x = which[i], b = bucket(me.x);
    const unsigned long long first = __ldcg(base + b);
    const int y0 = (int)(first >> 32), y1 = y0 + (int)(__ldcg(sum + b) >> 32);
    unsigned above = (unsigned)y0, before = (unsigned)first;
    int same = 0;
#pragma unroll 8
    for (int j = y0; j < y1; j++) {
      const ulonglong2 o = sorted[j];
      above += o.x > me.x;
      before += o.x > me.x ? (unsigned)(o.y >> 32) : 0u;
      same += o.x == me.x;
    }
    for (int j = y0; same > 1 && j < y1; j++) {  // of one level (intervis): by their chains
      const ulonglong2 o = sorted[j];
      if (o.x != me.x || j == i) continue;
      same--;
      if (chain_before(L.plist, L.pparent, ~0ull, which[j], ~0ull, x)) {
        above++;
        before += (unsigned)(o.y >> 32);
      }
    }
    place(above, before, me.y);
  }
}

// The bin of a cell, and the cell as row and column.
__device__ __forceinline__ int local_bin_of(int cell, int n, int side, int nbin, int *pos) {
  const int x = cell / n, y = cell - x * n;
  *pos = (int)((unsigned)x << 16) | y;
  return (x / side) * nbin + y / side;
}

// The whole selection of one job by the G CTAs of its group; k is this CTA's
// place in it.
__device__ __forceinline__ void site_local(const SiteArgs &a, LocalShared &s, int k,
                                           long long *phase, long long *tmark) {
  const LocalScratch &L = a.local;
  const int G = a.G, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = blockDim.x, nwarps = T >> 5;
  const int gtid = k * T + tid, gthreads = G * T;
  const int gwarp = warp * G + k, gwarps = nwarps * G;  // a CTA's warps far apart in work order
  const int n = a.n, roi = a.roi, nr = 2 * roi + 1, nwpr = (nr + 63) / 64, nb2 = nwpr + 1;
  const int cw = (n + 63) / 64, lim2 = 4 * roi * roi;
  const size_t per = (size_t)nr * nwpr;
  const int side = local_bin_side(n, roi), nbin = local_bins(n, roi), nbins = nbin * nbin;
  const int cap = local_cap(roi);
  uint64_t *N = reinterpret_cast<uint64_t *>(&s + 1);
  const bool iv = a.intervis;
  GroupBarrier gb{a.bar, (unsigned)G, 0u};
  auto mark = [&](int i) {
    if (k == 0 && tid == 0) {
      const long long now = clock64();
      phase[i] += now - *tmark;
      *tmark = now;
    }
  };

  // ---- candidates into bins (counted with the round-1 gains) ---------------------------
  if (k == 0) {  // exclusive prefix sums, in place
    const int each = (nbins + T - 1) / T, b0 = min(tid * each, nbins), b1 = min(b0 + each, nbins);
    unsigned sum = 0;
    for (int b = b0; b < b1; b++) sum += __ldcg(L.count + b);
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s.red[warp] = incl;
    __syncthreads();
    unsigned run = incl - sum;
    for (int w = 0; w < warp; w++) run += (unsigned)s.red[w];
    for (int b = b0; b < b1; b++) {
      const unsigned v = __ldcg(L.count + b);
      __stcg(L.count + b, run);
      run += v;
    }
    if (tid == 0) __stcg(L.count + nbins, (unsigned)a.nsheds);
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
  for (int c = gtid; c < a.nsheds; c += gthreads) {
    int pos;
    const int b = local_bin_of(__ldg(a.obs + c), n, side, nbin, &pos);
    const unsigned at = __ldcg(L.count + b) + atomicAdd(L.fill + b, 1u);
    __stcg(L.rec + at, make_int4(pos, __ldcg(a.gains + c), c, 0));
  }
  if (tid == 0) s.total = 0;
  if (iv)
    for (int i = gtid; i < G * kLocalSearch; i += gthreads) __stcg(L.search + i, 0u);
  if (!group_sync(gb, a.err, &s.flag)) return;
  mark(0);

  uint64_t *cum = a.cum0;
  int rounds = 0, np = 0;
  for (;; rounds++) {
    const int par = rounds & 1;
    // ---- A. the largest key of each bin --------------------------------------------
    if (k == 0 && tid == 0 && rounds) {
      __stcg(L.npick + (par ^ 1), 0u);
      __stcg(L.ndom + (par ^ 1), 0u);
    }
    unsigned long long mine = 0;
    for (int b0 = gwarp * 4; b0 < nbins; b0 += gwarps * 4) {
      const int b = b0 + (lane >> 3);
      const int i0 = b < nbins ? (int)__ldcg(L.count + b) : 0;
      const int i1 = b < nbins ? (int)__ldcg(L.count + b + 1) : 0;
      unsigned long long best = 0, other = 0;
      int at = -1;
      int4 top = make_int4(0, 0, -1, 0);
      for (int i = i0 + (lane & 7); i < i1; i += 8) {
        const int4 c = __ldcg(L.rec + i);
        if (!eligible(c)) {
          if (c.y > 0) other = max(other, local_key(c.y, c.z));
          continue;
        }
        const unsigned long long level = local_level(L, c);
        if (at < 0 || local_before(L, c, level, top, best)) {
          best = level;
          at = i;
          top = c;
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        other = max(other, __shfl_xor_sync(0xffffffffu, other, o));
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
        int4 t2;
        t2.x = __shfl_xor_sync(0xffffffffu, top.x, o);
        t2.y = __shfl_xor_sync(0xffffffffu, top.y, o);
        t2.z = __shfl_xor_sync(0xffffffffu, top.z, o);
        t2.w = __shfl_xor_sync(0xffffffffu, top.w, o);
        if (a2 >= 0 && (at < 0 || local_before(L, t2, l2, top, best))) {
          best = l2;
          at = a2;
          top = t2;
        }
      }
      if ((lane & 7) == 0 && b < nbins) {
        __stcg(L.binkey + b, best);
        if (iv) __stcg(L.bincap + b, max(best, other));
        __stcg(L.binat + b, make_int2(at, top.x));
      }
      mine = best > mine ? best : mine;
    }
    mine = warp_max64(mine);
    __syncthreads();
    if (lane == 0) s.red[warp] = mine;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < nwarps; w++) mine = s.red[w] > mine ? s.red[w] : mine;
      if (mine) atomicMax(L.gmax + par, mine);
    }
    mark(1);
    if (!group_sync(gb, a.err, &s.flag)) return;
    mark(2);
    // ---- the end: no area left, or every pick before the stop is taken ------------
    const unsigned long long M = __ldcg(L.gmax + par);
    if (M == 0) break;
    if ((long long)s.total >= a.stop_area) {
      unsigned long long above = 0;
      for (int i = tid; i < np; i += T) {
        if (__ldcg((iv ? L.preach : L.plist) + i) > M) above += __ldcg(L.plist + i) >> 32;
      }
      if ((long long)block_sum(above, s.red) >= a.stop_area) break;
    }
    // ---- B. dominant candidates -----------------------------------------------------
    if (k == 0)
      for (int i = tid; i < cap; i += T) {
        __stcg(L.ncount + (par ^ 1) * cap + i, 0);
      }
    const int ncell = local_cells(n, roi);
    if (iv)
      for (int i = gtid; i < ncell * ncell; i += gthreads)
        __stcg(L.bad + (par ^ 1) * ncell * ncell + i, 0);
    const unsigned least = (unsigned)((M >> 32) + 1) / 2;
    for (int cell = gwarp; cell < ncell * ncell; cell += gwarps) {
      const int bx = cell / ncell * kLocalCell, by = cell % ncell * kLocalCell;
      unsigned long long key = 0;
      int2 at = make_int2(0, 0);
      if (lane < kLocalCell * kLocalCell) {
        const int jx = bx + lane / kLocalCell, jy = by + lane % kLocalCell;
        if (jx < nbin && jy < nbin) {
          key = __ldcg(L.binkey + jx * nbin + jy);
          at = __ldcg(L.binat + jx * nbin + jy);
        }
      }
      const unsigned long long mx = warp_max64(key);
      if ((unsigned)(mx >> 32) < least || mx == 0) continue;
      unsigned ties = __ballot_sync(0xffffffffu, key == mx && lane < kLocalCell * kLocalCell);
      int from = __ffs(ties) - 1;
      int4 me = __ldcg(L.rec + __shfl_sync(0xffffffffu, at.x, from));
      for (ties &= ties - 1; ties; ties &= ties - 1) {  // equal levels: by their chains
        const int f2 = __ffs(ties) - 1;
        const int4 c2 = __ldcg(L.rec + __shfl_sync(0xffffffffu, at.x, f2));
        if (local_before(L, c2, mx, me, mx)) {
          me = c2;
          from = f2;
        }
      }
      at.x = __shfl_sync(0xffffffffu, at.x, from);
      at.y = __shfl_sync(0xffffffffu, at.y, from);
      const int pos = at.y, x = row_of(pos), y = pos & 0xffff;
      const int x0 = max(0, x - 2 * roi) / side, x1 = min(n - 1, x + 2 * roi) / side;
      const int y0 = max(0, y - 2 * roi) / side, y1 = min(n - 1, y + 2 * roi) / side;
      const int w = y1 - y0 + 1, cnt = (x1 - x0 + 1) * w;
      // the bins whose largest is larger (all loads in flight together), and
      // whether one of these is near
      unsigned larger = 0;
      bool hit = false;
#pragma unroll
      for (int i = 0; i < kLocalLook; i++) {
        const int j = lane + 32 * i;
        const int o = (x0 + j / w) * nbin + y0 + j % w;
        const int bx0 = (x0 + j / w) * side, by0 = (y0 + j % w) * side;
        const int ex = max(0, max(bx0 - x, x - (bx0 + side - 1)));
        const int ey = max(0, max(by0 - y, y - (by0 + side - 1)));
        if (j < cnt && ex * ex + ey * ey <= lim2 && __ldcg(L.binkey + o) >= mx) larger |= 1u << i;
      }
#pragma unroll
      for (int i = 0; i < kLocalLook; i++) {
        const int j = lane + 32 * i;
        const int o = (x0 + j / w) * nbin + y0 + j % w;
        if ((larger >> i) & 1u) {
          const int2 first = __ldcg(L.binat + o);
          if (__ldcg(L.binkey + o) == mx && !local_before(L, __ldcg(L.rec + first.x), mx, me, mx))
            larger &= ~(1u << i);  // nor does any other of the bin
          else
            hit |= within(first.y, pos, lim2);
        }
      }
      bool blocked = __any_sync(0xffffffffu, hit);
      // their other candidates: four bins at a time, eight lanes a bin
      if (!blocked) {
        uint16_t *todo = s.todo[warp];
        int nt = 0;
#pragma unroll
        for (int i = 0; i < kLocalLook; i++) {
          const unsigned bal = __ballot_sync(0xffffffffu, (larger >> i) & 1u);
          const int j = lane + 32 * i, t = nt + __popc(bal & ((1u << lane) - 1u));
          if (((larger >> i) & 1u) && t < kLocalTodo)
            todo[t] = (uint16_t)((x0 + j / w) * nbin + y0 + j % w);
          nt += __popc(bal);
        }
        __syncwarp();
        blocked = nt > kLocalTodo;  // too many to look at: not this round
        for (int t0 = 0; t0 < nt && !blocked; t0 += 4) {
          const int t = t0 + (lane >> 3), o = t < nt ? todo[t] : 0;
          const int i0 = t < nt ? (int)__ldcg(L.count + o) : 0;
          const int i1 = t < nt ? (int)__ldcg(L.count + o + 1) : 0;
          bool near = false;
          for (int i = i0 + (lane & 7); i < i1; i += 8) {
            const int4 c = __ldcg(L.rec + i);
            near |= eligible(c) && within(c.x, pos, lim2) &&
                    local_before(L, c, local_level(L, c), me, mx);
          }
          blocked = __any_sync(0xffffffffu, near);
        }
        __syncwarp();
      }
      if (!blocked && lane == 0) {
        const unsigned slot = atomicAdd((iv ? L.ndom : L.npick) + par, 1u);
        if (iv || slot < (unsigned)cap)  // a cell has one at most, and dom room for all
          __stcg((iv ? L.dom : L.pick) + slot, make_int4(at.x, me.z, pos, me.y));
      }
    }
    mark(3);
    if (!group_sync(gb, a.err, &s.flag)) return;
    mark(4);
    int m = iv ? (int)__ldcg(L.ndom + par) : min((int)__ldcg(L.npick + par), cap);
    int *bad = L.bad + par * ncell * ncell;
    if (iv) {
      // ---- B2. those that no newly covered neighbour can overtake; the CTAs share the
      // searches, several to one where they are few
      int parts = min(kLocalShare, G / max(m, 1));
      if (parts < kLocalShareMin) parts = 1;
      for (int d = k; d < m * parts; d += G) {
        const int4 c = __ldcg(L.dom + d % m);
        const int4 me = __ldcg(L.rec + c.x);
        bool top = local_level(L, me) == M;  // the first of all is the greedy's next pick
        if (top) {
          bool first = true;
          for (int j = tid; j < m; j += T) {
            const int4 o = __ldcg(L.rec + __ldcg(&L.dom[j].x));
            first &= local_level(L, o) != M || !local_before(L, o, M, me, M);
          }
          top = __syncthreads_and(first);
        }
        if (top) continue;
        if (parts == 1)
          local_threat<true>(a, s, reinterpret_cast<unsigned *>(s.pair_at), bad + d, c, side, nbin,
                             0, 1);
        else
          local_threat<false>(a, s, L.search + (size_t)(d % m) * kLocalSearch, bad + d % m, c, side,
                              nbin, d / m, parts);
      }
      mark(10);
      if (!group_sync(gb, a.err, &s.flag)) return;
      if (parts > 1)
        for (int i = gtid; i < m * kLocalSearch; i += gthreads) __stcg(L.search + i, 0u);
      mark(11);
    }
    // ---- C. the picks and their new bits -----------------------------------------------
    if (k == 0 && tid == 0) __stcg(L.gmax + par, 0ull);  // read by all; next used in two rounds
    unsigned long long areas = 0;
    if (iv) {  // the dominant candidates that nothing threatens, in the list's order
      int kept = 0;
      for (int i0 = 0; i0 < m; i0 += T) {
        const int i = i0 + tid;
        const bool ok = i < m && !__ldcg(bad + i);
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        __syncthreads();
        if (lane == 0) s.red[warp] = __popc(bal);
        __syncthreads();
        int j = kept + __popc(bal & ((1u << lane) - 1u));
        for (int w = 0; w < nwarps; w++) {
          j += w < warp ? (int)s.red[w] : 0;
          kept += (int)s.red[w];
        }
        if (ok && j < cap) s.order[j] = i;
      }
      m = min(kept, cap);
      __syncthreads();
    }
    if (m == 0) {  // never: the greedy's next pick is always among them
      if (k == 0 && tid == 0) atomicOr(a.err, kErrSiteMismatch);
      break;
    }
    for (int i = tid; i < m; i += T) {
      const int4 q = __ldcg(iv ? L.dom + s.order[i] : L.pick + i);
      s.at[i] = q.x;
      s.cand[i] = q.y;
      s.pos[i] = q.z;
      s.area[i] = q.w;
      areas += (unsigned)q.w;
      if (iv) {
        const int4 c = __ldcg(L.rec + q.x);
        s.reach[i] = local_level(L, c);
        s.parent[i] = parent_of(c);
      }
    }
    areas = block_sum(areas, s.red);  // (and the picks are in place)
    // the bin ranges of each pick's candidates
    for (int i = tid; i < m * kLocalRanges; i += T) {
      const int p = i / kLocalRanges, j = i - p * kLocalRanges;
      const int x = row_of(s.pos[p]), y = s.pos[p] & 0xffff;
      const int bx = max(0, x - 2 * roi) / side + j, bxe = min(n - 1, x + 2 * roi) / side;
      int r0 = 0, len = 0;
      if (bx <= bxe) {
        // columns that the circle reaches in these rows
        const int near = max(0, max(bx * side - x, x - (bx * side + side - 1)));
        const int half = min(2 * roi, (int)sqrtf((float)(lim2 - near * near)) + 1);
        r0 = (int)__ldcg(L.count + bx * nbin + max(0, y - half) / side);
        len = (int)__ldcg(L.count + bx * nbin + min(n - 1, y + half) / side + 1) - r0;
      }
      s.range0[i] = r0;
      s.prefix[i + 1] = len;
    }
    for (int i0 = (k * nwarps + warp) * 32; i0 < m * nr * nb2; i0 += gthreads) {
      const int i = i0 + lane;
      int cnt = 0, p = 0;
      if (i < m * nr * nb2) {
        const int row = i / nb2, q = i - row * nb2;
        p = row / nr;
        const int prow = row - p * nr;
        const int gr = row_of(s.pos[p]) - roi + prow, c0 = (s.pos[p] & 0xffff) - roi;
        const int w = (c0 >> 6) + q, fb = c0 & 63;
        uint64_t v = 0ull;
        if (gr >= 0 && gr < n && w >= 0 && w < cw) {
          const uint64_t *prw = a.sheds + (size_t)s.cand[p] * per + (size_t)prow * nwpr;
          const uint64_t cur = q < nwpr ? __ldg(prw + q) : 0ull;
          const uint64_t prev = q > 0 && fb ? __ldg(prw + q - 1) : 0ull;
          v = ((cur >> fb) | (fb ? prev << (64 - fb) : 0ull)) & ~__ldcg(cum + (size_t)gr * cw + w);
        }
        __stcg(a.nbits + i, v);
        cnt = __popcll(v);
      }
      const int p0 = __shfl_sync(0xffffffffu, p, 0);
      if (__all_sync(0xffffffffu, p == p0 || cnt == 0)) {
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0 && cnt) atomicAdd(L.ncount + par * cap + p0, cnt);
      } else if (cnt) {
        atomicAdd(L.ncount + par * cap + p, cnt);
      }
    }
    __syncthreads();
    {  // prefix sums of the ranges' lengths
      const int cntr = m * kLocalRanges, each = (cntr + T - 1) / T;
      const int b0 = min(tid * each, cntr), b1 = min(b0 + each, cntr);
      int sum = 0;
      for (int b = b0; b < b1; b++) sum += s.prefix[b + 1];
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) s.red[warp] = (unsigned)incl;
      __syncthreads();
      int run = incl - sum;
      for (int w = 0; w < warp; w++) run += (int)s.red[w];
      for (int b = b0; b < b1; b++) {
        run += s.prefix[b + 1];
        s.prefix[b + 1] = run;
      }
      if (tid == 0) s.prefix[0] = 0;
    }
    mark(5);
    if (!group_sync(gb, a.err, &s.flag)) return;
    mark(6);
    // ---- D. the neighbours' gains, the coverage ---------------------------------------
    for (int i = gtid; i < m * nr * nb2; i += gthreads) {
      const uint64_t v = __ldcg(a.nbits + i);
      if (!v) continue;
      const int row = i / nb2, p = row / nr, gr = row_of(s.pos[p]) - roi + (row - p * nr);
      const int w = (((s.pos[p] & 0xffff) - roi) >> 6) + (i - row * nb2);
      atomicOr(reinterpret_cast<unsigned long long *>(cum + (size_t)gr * cw + w), v);
    }
    if (k == 0)
      for (int i = tid; i < m; i += T) {
        __stcg(L.plist + np + i, local_key(s.area[i], s.cand[i]));
        if (iv) {
          __stcg(L.preach + np + i, s.reach[i]);
          // The chain's picks with larger keys than this one's never decide an order.
          const unsigned long long key = local_key(s.area[i], s.cand[i]);
          int q = s.parent[i];
          while (q >= 0 && __ldcg(L.plist + q) > key) q = __ldcg(L.pparent + q);
          __stcg(L.pparent + np + i, q);
        }
        __stcg(&L.rec[s.at[i]].y, 0);  // used
        if (__ldcg(L.ncount + par * cap + i) != s.area[i]) atomicOr(a.err, kErrSiteMismatch);
      }
    const int all = s.prefix[m * kLocalRanges];
    const int e0 = (int)((long long)all * k / G), e1 = (int)((long long)all * (k + 1) / G);
    const size_t nper = (size_t)nr * nb2;
    int have0 = 0, have1 = -1;  // picks whose N is in shared memory
    for (int c0 = e0; c0 < e1; c0 += T) {
      if (tid == 0) s.n = s.next = 0;
      __syncthreads();
      const int e = c0 + tid;
      if (e < e1) {
        int lo = 0, hi = m - 1;  // the last pick whose candidates start at or before e
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s.prefix[mid * kLocalRanges] <= e)
            lo = mid;
          else
            hi = mid - 1;
        }
        const int p = lo, pe = s.prefix[p * kLocalRanges];
        // A pick's candidates are taken in a strided order, so that every CTA gets
        // near ones, which share many rows with the pick, and far ones (in bin order
        // the busiest CTA took 2.5 times the mean).
        const int len = s.prefix[(p + 1) * kLocalRanges] - pe;
        const int stride = len % kLocalStride ? kLocalStride : kLocalStride + 8;  // both are prime
        const int at_e = pe + (int)((long long)(e - pe) * stride % len);
        lo = p * kLocalRanges;
        hi = lo + kLocalRanges - 1;  // the last range that starts at or before it
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s.prefix[mid] <= at_e)
            lo = mid;
          else
            hi = mid - 1;
        }
        const int at = s.range0[lo] + (at_e - s.prefix[lo]);
        const int4 rec = __ldcg(L.rec + at);
        const int cpos = rec.x;
        if (tid == 0) s.first = p;
        if (e == min(e1, c0 + T) - 1) s.last = p;
        if (within(cpos, s.pos[p], lim2) && at != s.at[p] && rec.y > 0) {
          const int j = atomicAdd(&s.n, 1), c = rec.z;
          s.pair_at[j] = at;
          s.pair_cand[j] = c;
          s.pair_pos[j] = cpos;
          s.pair_pick[j] = p;
          if (iv && !(rec.w & 1)) atomicOr(&L.rec[at].w, 1);  // touched
          const int dx = row_of(s.pos[p]) - row_of(cpos);  // the rows of its shed that count
          const int r0 = max(0, dx), r1 = min(nr - 1, dx + 2 * roi);
          prefetch_l2(a.sheds + (size_t)c * per + (size_t)r0 * nwpr, (size_t)(r1 - r0 + 1) * nwpr * 8);
        }
      }
      __syncthreads();
      const int first = s.first, last = s.last;
      const bool fits = (size_t)(last - first + 1) * nper <= (size_t)a.local_words;
      if (fits && (first < have0 || last > have1)) {
        const uint64_t *src = a.nbits + (size_t)first * nper;
        for (size_t i = tid; i < (size_t)(last - first + 1) * nper; i += T) N[i] = __ldcg(src + i);
        have0 = first;
        have1 = last;
        __syncthreads();
      }
      if (iv)
        for (int j = tid; j < s.n; j += T) {  // own cells that a pick covers
          const int p = s.pair_pick[j], px = row_of(s.pos[p]), py = s.pos[p] & 0xffff;
          const int row = row_of(s.pair_pos[j]) - px + roi, y = s.pair_pos[j] & 0xffff;
          const int w = (y >> 6) - ((py - roi) >> 6);
          if (row < 0 || row >= nr || w < 0 || w >= nb2) continue;
          const size_t i = (size_t)row * nb2 + w;
          const uint64_t v = fits ? N[(size_t)(p - have0) * nper + i] : __ldcg(a.nbits + (size_t)p * nper + i);
          if ((v >> (63 - (y & 63))) & 1ull)
            atomicOr(&L.rec[s.pair_at[j]].w, ((np + p) << 2) | 3);
        }
      if (fits)
        local_pairs<true>(a, s, N, have0, cw, lane);
      else
        local_pairs<false>(a, s, a.nbits, 0, cw, lane);
      __syncthreads();
    }
    if (tid == 0) s.total += areas;
    np += m;
    mark(7);
    if (!group_sync(gb, a.err, &s.flag)) return;
    mark(8);
  }

  // ---- the picks up to the stop, in the greedy's order -----------------------------------
  // A pick's place and the areas before it, by counting the picks before it.  Without
  // intervis these have larger keys.  With it a pick waits for the one that covered
  // its cell, and comes before another where the least key on its chain of such
  // picks, up to where the two chains meet, is larger.
  __syncthreads();
  unsigned long long kept = 0, area = 0;
  auto place = [&](unsigned above, unsigned before, unsigned long long mine) {
    if ((long long)before < a.stop_area) {  // areas sum to at most n^2 < 2^31
      const int c = (int)(0xFFFFFFFFu - (unsigned)mine);
      a.order[above] = c;
      a.selected[c] = 1;
      kept++;
      area += mine >> 32;
    }
  };
  if (np <= (iv ? kLocalDirectChains : kLocalDirect)) {  // against all picks, in shared memory
    unsigned long long *key = reinterpret_cast<unsigned long long *>(N), *reach = key + np;
    int *parent = reinterpret_cast<int *>(reach + np);
    for (int i = tid; i < np; i += T) {
      key[i] = __ldcg(L.plist + i);
      if (iv) {
        reach[i] = __ldcg(L.preach + i);
        parent[i] = __ldcg(L.pparent + i);
      }
    }
    __syncthreads();
    for (int x = k + G * tid; x < np; x += G * T) {
      const unsigned long long mine = key[x], rx = iv ? reach[x] : mine;
      unsigned above = 0, before = 0;
      for (int y = 0; y < np; y++) {
        const unsigned long long ry = iv ? reach[y] : key[y];
        bool first = ry > rx;
        if (iv && ry == rx && y != x) {
          unsigned long long mx = ~0ull, my = ~0ull;
          for (int cx = x, cy = y; cx != cy;) {  // a pick's parent was taken before it
            if (cx > cy) {
              mx = key[cx] < mx ? key[cx] : mx;
              cx = parent[cx];
            } else {
              my = key[cy] < my ? key[cy] : my;
              cy = parent[cy];
            }
          }
          first = my > mx;
        }
        if (first) {
          above++;
          before += (unsigned)(key[y] >> 32);
        }
      }
      place(above, before, mine);
    }
  } else {
    local_order(a, s, gb, k, np, place);
  }
  kept = block_sum(kept, s.red);
  area = block_sum(area, s.red);
  mark(9);
  if (tid == 0) {
    unsigned long long *out = reinterpret_cast<unsigned long long *>(a.out);
    if (kept) atomicAdd(out, kept);
    if (area) atomicAdd(out + 1, area);
    if (k == 0) {
      a.out[2] = rounds;
      for (int i = 0; i < kSitePhases; i++) a.out[3 + i] = phase[i];
    }
  }
}

}  // namespace
}  // namespace siting
