// SITE without intervisibility, by locally dominant picks.
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
// Candidates are sorted into square bins of a quarter of roi, row-major, so a run of
// bins in a bin row is one range of the sorted arrays.  A round:
//   A. eight lanes a bin find its largest key;
//   B. of each cell of 4x4 bins (any two of its candidates are within 2*roi) only
//      the largest can be dominant: a warp compares it with the largest of the
//      bins within 2*roi, and with the single candidates of those whose largest is
//      greater but too far; dominant ones of at least half the largest area are
//      this round's picks (below that, a pick may well lie beyond the stop);
//   C. the rows of the picks' new bits N = placed(shed) & ~coverage, spread over
//      all threads;
//   D. |V_u n N| for each (pick, unused candidate u within 2*roi): the candidates
//      in the picks' bin ranges are split evenly over the CTAs; a CTA lists its
//      pairs, copies the one or two picks' N that it needs to shared memory, and its
//      warps count a pair at a time, a lane a row.  Picks are more than 2*roi
//      apart, so their new bits are disjoint and the gains' decreases add up.
// Four group barriers a round.
#pragma once

#include "common.cuh"

namespace siting {
namespace {

constexpr int kLocalMaxBins = 256;   // bins a side at most
constexpr int kLocalMaxPicks = 256;  // picks of a round at most
constexpr int kLocalRanges = 20;     // bin rows a pick's candidates can span (4*roi+1 cells and a margin)
constexpr int kLocalCell = 4;        // bins a side of a cell of B
constexpr int kLocalTodo = 64;
constexpr int kLocalStride = 7919;   // order of a pick's candidates
constexpr int kLocalLook = 12;       // 32s of bins within reach: at most 19 a side

// Bins: side (cells of the DEM) and count a side.
__host__ __device__ __forceinline__ int local_bin_side(int n, int roi) {
  const int least = (n + kLocalMaxBins - 1) / kLocalMaxBins, quarter = (roi + 3) / 4;
  return quarter > least ? quarter : least;
}
__host__ __device__ __forceinline__ int local_bins(int n, int roi) {
  const int s = local_bin_side(n, roi);
  return (n + s - 1) / s;
}
// Picks a round takes at most: more for many candidates, while their new bits
// take at most 8 MB.
__host__ __device__ __forceinline__ int local_cap(int nsheds, int roi) {
  const size_t nr = 2 * (size_t)roi + 1, one = nr * ((nr + 63) / 64 + 1) * 8;
  const int want = nsheds >= 131072 ? 256 : nsheds >= 32768 ? 128 : 64;
  return want * one <= (size_t)8 << 20 ? want : 64;
}

// Shared memory of a CTA, sized for the largest job; the picks' new bits follow.
struct LocalShared {
  int at[kLocalMaxPicks], cand[kLocalMaxPicks], pos[kLocalMaxPicks], area[kLocalMaxPicks];
  int range0[kLocalMaxPicks * kLocalRanges];        // range starts in the sorted arrays
  int prefix[kLocalMaxPicks * kLocalRanges + 4];    // candidates before each range
  int pair_at[1024], pair_cand[1024], pair_pos[1024], pair_pick[1024];
  int todo[32][kLocalTodo];  // a warp's bins to look into
  unsigned long long red[32];
  unsigned long long hist[256];
  unsigned long long total, sum;
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
    if (d && lane == 0) atomicSub(a.local.gain + s.pair_at[j], d);
  }
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
  const int cap = local_cap(a.nsheds, roi);
  uint64_t *N = reinterpret_cast<uint64_t *>(&s + 1);
  GroupBarrier gb{a.bar, (unsigned)G, 0u};
  auto mark = [&](int i) {
    if (k == 0 && tid == 0) {
      const long long now = clock64();
      phase[i] += now - *tmark;
      *tmark = now;
    }
  };

  // ---- candidates into bins ------------------------------------------------------
  auto bin_of = [&](int cell, int *pos) {
    const int x = cell / n, y = cell - x * n;
    *pos = (int)((unsigned)x << 16) | y;
    return (x / side) * nbin + y / side;
  };
  for (int c = gtid; c < a.nsheds; c += gthreads) {
    int pos;
    atomicAdd(L.count + bin_of(__ldg(a.obs + c), &pos), 1u);
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
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
    const int b = bin_of(__ldg(a.obs + c), &pos);
    const unsigned at = __ldcg(L.count + b) + atomicAdd(L.fill + b, 1u);
    __stcg(L.cand + at, c);
    __stcg(L.pos + at, pos);
    __stcg(L.gain + at, __ldcg(a.gains + c));
  }
  if (tid == 0) s.total = 0;
  if (!group_sync(gb, a.err, &s.flag)) return;
  mark(0);

  uint64_t *cum = a.cum0;
  int rounds = 0, np = 0;
  for (;; rounds++) {
    const int par = rounds & 1;
    // ---- A. the largest key of each bin --------------------------------------------
    if (k == 0 && tid == 0 && rounds) __stcg(L.npick + (par ^ 1), 0u);
    unsigned long long mine = 0;
    for (int b0 = gwarp * 4; b0 < nbins; b0 += gwarps * 4) {
      const int b = b0 + (lane >> 3);
      const int i0 = b < nbins ? (int)__ldcg(L.count + b) : 0;
      const int i1 = b < nbins ? (int)__ldcg(L.count + b + 1) : 0;
      unsigned long long best = 0;
      int at = -1;
      for (int i = i0 + (lane & 7); i < i1; i += 8) {
        const int g = __ldcg(L.gain + i);
        const unsigned long long key = g > 0 ? local_key(g, __ldcg(L.cand + i)) : 0ull;
        if (key > best) {
          best = key;
          at = i;
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
        if (k2 > best) {  // keys are unique
          best = k2;
          at = a2;
        }
      }
      if ((lane & 7) == 0 && b < nbins) {
        __stcg(L.binkey + b, best);
        __stcg(L.binat + b, make_int2(at, at >= 0 ? __ldcg(L.pos + at) : 0));
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
        const unsigned long long key = __ldcg(L.plist + i);
        if (key > M) above += key >> 32;
      }
      if ((long long)block_sum(above, s.red) >= a.stop_area) break;
    }
    // ---- B. dominant candidates -----------------------------------------------------
    if (k == 0)
      for (int i = tid; i < cap; i += T) __stcg(L.ncount + (par ^ 1) * cap + i, 0);
    const unsigned least = (unsigned)((M >> 32) + 1) / 2;
    const int ncell = (nbin + kLocalCell - 1) / kLocalCell;
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
      const int from = __ffs(__ballot_sync(0xffffffffu, key == mx)) - 1;
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
        if (j < cnt && ex * ex + ey * ey <= lim2 && __ldcg(L.binkey + o) > mx) larger |= 1u << i;
      }
#pragma unroll
      for (int i = 0; i < kLocalLook; i++) {
        const int j = lane + 32 * i;
        const int o = (x0 + j / w) * nbin + y0 + j % w;
        if ((larger >> i) & 1u) hit |= within(__ldcg(&L.binat[o].y), pos, lim2);
      }
      bool blocked = __any_sync(0xffffffffu, hit);
      // their other candidates: four bins at a time, eight lanes a bin
      if (!blocked) {
        int *todo = s.todo[warp];
        int nt = 0;
#pragma unroll
        for (int i = 0; i < kLocalLook; i++) {
          const unsigned bal = __ballot_sync(0xffffffffu, (larger >> i) & 1u);
          const int j = lane + 32 * i, t = nt + __popc(bal & ((1u << lane) - 1u));
          if (((larger >> i) & 1u) && t < kLocalTodo) todo[t] = (x0 + j / w) * nbin + y0 + j % w;
          nt += __popc(bal);
        }
        __syncwarp();
        blocked = nt > kLocalTodo;  // too many to look at: not this round
        for (int t0 = 0; t0 < nt && !blocked; t0 += 4) {
          const int t = t0 + (lane >> 3), o = t < nt ? todo[t] : 0;
          const int i0 = t < nt ? (int)__ldcg(L.count + o) : 0;
          const int i1 = t < nt ? (int)__ldcg(L.count + o + 1) : 0;
          bool near = false;
          for (int c = i0 + (lane & 7); c < i1; c += 8) {
            const int g = __ldcg(L.gain + c);
            near |= g > 0 && local_key(g, __ldcg(L.cand + c)) > mx &&
                    within(__ldcg(L.pos + c), pos, lim2);
          }
          blocked = __any_sync(0xffffffffu, near);
        }
        __syncwarp();
      }
      if (!blocked && lane == 0) {
        const unsigned slot = atomicAdd(L.npick + par, 1u);
        if (slot < (unsigned)cap)
          __stcg(L.pick + slot, make_int4(at.x, (int)(0xFFFFFFFFu - (unsigned)mx), pos, (int)(mx >> 32)));
      }
    }
    mark(3);
    if (!group_sync(gb, a.err, &s.flag)) return;
    mark(4);
    // ---- C. the picks and their new bits -----------------------------------------------
    if (k == 0 && tid == 0) __stcg(L.gmax + par, 0ull);  // read by all; next used in two rounds
    const int m = min((int)__ldcg(L.npick + par), cap);
    unsigned long long areas = 0;
    for (int i = tid; i < m; i += T) {
      const int4 q = __ldcg(L.pick + i);
      s.at[i] = q.x;
      s.cand[i] = q.y;
      s.pos[i] = q.z;
      s.area[i] = q.w;
      areas += (unsigned)q.w;
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
        __stcg(L.gain + s.at[i], 0);  // used
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
        const int at = s.range0[lo] + (at_e - s.prefix[lo]), cpos = __ldcg(L.pos + at);
        if (tid == 0) s.first = p;
        if (e == min(e1, c0 + T) - 1) s.last = p;
        if (within(cpos, s.pos[p], lim2) && at != s.at[p] && __ldcg(L.gain + at) > 0) {
          const int j = atomicAdd(&s.n, 1), c = __ldcg(L.cand + at);
          s.pair_at[j] = at;
          s.pair_cand[j] = c;
          s.pair_pos[j] = cpos;
          s.pair_pick[j] = p;
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

  // ---- the picks up to the stop, in order of falling key ---------------------------------
  if (np <= 1024) {  // one CTA: each pick's rank and the areas before it, by counting
    if (k != 0) return;
    unsigned long long *key = reinterpret_cast<unsigned long long *>(s.pair_at);  // 8 KB
    for (int i = tid; i < np; i += T) key[i] = __ldcg(L.plist + i);
    __syncthreads();
    unsigned long long kept = 0, area = 0;
    for (int i = tid; i < np; i += T) {
      const unsigned long long mine = key[i];
      unsigned above = 0, before = 0;  // areas sum to at most n^2 < 2^31
#pragma unroll 8
      for (int j = 0; j < np; j++) {
        const unsigned long long o = key[j];
        above += o > mine;
        before += o > mine ? (unsigned)(o >> 32) : 0u;
      }
      if ((long long)before < a.stop_area) {
        const int c = (int)(0xFFFFFFFFu - (unsigned)mine);
        a.order[above] = c;
        a.selected[c] = 1;
        kept++;
        area += mine >> 32;
      }
    }
    kept = block_sum(kept, s.red);
    area = block_sum(area, s.red);
    mark(9);
    if (tid == 0) {
      a.out[0] = (long long)kept;
      a.out[1] = (long long)area;
      a.out[2] = rounds;
      for (int i = 0; i < kSitePhases; i++) a.out[3 + i] = phase[i];
    }
    return;
  }
  // T: the largest key with the areas of the keys >= T reaching the stop (0: they
  // never do), found 8 bits at a time, alike in every CTA
  unsigned long long thr = 0;
  if ((long long)s.total >= a.stop_area) {
    unsigned long long need = (unsigned long long)a.stop_area, mask = 0;
    for (int sft = 56; sft >= 0; sft -= 8) {
      for (int i = tid; i < 256; i += T) s.hist[i] = 0;
      __syncthreads();
      for (int i = tid; i < np; i += T) {
        const unsigned long long key = __ldcg(L.plist + i);
        if ((key & mask) == thr) atomicAdd(&s.hist[(key >> sft) & 255], key >> 32);
      }
      __syncthreads();
      if (warp == 0) {  // the digit: eight a lane from the largest down
        unsigned long long sum = 0;
        for (int j = 0; j < 8; j++) sum += s.hist[255 - 8 * lane - j];
        unsigned long long incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (incl >= need && incl - sum < need) {  // one lane
          unsigned long long left = need - (incl - sum);
          int d = 255 - 8 * lane;
          while (s.hist[d] < left) left -= s.hist[d--];
          s.n = d;
          s.sum = left;
        }
      }
      __syncthreads();
      thr |= (unsigned long long)s.n << sft;
      need = s.sum;
      mask |= 255ull << sft;
      __syncthreads();
    }
  }
  unsigned long long kept = 0, area = 0;
  for (int i = tid; i < np; i += T) {
    const unsigned long long key = __ldcg(L.plist + i);
    if (key >= thr) {
      kept++;
      area += key >> 32;
    }
  }
  kept = block_sum(kept, s.red);
  area = block_sum(area, s.red);
  // rank: larger keys, counted 1024 at a time
  const int nch = (np + 1023) / 1024;  // at least 2
  for (int it = gtid; it < np * nch; it += gthreads) {
    const int ch = it / np, i = it - ch * np;
    const unsigned long long key = __ldcg(L.plist + i);
    if (key < thr) continue;
    unsigned above = 0;
    const int j1 = min(np, (ch + 1) * 1024);
#pragma unroll 8
    for (int j = ch * 1024; j < j1; j++) above += __ldcg(L.plist + j) > key;
    atomicAdd(L.rank + i, above);
    if (ch == 0) a.selected[0xFFFFFFFFu - (unsigned)key] = 1;
  }
  if (!group_sync(gb, a.err, &s.flag)) return;
  for (int i = gtid; i < np; i += gthreads) {
    const unsigned long long key = __ldcg(L.plist + i);
    if (key >= thr) a.order[__ldcg(L.rank + i)] = (int)(0xFFFFFFFFu - (unsigned)key);
  }
  mark(9);
  if (k == 0 && tid == 0) {
    a.out[0] = (long long)kept;
    a.out[1] = (long long)area;
    a.out[2] = rounds;
    for (int i = 0; i < kSitePhases; i++) a.out[3 + i] = phase[i];
  }
}

}  // namespace
}  // namespace siting
