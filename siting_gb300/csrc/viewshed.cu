// VIEWSHED: bit-packed viewshed of every tentative observer
// (siting.cpp:247-360).
//
// From observer o, rays go to each of the 8*roi perimeter cells of the
// (2roi+1)^2 box (perimeter order of siting.cpp:291-304).  A ray steps the
// major axis, puts the minor coordinate at o + round(i*slope), stops at the
// DEM edge or outside the roi circle, keeps the running maximum horizon slope
// s = (elev - oalt)/|i| and marks the cell when elev + tht >= oalt + hs*|i|.
// Bit (row, col) of a shed is word row*nwpr + col/64, bit 63 - col%64.
//
// GB300 mapping: a thread sweeps a pair of rays that mirror each other about the
// observer's column (or a quadrant's diagonal): the rounded minor offset, the step
// table and the mark's line are the same for both, and the FP32 operations of the
// two are packed pairs.  The observer's window is loaded into shared memory by TMA
// bulk-tensor copies, whole, as the halves above and below the observer, or as
// quarters, one CTA each (shed_staged_plan); windows that do not fit even so are
// read through L1 by the same code.  Visible cells are marked in a shared-memory
// image of the shed, which is then written to HBM with coalesced stores.
//
// Bound by instruction issue and shared-memory wavefronts alike (76% and 82% of
// their peaks at roi 100).  2048^2, ms before (one ray a thread) and after: 102400
// observers of roi 10 0.205, 0.195; roi 20 0.512, 0.451; roi 30 0.982, 0.646; 65536 of roi
// 50 1.523, 1.070; 45511 of roi 60 1.490, 0.959; 16384 of roi 100 1.241, 0.934; 6400 of
// roi 160 1.488, 0.999; 4096 of roi 200 1.604, 1.044; 2844 of roi 240 1.872, 1.431.
//
// Half windows: every ray to a target row tx <= ox stays in rows ox-roi..ox,
// every other ray in rows ox..ox+roi, so the sides can be swept apart.  The
// observer's row is the upper side's: the lower side's rays meet it only in a
// prefix of steps k with round(k*slope) = 0, and such a prefix samples the cells
// (ox, oy+-k) in the order and at the steps of the straight ray to (ox, oy+-roi)
// of the upper side, with the same horizons, so its marks there are a subset of
// that ray's.  The same holds for the observer's column, which rows take from the
// straight rays along it.
//
// Bit-exactness: separately rounded FP32 operations, IEEE division for the
// slopes (of which the sign goes with the strides, as rounding is symmetric),
// round-half-away-from-zero for the minor coordinate.  The horizon
// slope s = RN(a/k) (a an integer elevation difference, k the step) is
// q0 = RN(a*y), s = RN(q0 + RN(a - k*q0)*y) with y = RN(1/k) from a per-CTA
// table: one fused correction of a quotient within an ulp, given a correctly
// rounded reciprocal, yields the correctly rounded quotient (Markstein's
// theorem), and an exhaustive check of every |a| <= 2^21, k <= 2048 (the
// validated heights and rois) against IEEE division agrees bit for bit.
// Beyond that range the kernel divides.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace siting {
namespace {

// 32x32 bit transpose: lane j's bit i becomes lane i's bit j.
__device__ __forceinline__ unsigned warp_transpose(unsigned x, int lane) {
  // halves and bytes are exchanged by byte permutations, the rest by masks
  unsigned o = __shfl_xor_sync(0xffffffffu, x, 16);
  x = __byte_perm(x, o, (lane & 16) ? 0x3276 : 0x5410);
  o = __shfl_xor_sync(0xffffffffu, x, 8);
  x = __byte_perm(x, o, (lane & 8) ? 0x3715 : 0x6240);
#pragma unroll
  for (int sh = 4; sh >= 1; sh >>= 1) {
    const unsigned m = sh == 4 ? 0x0F0F0F0Fu : sh == 2 ? 0x33333333u : 0x55555555u;
    o = __shfl_xor_sync(0xffffffffu, x, sh);
    x = (lane & sh) ? (x & ~m) | ((o >> sh) & m) : (x & m) | ((o << sh) & ~m);
  }
  return x;
}

struct ShedArgs {
  const uint16_t *dem;
  int pitch, n, roi, oht, tht;
  const int32_t *obs;
  uint64_t *sheds;
  int *err;
  int items, chunk;  // quarters: halves of observers in all and to a cluster
  unsigned long long rn;  // ceil(2^64/n)
  unsigned rw, rb;        // ceil(2^16/nwpr), ceil(2^16/nw): a thread's or block's number by these
};

// floor(v / n), 0 <= v < 2^31: v*rn exceeds 2^64*v/n by less than 2^64/n.
__device__ __forceinline__ int div_n(int v, const ShedArgs &a) {
  return a.n > 1 ? (int)__umul64hi((unsigned long long)(unsigned)v, a.rn) : v;
}

// One CTA's share of an observer: rows on one side of it (kHalves = 1, block
// 2o the upper side of observer o, 2o+1 the lower) or all (kHalves = 2).
//
// Shared memory: the window, the step table {RN(1/k), RN(1/k), -k, -k} and a pair
// of bit images for each side.
// An image has a line per minor offset 0..roi (`ls` words, odd, so that lines
// start in distinct banks) with a bit per step k-1, the right and the left ray's
// words interleaved: image X holds the x-major rays (line = column distance, bit
// = row distance - 1), image Y the y-major ones (line = row distance, bit =
// column distance - 1).
__host__ __device__ __forceinline__ int pair_words(int roi) { return (roi + 31) / 32; }
__host__ __device__ __forceinline__ int pair_line(int roi) { return 2 * pair_words(roi) + 1; }
// The window's boxes.  A row pitch of an odd multiple of 4 words (the finest that
// a tensor copy gives) starts 8 successive rows in distinct banks.
struct WinGeom {
  int w, box_rows, nboxes;
  __host__ __device__ size_t bytes() const { return (size_t)nboxes * box_rows * w * 2; }
};

__host__ __device__ __forceinline__ WinGeom win_geom(int roi, int halves, bool staged) {
  if (!staged) return WinGeom{0, 0, 0};
  const int rows = halves == 2 ? 2 * roi + 1 : roi + 1;
  WinGeom g;
  g.w = ((2 * roi + 8 + 7) & ~7) | 8;
  g.nboxes = (rows + 255) / 256;
  g.box_rows = ((rows + g.nboxes - 1) / g.nboxes + 7) & ~7;  // boxes start on 128 bytes
  return g;
}

// The first kNearSteps steps of the rays mark bytes instead of image bits: near
// the observer many lanes of a warp meet in one cell, whose stores then merge,
// where atomic ORs would queue up (at step k about roi/k lanes to a cell).  Line =
// minor offset, byte = step - 1, an odd number of words a line; one such map
// for each image and side.  Large quarters map more steps (quad_near): at radius 200 the
// ORs' conflicts are a quarter of all shared wavefronts, three in four of them between
// steps 17 and 48.
constexpr int kNearSteps = 16, kFarNearSteps = 48;
__host__ __device__ constexpr int near_line(int steps) { return steps + 4; }  // bytes
__host__ __device__ constexpr int near_map(int steps) { return (steps + 1) * near_line(steps); }

// Words of the images and near maps.
__host__ __device__ __forceinline__ int pair_mark_words(int roi, int halves) {
  return halves * (2 * (roi + 1) * pair_line(roi) + near_map(kNearSteps));  // 4 maps of bytes a side
}

size_t pair_smem_bytes(int roi, int halves, bool staged) {
  return win_geom(roi, halves, staged).bytes() + (size_t)(roi + 1) * 16 + 16 +
         (((size_t)pair_mark_words(roi, halves) * 4 + 15) & ~(size_t)15);
}

// Elevation at `at`: a shared-memory address in the staged window, or an element
// offset of the DEM read through L1.
template <bool kStaged>
__device__ __forceinline__ int elevation(const uint16_t *dem, int at) {
  if constexpr (kStaged) {
    int v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
  } else {
    return __ldg(dem + at);
  }
}

// A table entry that the compiler cannot fold; ordered with the stores and barriers before.
__device__ __forceinline__ float ld_shared_f32(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

constexpr float kNoHorizon = -99999.f;

// The steps k..k1 of a pair of rays: A and B are mirror images about the
// observer's column, so the minor offset, the table entry and the image line
// are shared and the FP32 operations are packed pairs.
struct PairRays {
  const uint16_t *dem;
  int p0;      // the observer's cell (see elevation())
  int pA, pB;  // cells of step k-1 at minor offset 0
  int mA, mB;  // a step along the major axis
  int sA, sB;  // a step along the minor axis
  float sl;         // |slope|
  unsigned long long hs;  // horizons
  unsigned long long nalt, tht;  // -observer height, target height
  unsigned long long one;  // 1, from memory
  uint32_t img;     // image line 0
  uint32_t near;    // near map line 0 of the right ray; the left one's follows
  int ls4;          // bytes of an image line
  const float4 *tab;  // step table
};

// Steps k..k+3 (k = 1 modulo 4: within one word of the image).  kClamp: a ray's
// last group, whose steps beyond k1 repeat step k1, which changes nothing.
// kNear: the near maps' steps, which mark bytes there; 0: bits of the image.
template <bool kStaged, bool kRcp, int kNear, bool kClamp>
__device__ __forceinline__ void pair_group(PairRays &r, int k, int k1) {
  float4 t[4];
  int off[4], ea[4], eb[4], kk[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    kk[i] = kClamp ? min(k + i, k1) : k + i;
    t[i] = r.tab[kk[i]];
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    // round(k*|slope|), half away from zero
    off[i] = f2i(__fsub_rn(0x1.fffffep-2f, fmul(t[i].z, r.sl)));
    int cA, cB;  // the step's cells at minor offset 0
    if constexpr (kClamp) {
      cA = r.p0 + kk[i] * r.mA;
      cB = r.p0 + kk[i] * r.mB;
    } else {
      cA = r.pA += r.mA;
      cB = r.pB += r.mB;
    }
    ea[i] = elevation<kStaged>(r.dem, cA + off[i] * r.sA);
    eb[i] = elevation<kStaged>(r.dem, cB + off[i] * r.sB);
  }
  const uint32_t mk = r.img + 8u * (uint32_t)((k - 1) >> 5);
  const unsigned bit0 = 1u << ((k - 1) & 31);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const unsigned long long y = f2_pack(t[i].x, t[i].y), nk = f2_pack(t[i].z, t[i].w);
    const unsigned long long e = f2_pack(i2f(ea[i]), i2f(eb[i]));
    // elevations and offsets are integers below 2^24: differences are exact
    const unsigned long long a = f2_add(e, r.nalt);
    unsigned long long s;  // RN(a/k)
    if constexpr (kRcp) {
      const unsigned long long q = f2_mul(a, y);
      s = f2_fma(f2_fma(q, nk, a), y, q);
    } else {
      s = f2_pack(fdiv(f2_lo(a), -t[i].z), fdiv(f2_hi(a), -t[i].z));
    }
    r.hs = f2_pack(fmaxf(f2_lo(r.hs), f2_lo(s)), fmaxf(f2_hi(r.hs), f2_hi(s)));
    // elev + tht >= oalt + hs*k, the right side carried negated
    const unsigned long long nv = f2_fma(f2_mul(r.hs, nk), r.one, r.nalt);
    const unsigned long long v = f2_add(e, r.tht);
    if constexpr (kNear > 0) {
      const uint32_t m = r.near + (uint32_t)(off[i] * near_line(kNear) + kk[i] - 1);
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %1, %2;\n\t@p st.shared.u8 [%0], %3;\n\t}" ::"r"(m),
                   "f"(f2_lo(v)), "f"(-f2_lo(nv)), "r"(1)
                   : "memory");
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %1, %2;\n\t@p st.shared.u8 [%0+%4], %3;\n\t}" ::"r"(m),
                   "f"(f2_hi(v)), "f"(-f2_hi(nv)), "r"(1), "n"(near_map(kNear))
                   : "memory");
    } else {
      // an invisible cell ORs nothing: a predicated OR would be a branch, with no
      // overlap of the steps on either side
      const uint32_t m = mk + (uint32_t)(off[i] * r.ls4);
      const unsigned bit = bit0 << (kk[i] - k);
      asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(m), "r"(f2_lo(v) >= -f2_lo(nv) ? bit : 0u)
                   : "memory");
      asm volatile("red.shared.or.b32 [%0+4], %1;" ::"r"(m), "r"(f2_hi(v) >= -f2_hi(nv) ? bit : 0u)
                   : "memory");
    }
  }
}

// RN(m/k) by the table entry of k, as in pair_group.  (Whole and half windows are half
// ends at small radii: this, the search of pair_last from within a step of the end, and
// the divisions by n and nwpr as products took roi 30 from 0.705 to 0.655 ms at 2048^2,
// 1.6 G cells of rays, 74 1.039 to 0.997, 118 0.957 to 0.925; the long sweeps of the
// quarters gain nothing by the first and the last.)
__device__ __forceinline__ float step_slope(const float4 &t, int m) {
  const float a = i2f(m), q = fmul(a, t.x);
  return __fmaf_rn(__fmaf_rn(q, t.z, a), t.x, q);
}

// Steps of the two rays of slope sl.  A ray stops outside the roi circle, at
// the DEM edge along the major axis (maj cells away), or when the minor
// coordinate leaves the DEM (min cells away) (siting.cpp:333-334); the offset
// never decreases with k, so each holds from some step on.
__device__ __forceinline__ void pair_last(float sl, int roi, int majA, int minA, int majB, int minB,
                                          int &kA, int &kB) {
  const int roi2 = roi * roi;
  auto off = [&](int k) { return f2i(fadd(fmul(i2f(k), sl), 0x1.fffffep-2f)); };
  // an offset at most half below the line lets the ray stay inside the circle for at
  // most sl/(2 + 2*sl^2) <= 1/4 step longer than the line, so the search starts there
  int kc = min(roi, (int)(i2f(roi) * rsqrtf(1.f + sl * sl) + 0.2525f));
  for (int o = off(kc); kc * kc + o * o > roi2; o = off(kc)) kc--;
  auto last = [&](int hi, int lim) {  // the last step <= hi with offset <= lim
    int lo = 0;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off(mid) <= lim)
        lo = mid;
      else
        hi = mid - 1;
    }
    return lo;
  };
  kA = min(kc, majA);
  kB = min(kc, majB);
  if (off(kA) > minA) kA = last(kA, minA);
  if (off(kB) > minB) kB = last(kB, minB);
}

// Steps k..k1 (k = 1 modulo 4).
template <bool kStaged, bool kRcp, int kNear>
__device__ __forceinline__ void pair_steps(PairRays &r, int k, int k1) {
  r.pA = r.p0 + (k - 1) * r.mA;
  r.pB = r.p0 + (k - 1) * r.mB;
  for (; k <= kNear && k + 3 <= k1; k += 4) pair_group<kStaged, kRcp, kNear, false>(r, k, k1);
  for (; k + 3 <= k1; k += 4) pair_group<kStaged, kRcp, 0, false>(r, k, k1);
  if (k > k1) return;
  if (k <= kNear)
    pair_group<kStaged, kRcp, kNear, true>(r, k, k1);
  else
    pair_group<kStaged, kRcp, 0, true>(r, k, k1);
}

// Sweeps A to step kA and B to step kB: first both rays to the nearer end, then,
// where the ends differ, the longer one alone; the other stays at the observer
// with its targets out of sight.
template <bool kStaged, bool kRcp, int kNear>
__device__ __forceinline__ void pair_sweep(PairRays &r, int kA, int kB) {
  const int kmin = min(kA, kB);
  pair_steps<kStaged, kRcp, kNear>(r, 1, kmin);
  if (kA != kB) {
    const bool a_on = kA > kB;
    r.tht = a_on ? f2_pack(f2_lo(r.tht), -3e38f) : f2_pack(-3e38f, f2_hi(r.tht));
    if (!a_on) r.mA = r.sA = 0;
    if (a_on) r.mB = r.sB = 0;
    // from the last group on again: a step done twice changes nothing
    pair_steps<kStaged, kRcp, kNear>(r, (kmin & ~3) + 1, max(kA, kB));
  }
}

// ORs line `line` of a near map into the words of an image line, two apart.
template <int kNear>
__device__ __forceinline__ void near_bits(const unsigned char *map, int line, unsigned *dst) {
  const unsigned *src = reinterpret_cast<const unsigned *>(map + line * near_line(kNear));
#pragma unroll
  for (int w = 0; w < (kNear + 31) / 32; w++) {
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < 8 && w * 8 + j < kNear / 4; j++)  // four bytes of 0 or 1 to a nibble
      bits |= (src[w * 8 + j] * 0x01020408u) >> 24 << (4 * j);
    if (bits) dst[2 * w] |= bits;
  }
}

// kSmall: a CTA of one warp for a small radius (kSmallMinRoi), whose pairs are a few more
// than its lanes.  It takes the straight y-major pair a lane a step and loops over the rest.
template <int kHalves, bool kStaged, bool kRcp, bool kSmall = false>
__global__ void __launch_bounds__(448, 2)
    shed_kernel(const __grid_constant__ CUtensorMap map, const ShedArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int roi = a.roi, n = a.n, nr = 2 * roi + 1, nwpr = (nr + 63) / 64, nwords = nr * nwpr;
  const int half0 = kHalves == 1 ? (int)(blockIdx.x & 1u) : 0;
  const int obi = kHalves == 1 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  uint64_t *dst = a.sheds + (size_t)obi * nwords;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  // shed rows this CTA writes: the upper side owns the observer's row
  const int wr0 = kHalves == 1 && half0 ? roi + 1 : 0, wr1 = kHalves == 1 && !half0 ? roi + 1 : nr;
  const int ob = a.obs[obi];
  if (ob < 0 || ob >= n * n) {  // invalid observer: empty shed, flagged
    for (int i = wr0 * nwpr + tid; i < wr1 * nwpr; i += blockDim.x) dst[i] = 0ull;
    if (tid == 0) atomicOr(a.err, kErrBadInput);
    return;
  }
  const int ox = div_n(ob, a), oy = ob - ox * n;
  const WinGeom g = win_geom(roi, kHalves, kStaged);
  const int W2 = 2 * g.w, nw = pair_words(roi);  // W2: row pitch, bytes
  const int ls = pair_line(roi), ximg = (roi + 1) * ls;  // words of an image
  const int hx0 = kHalves == 1 && half0 ? ox : ox - roi;  // window origin
  const int hy0 = (oy - roi) & ~7;  // TMA inner coordinate: 16-byte aligned
  const uint32_t win = smem_u32(sm);
  float4 *tab = reinterpret_cast<float4 *>(sm + g.bytes());
  uint64_t *mbar = reinterpret_cast<uint64_t *>(tab + roi + 1);
  unsigned *img = reinterpret_cast<unsigned *>(mbar + 2);
  unsigned char *near = reinterpret_cast<unsigned char *>(img + kHalves * 2 * ximg);
  if (kStaged && tid == 0) {
    mbar_init(mbar, 1);
    mbar_expect_tx(mbar, (uint32_t)g.bytes());
    for (int b = 0; b < g.nboxes; b++)
      tma_load_window(sm + (size_t)b * g.box_rows * g.w * 2, &map, hy0, hx0 + b * g.box_rows, mbar);
  }
  for (int i = tid; i <= roi; i += blockDim.x) {
    const float y = i ? __frcp_rn((float)i) : 0.f;
    tab[i] = make_float4(y, y, -(float)i, -(float)i);
  }
  for (int i = tid; i < (pair_mark_words(roi, kHalves) + 3) / 4; i += blockDim.x)
    reinterpret_cast<uint4 *>(img)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  if (kStaged && !__all_sync(0xffffffffu, mbar_wait(mbar, 0))) {
    if (tid == 0) atomicOr(a.err, kErrTmaTimeout);
    return;
  }

  // ---- rays: roi+1 x-major pairs and then the y-major ones of each side; the
  // straight y-major ray (minor offset 0) belongs to the upper side
  constexpr int kStraight = kSmall ? 0 : 1;
  const int up = 2 * roi + kStraight, npairs = kHalves == 2 ? 4 * roi + kStraight : half0 ? 2 * roi : up;
  // (a staged CTA has a thread for every pair: as a loop over pairs, the compiler
  // lets a warp's rays part at their ends, 15% more instructions)
  for (int t0 = tid; t0 < npairs; t0 += blockDim.x) {
    const int half = kHalves == 2 ? t0 >= up : half0;
    const int t = kHalves == 2 && half ? t0 - up : t0;
    const bool xm = t <= roi;
    // adjacent lanes take every second ray of their group: half as many meet in
    // one image word (2048^2, roi 100: 1.018 -> 0.980 ms; every third 0.992, as the
    // lengths of a warp's rays then differ more)
    const int first = kSmall ? 1 : half;  // the least minor offset of the y-major rays
    const int mt = xm ? t : t - (roi + 1), evens = ((xm ? roi + 1 : roi - first) + 1) / 2;
    const int m = (mt < evens ? 2 * mt : 2 * (mt - evens) + 1) + (xm ? 0 : first);
    const int rowlim = half ? n - 1 - ox : ox;  // rows on this side of the observer
    const int collimA = n - 1 - oy, collimB = oy;
    const float sl = kRcp ? step_slope(tab[roi], m) : fdiv(i2f(m), i2f(roi));
    int kA, kB;
    pair_last(sl, roi, xm ? rowlim : collimA, xm ? collimA : rowlim, xm ? rowlim : collimB,
              xm ? collimB : rowlim, kA, kB);
    PairRays r;
    // strides: bytes of the window, or elements of the DEM
    const int cell = kStaged ? 2 : 1, rowstep = (half ? 1 : -1) * (kStaged ? W2 : a.pitch);
    const int p0 = kStaged ? (int)win + (ox - hx0) * W2 + 2 * (oy - hy0) : ox * a.pitch + oy;
    r.dem = a.dem;
    r.p0 = p0;
    r.mA = xm ? rowstep : cell;
    r.mB = xm ? rowstep : -cell;
    r.sA = xm ? cell : rowstep;
    r.sB = xm ? -cell : rowstep;
    r.sl = sl;
    const float nalt = -i2f(elevation<kStaged>(a.dem, p0) + a.oht), tht = i2f(a.tht);
    r.nalt = f2_pack(nalt, nalt);
    // A product times 1 plus a sum keeps the product's own rounding: ptxas 13.0
    // contracts mul.rn.f32x2 into an add.rn.f32x2 that it feeds.
    const float one = ld_shared_f32(smem_u32(tab + 1));  // RN(1/1)
    r.one = f2_pack(one, one);
    r.img = smem_u32(img + ((kHalves == 2 && half ? 2 : 0) + (xm ? 0 : 1)) * ximg);
    r.near = smem_u32(near + ((kHalves == 2 && half ? 2 : 0) + (xm ? 0 : 1)) * 2 * near_map(kNearSteps));
    r.ls4 = 4 * ls;
    r.tab = tab;
    r.hs = f2_pack(kNoHorizon, kNoHorizon);
    r.tht = f2_pack(tht, tht);
    pair_sweep<kStaged, kRcp, kNearSteps>(r, kA, kB);
    if (kStaged && !kSmall) break;
  }
  if constexpr (kSmall) {
    // the observer's row: lanes 0..15 the steps to the right, 16..31 to the left, the
    // horizon a running maximum over the lanes
    const int side = lane >> 4, k = (lane & 15) + 1;
    const bool on = k <= min(roi, side ? oy : n - 1 - oy);
    const int p0 = (int)win + (ox - hx0) * W2 + 2 * (oy - hy0);
    const float e = i2f(elevation<true>(a.dem, on ? p0 + (side ? -2 : 2) * k : p0));
    const float nalt = -i2f(elevation<true>(a.dem, p0) + a.oht);
    const float4 t = tab[min(k, roi)];
    const float d = fadd(e, nalt), q = fmul(d, t.x);
    float hs = on ? __fmaf_rn(__fmaf_rn(q, t.z, d), t.x, q) : kNoHorizon;
    hs = fmaxf(hs, kNoHorizon);
    for (int o = 1; o < 16; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, hs, o, 16);
      if ((lane & 15) >= o) hs = fmaxf(hs, v);
    }
    // elev + tht >= oalt + hs*k, as in pair_group
    if (on && fadd(e, i2f(a.tht)) >= -fadd(fmul(hs, t.z), nalt))
      near[(2 + side) * near_map(kNearSteps) + k - 1] = 1;
  }
  __syncthreads();

  // ---- near maps into the images: a thread packs a line
  const int nlines = min(roi, kNearSteps) + 1, lsh2 = 32 - __clz(nlines - 1);  // lines, as 2^lsh2 slots
  for (int i = tid; i < kHalves * 4 << lsh2; i += blockDim.x) {
    const int map = i >> lsh2, line = i - (map << lsh2);
    if (line >= nlines) continue;
    near_bits<kNearSteps>(near + map * near_map(kNearSteps), line,
                          img + (map >> 1) * ximg + line * ls + (map & 1));
  }
  __syncthreads();

  // ---- X into Y: one warp per 32x32 block; lane j holds column distance
  // lb*32+1+j's bits of row distances w*32+1.., a 5-stage butterfly transpose
  // leaves row distance w*32+1+i in lane i (bit j), Y's own order
  const int nblk = nw * nw * 2;
  for (int b0 = warp; b0 < kHalves * nblk; b0 += nwarps) {
    const int hb = kHalves == 2 && b0 >= nblk, b = b0 - hb * nblk;
    const int side = b & 1, lb = (int)((unsigned)(b >> 1) * a.rb >> 16), w = (b >> 1) - lb * nw;
    unsigned *X = img + hb * 2 * ximg, *Y = X + ximg;
    const int line = lb * 32 + 1 + lane;
    unsigned x = line <= roi ? X[line * ls + 2 * w + side] : 0u;
    if (!__any_sync(0xffffffffu, x != 0u)) continue;
    x = warp_transpose(x, lane);
    const int d = w * 32 + 1 + lane;
    if (d <= roi && x) Y[d * ls + 2 * lb + side] |= x;
  }
  __syncthreads();

  // ---- rows out.  A row is one number of 64*nwpr bits, column 0 the highest;
  // the observer's column is bit S, the left string (bit 0 = column distance
  // 1) starts at S+1 and the right one runs downwards from S-1.
  // A thread keeps one word column q, so that its string positions are fixed.
  const int S = 64 * nwpr - 1 - roi;
  auto by_nwpr = [&](int t) { return (int)((unsigned)t * a.rw >> 16); };
  const int per = by_nwpr(blockDim.x);  // rows a pass (blockDim > nwpr)
  const int tr = by_nwpr(tid), q = tid - tr * nwpr, z = 2 * (nwpr - 1 - q);  // bits 32z..32z+63
  const int l0 = 32 * z - (S + 1), r0 = S - 1 - 32 * z - 31;
  const int li = l0 >> 5, ri = r0 >> 5, lsh = l0 & 31, rsh = r0 & 31;
  const bool centre = (S >> 6) == (z >> 1);
  for (int row = wr0 + tr; row < wr1; row += per) {
    if (tid >= per * nwpr) break;
    const int d = abs(row - roi), hb = kHalves == 2 && row > roi;
    const unsigned *X = img + hb * 2 * ximg, *line = X + ximg + d * ls;
    auto at = [&](const unsigned *w, int i) { return (unsigned)i < (unsigned)nw ? w[2 * i] : 0u; };
    const unsigned L0 = at(line + 1, li), L1 = at(line + 1, li + 1), L2 = at(line + 1, li + 2);
    const unsigned R0 = at(line, ri - 1), R1 = at(line, ri), R2 = at(line, ri + 1);
    uint64_t v = ((uint64_t)(__funnelshift_r(L1, L2, lsh) | __brev(__funnelshift_r(R0, R1, rsh)))
                  << 32) |
                 (__funnelshift_r(L0, L1, lsh) | __brev(__funnelshift_r(R1, R2, rsh)));
    if (centre) {
      // the observer's column: image X's line 0, the observer itself (siting.cpp:279)
      const unsigned c = d == 0 ? 1u : (X[2 * ((d - 1) >> 5)] >> ((d - 1) & 31)) & 1u;
      v |= (uint64_t)c << (S & 63);
    }
    dst[row * nwpr + q] = v;
  }
}

// ---- quadrant windows ------------------------------------------------------------

// A quarter of an observer a CTA, for radii whose half windows leave one CTA an
// SM.  The pairs mirror about the quadrant's diagonal: A is x-major, B y-major, so
// one image holds both (A: line = column distance, bit = row distance - 1; B: line
// = row distance, bit = column distance - 1).  The two sides of a row share the word
// of the observer's column, so they form a cluster and the left one hands its bits of
// that word to the right one.  A cluster takes `chunk` halves (2o + lower of observer o)
// in turn.
//
// At radius 200 two CTAs (14 warps) fill an SM: 59% of issue slots, shared-memory
// pipe 64%, a quarter of the warps' time at the barriers between the sweep and the rows
// out.  Reading a group's elevations ahead of the marks before them does not help (1.14
// -> 1.17 ms).
__host__ __device__ __forceinline__ WinGeom quad_geom(int roi) {
  WinGeom g;
  g.w = ((roi + 1 + 7 + 7) & ~7) | 8;
  g.nboxes = (roi + 1 + 255) / 256;
  g.box_rows = g.nboxes == 1 ? roi + 1 : ((roi + g.nboxes) / g.nboxes + 7) & ~7;
  return g;
}

// Words of the image and the two near maps.
__host__ __device__ __forceinline__ int quad_mark_words(int roi, int near) {
  return (roi + 1) * pair_line(roi) + near_map(near) / 2;
}

size_t quad_smem_bytes(int roi, int near) {
  return quad_geom(roi).bytes() + (size_t)(roi + 1) * (16 + 8) + 16 +
         (((size_t)quad_mark_words(roi, near) * 4 + 15) & ~(size_t)15) + 16;
}

constexpr int kQuadMaxThreads = 320;

template <int kNear>
__global__ void __cluster_dims__(2) __launch_bounds__(kQuadMaxThreads, 2)
    shed_quad_kernel(const __grid_constant__ CUtensorMap map, const ShedArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int roi = a.roi, n = a.n, nr = 2 * roi + 1, nwpr = (nr + 63) / 64, nwords = nr * nwpr;
  const bool left = blockIdx.x & 1u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const WinGeom g = quad_geom(roi);
  const int W2 = 2 * g.w, nw = pair_words(roi), ls = pair_line(roi);
  const uint32_t win = smem_u32(sm);
  float4 *tab = reinterpret_cast<float4 *>(sm + g.bytes());
  uint64_t *mbar = reinterpret_cast<uint64_t *>(tab + roi + 1);
  uint64_t *cbuf = mbar + 2;  // the left side's bits of the shared word, by row distance
  unsigned *img = reinterpret_cast<unsigned *>(cbuf + ((roi + 2) & ~1));
  unsigned char *near = reinterpret_cast<unsigned char *>(img + (roi + 1) * ls);
  auto valid = [&](int ob) { return ob >= 0 && ob < n * n; };
  auto load = [&](int item, int ob) {  // the item's window, by one thread
    const int ox = ob / n, oy = ob - ox * n;
    const int hx0 = item & 1 ? ox : ox - roi, hy0 = (left ? oy - roi : oy) & ~7;
    mbar_expect_tx(mbar, (uint32_t)g.bytes());
    for (int b = 0; b < g.nboxes; b++)
      tma_load_window(sm + (size_t)b * g.box_rows * W2, &map, hy0, hx0 + b * g.box_rows, mbar);
  };
  int item = (int)(blockIdx.x >> 1) * a.chunk;
  const int end = min(a.items, item + a.chunk);
  int ob = __ldg(a.obs + (item >> 1));
  if (tid == 0) {
    mbar_init(mbar, 1);
    if (valid(ob)) load(item, ob);
  }
  for (int i = tid; i <= roi; i += blockDim.x) {
    const float y = i ? __frcp_rn((float)i) : 0.f;
    tab[i] = make_float4(y, y, -(float)i, -(float)i);
  }
  unsigned parity = 0;
  for (; item < end; item++) {
    const int half = item & 1, next = item + 1 < end ? __ldg(a.obs + ((item + 1) >> 1)) : -1;
    uint64_t *dst = a.sheds + (size_t)(item >> 1) * nwords;
    if (!valid(ob)) {  // invalid observer: empty shed, flagged (by the whole cluster)
      const int wr0 = half ? roi + 1 : 0, wr1 = half ? nr : roi + 1;
      if (!left)
        for (int i = wr0 * nwpr + tid; i < wr1 * nwpr; i += blockDim.x) dst[i] = 0ull;
      if (tid == 0) {
        atomicOr(a.err, kErrBadInput);
        if (valid(next)) load(item + 1, next);
      }
      ob = next;
      continue;
    }
    const int ox = ob / n, oy = ob - (ob / n) * n;
    const int hx0 = half ? ox : ox - roi;                 // window origin
    const int hy0 = (left ? oy - roi : oy) & ~7;          // TMA inner coordinate: 16-byte aligned
    for (int i = tid; i < (quad_mark_words(roi, kNear) + 3) / 4; i += blockDim.x)
      reinterpret_cast<uint4 *>(img)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    cluster_arrive();  // the peer may write to cbuf once this CTA runs
    if (__all_sync(0xffffffffu, mbar_wait(mbar, parity))) {
      if (const int t = tid; t <= roi) {
        // every second ray, as in the half windows
        const int evens = (roi + 2) / 2, m = t < evens ? 2 * t : 2 * (t - evens) + 1;
        const float sl = fdiv(i2f(m), i2f(roi));
        const int rowlim = half ? n - 1 - ox : ox, collim = left ? oy : n - 1 - oy;
        int kA, kB;
        pair_last(sl, roi, rowlim, collim, collim, rowlim, kA, kB);
        const int rowstep = half ? W2 : -W2, cell = left ? -2 : 2;
        const int p0 = (int)win + (ox - hx0) * W2 + 2 * (oy - hy0);
        PairRays r;
        r.dem = a.dem;
        r.p0 = p0;
        r.mA = r.sB = rowstep;
        r.mB = r.sA = cell;
        r.sl = sl;
        const float nalt = -i2f(elevation<true>(a.dem, p0) + a.oht), tht = i2f(a.tht);
        r.nalt = f2_pack(nalt, nalt);
        const float one = ld_shared_f32(smem_u32(tab + 1));  // RN(1/1)
        r.one = f2_pack(one, one);
        r.img = smem_u32(img);
        r.near = smem_u32(near);
        r.ls4 = 4 * ls;
        r.tab = tab;
        r.hs = f2_pack(kNoHorizon, kNoHorizon);
        r.tht = f2_pack(tht, tht);
        pair_sweep<true, true, kNear>(r, kA, kB);
      }
    } else if (tid == 0) {
      atomicOr(a.err, kErrTmaTimeout);
    }
    parity ^= 1u;
    __syncthreads();
    if (tid == 0 && valid(next)) load(item + 1, next);  // the window is free
    const int nlines = min(roi, kNear) + 1;
    for (int i = tid; i < 2 * nlines; i += blockDim.x) {
      const int map = i >= nlines, line = i - map * nlines;
      near_bits<kNear>(near + map * near_map(kNear), line, img + line * ls + map);
    }
    __syncthreads();
    // A into B, as X into Y above
    for (int b = warp; b < nw * nw; b += nwarps) {
      const int lb = (int)((unsigned)b * a.rb >> 16), w = b - lb * nw, line = lb * 32 + 1 + lane;
      unsigned x = line <= roi ? img[line * ls + 2 * w] : 0u;
      if (!__any_sync(0xffffffffu, x != 0u)) continue;
      x = warp_transpose(x, lane);
      const int d = w * 32 + 1 + lane;
      if (d <= roi && x) img[d * ls + 2 * lb + 1] |= x;
    }
    __syncthreads();
    // rows out (see shed_kernel): this side's words, the shared word by the right one
    const int S = 64 * nwpr - 1 - roi, qc = nwpr - 1 - (S >> 6);
    const int q0 = left ? 0 : qc, nq = left ? qc + 1 : nwpr - qc;
    const int per = blockDim.x / nq, q = q0 + tid % nq, z = 2 * (nwpr - 1 - q);
    const int s0 = left ? 32 * z - (S + 1) : S - 1 - 32 * z - 63, si = s0 >> 5, sh = s0 & 31;
    auto word = [&](int d) {  // the string's 64 bits of word q, row distance d
      const unsigned *line = img + d * ls + 1;
      auto at = [&](int i) { return (unsigned)i < (unsigned)nw ? line[2 * i] : 0u; };
      const unsigned w0 = at(si), w1 = at(si + 1), w2 = at(si + 2);
      const unsigned lo = __funnelshift_r(w0, w1, sh), hi = __funnelshift_r(w1, w2, sh);
      return left ? ((uint64_t)hi << 32) | lo : ((uint64_t)__brev(lo) << 32) | __brev(hi);
    };
    const int r0 = tid / nq + half;  // row distances half..roi
    const bool mine = tid < per * nq;
    __syncwarp();
    cluster_wait();
    if (left && mine) {
      for (int d = r0; d <= roi; d += per) {
        const uint64_t v = word(d);
        if (q == qc)
          cluster_store_u64(smem_u32(cbuf + d), 0, v);
        else
          dst[(half ? roi + d : roi - d) * nwpr + q] = v;
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (!left && mine) {
      for (int d = r0; d <= roi; d += per) {
        uint64_t v = word(d);
        if (q == qc) {
          const unsigned c = d == 0 ? 1u : (img[2 * ((d - 1) >> 5)] >> ((d - 1) & 31)) & 1u;
          v |= cbuf[d] | (uint64_t)c << (S & 63);
        }
        dst[(half ? roi + d : roi - d) * nwpr + q] = v;
      }
    }
    __syncthreads();  // the images are free
    ob = next;
  }
}

constexpr size_t kMaxSmem = 220 * 1024;
constexpr size_t kTwoCtaSmem = 113 * 1024;  // two CTAs of an SM's 228 KB, 1 KB reserved for each

constexpr int kPairMaxThreads = 448;  // the register budget of two CTAs an SM

// Threads of a CTA: a pair of rays each, in even rounds where they are more than
// kPairMaxThreads (the form read through L1 alone).
int pair_threads(int pairs) {
  const int rounds = (pairs + kPairMaxThreads - 1) / kPairMaxThreads;
  return ((pairs + rounds - 1) / rounds + 31) / 32 * 32;
}

ShedPlan shed_l1_plan(int roi) {
  return ShedPlan{pair_threads(2 * roi + 1), false, true, false, false};
}

// Halves where they fit, with a thread for every pair, as a staged CTA sweeps one each.
ShedPlan shed_half_plan(int roi) {
  if (2 * roi + 1 > kPairMaxThreads || pair_smem_bytes(roi, 1, true) > kMaxSmem) return shed_l1_plan(roi);
  return ShedPlan{pair_threads(2 * roi + 1), true, true, false, false};
}

ShedPlan shed_quad_plan(int roi) {
  return ShedPlan{(roi + 1 + 31) / 32 * 32, true, false, true, false};
}

// Radii whose whole windows have more pairs of rays than a warp has lanes, by so few that
// most of a second warp idles, and the observers from which one warp that loops is faster
// (2048^2, 102 400 observers, ms with a thread a ray, a thread a pair, and so: radius 8
// 0.154, 0.222, 0.144; 10 0.205, 0.222, 0.196; 12 0.226, 0.247, 0.209; 15 0.332, 0.247,
// 0.222; 4096 observers of radius 12 16, 17, 17 us, 1024 9, 9, 11).
constexpr int kSmallMinRoi = 8, kSmallMaxRoi = 15, kSmallMinObs = 4096;

// The staged form of a radius.  The SM holds few CTAs of a large window, so the
// window shrinks with the radius (ms at 2048^2, 1.6 G cells of rays; whole, half,
// quarter): roi 30 0.454, 0.484; 60 1.016, 1.021, 1.233; 70 1.018, 1.056, 1.240;
// 90 1.018, 0.987, 0.945; 100 1.032, 0.981, 1.067; 118 -, 0.956, 0.957; 125 -,
// 1.039, 0.904; 140 -, 1.056, 0.962; 200 -, 1.390, 1.138.  From roi 209 quarters
// are one CTA an SM and halves are faster while they fit (212: 1.344, 1.744).
constexpr int kHalfMinRoi = 75, kQuadMinRoi = 119, kOneCtaMinRoi = 209, kOutsideMinRoi = 16;

ShedPlan shed_staged_plan(int roi, bool half) {
  if (roi < 1) return shed_l1_plan(roi);
  if (!half && 4 * roi + 1 <= kPairMaxThreads && pair_smem_bytes(roi, 2, true) <= kMaxSmem)
    return ShedPlan{pair_threads(4 * roi + 1), true, false, false, false};
  const bool quad_fits =
      (roi + 1 + 31) / 32 * 32 <= kQuadMaxThreads && quad_smem_bytes(roi, kNearSteps) <= kMaxSmem;
  if (roi >= kQuadMinRoi && quad_smem_bytes(roi, kNearSteps) <= kTwoCtaSmem)
    return shed_quad_plan(roi);
  const ShedPlan half_plan = shed_half_plan(roi);
  return half_plan.use_smem || !quad_fits ? half_plan : shed_quad_plan(roi);
}

}  // namespace

namespace {

// Steps of a quarter's near maps: 48 where they leave as many CTAs an SM as 16 (ms at
// 2048^2 with 16 and 48: roi 137 0.986, 0.972; 200 1.130, 1.080; 208 1.061, 1.031; at 170
// 48 would cost the third CTA: 0.989, 1.248).
int quad_near(int roi) {
  auto ctas = [&](int steps) { return 228 * 1024 / (quad_smem_bytes(roi, steps) + 1024); };
  return quad_smem_bytes(roi, kFarNearSteps) <= kMaxSmem && ctas(kFarNearSteps) == ctas(kNearSteps)
             ? kFarNearSteps
             : kNearSteps;
}

}  // namespace

size_t shed_smem_bytes(const ShedPlan &p, int roi) {
  return p.quad ? quad_smem_bytes(roi, quad_near(roi)) : pair_smem_bytes(roi, p.half ? 1 : 2, p.use_smem);
}

ShedPlan shed_default_plan(int roi) {
  ShedPlan p = shed_staged_plan(roi, roi >= kHalfMinRoi);
  p.any = p.use_smem;
  return p;
}

namespace {

// Whether the default plan reads a job's windows through L1, where its DEM's row pitch
// allows: staged CTAs of radius 209 and more are alone on their SM, 7 to 14 warps whose
// starts and ends nothing overlaps, and a window that lies mostly outside the DEM is staged
// and cleared for short rays.  Few observers do not fill the SMs: quarters are more CTAs.
// Ms of 4000 observers with one ray a thread through L1, staged, and so: radius 216, 432^2
// 1.23, 1.79, 1.15; 1296^2 1.48, 1.80, 1.23; 260, 1560^2 2.41, 2.53, 1.72; 200, 240^2 0.92,
// 1.01, 0.86; 60, 72^2 0.20, 0.20, 0.11.
bool shed_prefers_l1(int n, int roi, int nsheds, int sms) {
  return nsheds >= sms && (roi >= kOneCtaMinRoi || (roi >= kOutsideMinRoi && 4 * n <= 5 * roi));
}

}  // namespace

int shed_dem_pitch(int nrows, int roi, int nsheds, int sm_count) {
  const int pitch = (nrows + 7) & ~7;
  return pitch % 32 == 0 && nrows < 7 * roi && shed_prefers_l1(nrows, roi, nsheds, sm_count) ? pitch + 8
                                                                                          : pitch;
}

// smem: 1 half windows staged, 2 the whole window staged (as 1 where it does
// not fit), 0 the window read through L1 (as 1 and 2 are where half a window
// does not fit), -1 the default.
ShedPlan shed_plan_for(int roi, int smem) {
  if (smem == 1 || smem == 2) return shed_staged_plan(roi, smem == 1);
  return smem == 0 ? shed_l1_plan(roi) : shed_default_plan(roi);
}

cudaError_t launch_sheds(const DemView &dem, int roi, int oht, int tht, int nsheds,
                         const int32_t *obs, uint64_t *sheds, const ShedPlan &plan, int *d_err,
                         cudaStream_t st) {
  if (nsheds <= 0) return cudaSuccess;
  // radii up to 475: two bit images of a whole shed and a reciprocal a step fit a CTA
  const size_t nr = 2 * (size_t)roi + 1, w32 = (nr + 31) / 32, w64 = (nr + 63) / 64;
  if (4 * (nr * (2 * w64 | 1) + 32 * w32 * (w32 | 1) + roi + 1) + 16 > 227 * 1024)
    return cudaErrorInvalidValue;
  ShedArgs a{dem.data, dem.pitch, dem.nrows, roi, oht, tht, obs, sheds, d_err, 2 * nsheds, 1,
             ~0ull / (unsigned)dem.nrows + 1ull, 65536u / (unsigned)w64 + 1u,
             65536u / (unsigned)pair_words(roi) + 1u};
  // the reciprocal-table division is exhaustively checked for |a| <= 2^21
  // (heights up to 10^6 over 16-bit elevations) and steps up to 2048
  const bool rcp = oht >= 0 && oht <= 1000000;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // a pitch of whole cache lines puts a column's cells at one place of their lines, and
  // lanes on one column then leave theirs together (2048^2, radius 225, 3000 observers:
  // 1.75 ms at a pitch of 2048, 0.98 at 2056)
  const bool l1 = plan.any && dem.pitch % 64 && shed_prefers_l1(dem.nrows, roi, nsheds, sms);
  ShedPlan eff = l1 || (plan.use_smem && !dem.tma_ok) ? shed_l1_plan(roi) : plan;
  if (eff.quad && !rcp) eff = shed_half_plan(roi);  // quarters have no build that divides
  const size_t shm = shed_smem_bytes(eff, roi);
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (eff.use_smem) {
    const WinGeom g = eff.quad ? quad_geom(roi) : win_geom(roi, eff.half ? 1 : 2, true);
    if (!make_dem_tensor_map(&map, dem, g.w, g.box_rows)) return cudaErrorInvalidValue;
  }
  const bool small = rcp && eff.use_smem && !eff.quad && !eff.half && roi >= kSmallMinRoi &&
                     roi <= kSmallMaxRoi && (roi == kSmallMinRoi || nsheds >= kSmallMinObs);
  auto kern = !eff.use_smem ? (rcp ? shed_kernel<1, false, true> : shed_kernel<1, false, false>)
              : eff.quad    ? (quad_near(roi) == kNearSteps ? shed_quad_kernel<kNearSteps>
                                                            : shed_quad_kernel<kFarNearSteps>)
              : eff.half    ? (rcp ? shed_kernel<1, true, true> : shed_kernel<1, true, false>)
              : small       ? shed_kernel<2, true, true, true>
              : rcp         ? shed_kernel<2, true, true>
                            : shed_kernel<2, true, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
  if (e != cudaSuccess) return e;
  const int threads = small ? 32 : eff.threads;
  int grid = nsheds * (eff.half ? 2 : 1);
  if (eff.quad) {
    // One CTA an SM has nothing to run while a window arrives: there a cluster takes up
    // to 4 halves in turn and asks for the next window when the rays of one are done (roi
    // 216 1.69 -> 1.63 ms, 240 1.56 -> 1.46, 300 1.46 -> 1.37), in 8 or more rounds of
    // clusters.  With two CTAs an SM their ends overlap anyhow (200: 1.08, 1.15).
    if (shm > kTwoCtaSmem) a.chunk = std::max(1, std::min(4, a.items / (8 * std::max(1, sms / 2))));
    grid = 2 * ceil_div(a.items, a.chunk);
  }
  kern<<<grid, threads, shm, st>>>(map, a);
  return cudaGetLastError();
}

}  // namespace siting
