// VIX: approximate visibility index of every DEM cell (siting.cpp:137-198).
//
// Each cell tests `ntests` random targets within roi; a target is visible when
// no sampled ground point on the line of sight (offsets 1,2,4,8,... along the
// major axis) rises above the sight line.  VIX = min(255, (int)(nvis/ntests *
// 255.999f)).
//
// GB300 mapping: one CTA per T x T cell tile.  A window of the DEM around the
// tile is loaded into shared memory by TMA bulk-tensor copies: the whole halo
// (T+2roi rows) while it fits, so that every line-of-sight sample is a
// shared-memory gather, else (large roi) the cells within 64 of the tile, which
// hold the samples at offsets 1..64, and the target itself and the samples at
// offsets 128, 256, ... are read through L1.  Each thread keeps one cell per
// pass and takes every L-th of its targets (L threads a cell); the target of
// item (cell, t) comes from the LCG state after 2t+1 steps from the seed,
// obtained by an affine jump-ahead table instead of a serial chain.  The counts
// become VIX bytes through a host-computed table.
//
// Bound by instruction issue (92-95% of the slots at roi 100).  2048^2, roi
// 100, 100 targets: 157 -> 133 thread instructions a target and 1.894 -> 1.473
// ms (285 G targets/s) with offsets as magnitudes whose signs go with the
// strides (one rounding addend, no sign handling a sample), the samples unrolled
// with one FMA for each scaled sum, the draws doubled modulo 2^32, and 32x32
// instead of 16x16 tiles now that no per-cell table shares the window's memory.
// roi 200, 64 targets: all samples through L1 1.688 ms, the near window staged
// 1.262 ms.
//
// Bit-exactness: every FP32 operation rounds once where the reference's does (an
// FMA only where its product is exact), the reference's drecip = (float)(1.0/d)
// comes from a host table, and C's truncating integer division and
// round-half-away-from-zero are kept.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace siting {
namespace {

// Staged samples of the far form.
constexpr int kFarNear = 7;

// The whole halo staged, also for radii up to 8 (a kernel of its own: as one more case of the
// samples it costs radii up to 32 3%), the cells near the tile, or the tile alone.
constexpr int kStagedForm = 0, kSmallForm = 1, kFarForm = 2, kBareForm = 3, kForms = 4;
constexpr int kSmallRoi = 8;

struct VixArgs {
  const uint16_t *dem;
  int pitch, n, roi, oht, tht, ntests;
  uint8_t *vix;
  int tile, tiles_per_row;
  int halo;  // cells staged around the tile
  int halo_w, box_rows, nboxes;
  const uint32_t *jump;  // ntests pairs: LCG map of 2t+1 steps
  const float *rtab;     // roi+1
  const uint8_t *vtab;   // ntests+1
  int *err;
};

// The staged samples of a sight line, at offsets id = 1, 2, 4, ...: a sample
// rounds slope*id to the minor offset, forms the sight line's height
// oz + id*zslope and takes the cell's height above it; the line is clear when
// the largest of these is not positive (a difference of floats has the exact
// difference's sign).  A lane whose target is nearer than id keeps the
// previous sample's difference, which is counted already.  The offset is at
// least 0 here (signs go with the strides), so adding 2^23 toward zero leaves
// its floor in the low bits, on an idler pipe than a conversion's; the strides'
// share of 2^23's own bits is taken out of the base address.  Scaling by a power
// of two is exact, so one FMA rounds once, as the reference's sum with the
// scaled product does.  Written as one asm statement for its predicated
// subtraction: as comparisons combined in a predicate the compiler spends 13
// instructions a sample instead of 10.
#define VIX_SAMPLE(D, ID, FID)            \
  "setp.gt.s32 p, %1, " ID ";\n\t"       \
  "fma.rn.f32 f, %2, " FID ", %5;\n\t"   \
  "fma.rn.f32 h, %3, " FID ", %4;\n\t"   \
  "add.rz.f32 f, f, 0f4B000000;\n\t"    \
  "mov.b32 o, f;\n\t"                   \
  "mad.lo.s32 t, %7, " ID ", z;\n\t"    \
  "mad.lo.s32 t, o, %8, t;\n\t"         \
  "@p ld.shared.u16 e, [t];\n\t"        \
  "cvt.rn.f32.s32 g, e;\n\t"            \
  "@p sub.rn.f32 " D ", g, h;\n\t"
#define VIX_MAX "max.f32 m, m, d0, d1;\n\t"
#define VIX_SAMPLES(BODY)                                                           \
  asm("{\n\t.reg .pred p;\n\t.reg .f32 f, h, g, m, d0, d1;\n\t.reg .s32 o, t, e, z;\n\t" \
      "mad.lo.s32 z, %8, 0xB5000000, %6;\n\tmov.s32 e, 0;\n\tmov.f32 d0, 0fBF800000;\n\tmov.f32 d1, 0fBF800000;\n\t"      \
      "mov.f32 m, 0fBF800000;\n\t" BODY "max.f32 %0, m, d0, d1;\n\t}"                 \
      : "=f"(over)                                                                  \
      : "r"(ad), "f"(slope), "f"(zslope), "f"(foz), "f"(0x1.fffffep-2f), "r"(ob2), \
        "r"(smaj), "r"(smin))
#define VIX_S1 VIX_SAMPLE("d0", "1", "0f3F800000")
#define VIX_S3                                                                        \
  VIX_S1 VIX_SAMPLE("d1", "2", "0f40000000") VIX_MAX VIX_SAMPLE("d0", "4", "0f40800000")
#define VIX_S5                                                                        \
  VIX_SAMPLE("d0", "1", "0f3F800000") VIX_SAMPLE("d1", "2", "0f40000000") VIX_MAX       \
  VIX_SAMPLE("d0", "4", "0f40800000") VIX_SAMPLE("d1", "8", "0f41000000") VIX_MAX       \
  VIX_SAMPLE("d0", "16", "0f41800000")
#define VIX_S6 VIX_S5 VIX_SAMPLE("d1", "32", "0f42000000")
#define VIX_S7 VIX_S6 VIX_MAX VIX_SAMPLE("d0", "64", "0f42800000")
#define VIX_S8 VIX_S7 VIX_SAMPLE("d1", "128", "0f43000000")

template <int kNear>
__device__ __forceinline__ int near_samples(int ad, float slope, float zslope, float foz,
                                            uint32_t ob2, int smaj, int smin) {
  float over;
  if constexpr (kNear == 1) VIX_SAMPLES(VIX_S1);
  if constexpr (kNear == 3) VIX_SAMPLES(VIX_S3);
  if constexpr (kNear == 5) VIX_SAMPLES(VIX_S5);
  if constexpr (kNear == 6) VIX_SAMPLES(VIX_S6);
  if constexpr (kNear == 7) VIX_SAMPLES(VIX_S7);
  if constexpr (kNear == 8) VIX_SAMPLES(VIX_S8);
  return !(over > 0.f);
}

// What a thread keeps of its cell.
struct VixCell {
  uint32_t ob2;  // shared-memory byte address of the cell in the window
  int ctz;       // tht - observer height
  float foz;     // observer height
  uint32_t seed;
  int ox, oy, gbase;  // DEM coordinates and element offset
};

// One random target of one cell (siting.cpp:155-175 and 54-135).  kInterior:
// every cell of the tile is at least roi from the DEM edge, so no target can
// fall outside it and the bounds test is dropped.  kNear: samples at offsets
// 1 .. 2^(kNear-1) are read from the staged window.  kFar: the target itself
// and the samples beyond are read from the DEM through L1.
template <int kNear, bool kFar, bool kInterior>
__device__ __forceinline__ int vix_target(const VixArgs &a, const VixCell &c, int W2, int roi2,
                                          unsigned long long span2, uint2 j, const float *rtab) {
  // Both draws (siting.cpp:29-33) are carried doubled, modulo 2^32: the
  // reference's modulus 2^31 then needs no masking, and a float of the doubled
  // draw is twice the draw's (span arrives scaled by 2^-32).
  const uint32_t r1 = j.x * c.seed + j.y;
  const uint32_t r2 = 1103515245u * r1 + 2u * 12345u;
  // (int)((2*roi+0.99999f)*r/RANDOM_MAX): the divisor is 2^31, and scaling
  // by a power of two commutes with rounding (no overflow or underflow
  // here), so RN(span*r)/2^31 = RN((span*2^-31)*r).  The products are in
  // [0, 2^23): adding 2^23 toward zero leaves their floor in the low bits.
  const unsigned long long dd = f2_mul(span2, f2_pack(__uint2float_rn(r1), __uint2float_rn(r2)));
  const unsigned long long fl = f2_add_rz(dd, f2_pack(8388608.f, 8388608.f));
  const int dx = __float_as_int(f2_lo(fl)) - (0x4b000000 + a.roi);
  const int dy = __float_as_int(f2_hi(fl)) - (0x4b000000 + a.roi);
  const bool fold = dx * dx + dy * dy > roi2;  // fold into the circle (siting.cpp:162-166)
  unsigned adx = abs(dx), ady = abs(dy);
  if (kFar) {
    if (fold) {
      adx /= 3u;
      ady /= 3u;
    }
  } else {  // |v| / 3 = |v| * 43691 >> 17 for |v| < 2^16 (a staged window's roi is far smaller)
    const unsigned m = fold ? 43691u : 131072u;
    adx = (adx * m) >> 17;
    ady = (ady * m) >> 17;
  }
  if (!kInterior) {
    const int x = c.ox + (dx < 0 ? -(int)adx : (int)adx), y = c.oy + (dy < 0 ? -(int)ady : (int)ady);
    if ((unsigned)x >= (unsigned)a.n || (unsigned)y >= (unsigned)a.n) return 0;
  }
  // From here on offsets are magnitudes and the signs go with the strides:
  // slope, rounding and products are symmetric about zero.
  const int sx = dx < 0 ? -W2 : W2, sy = dy < 0 ? -2 : 2;
  int ev;
  if constexpr (kFar) {
    const int gx = dx < 0 ? -(int)adx : (int)adx, gy = dy < 0 ? -(int)ady : (int)ady;
    ev = __ldg(a.dem + (c.gbase + gx * a.pitch + gy));
  } else {
    asm("ld.shared.u16 %0, [%1];"
        : "=r"(ev)
        : "r"(c.ob2 + (uint32_t)((int)adx * sx) + (uint32_t)((int)ady * sy)));
  }
  const bool mx = adx >= ady;
  const int ad = mx ? adx : ady, am = mx ? ady : adx;
  const int smaj = mx ? sx : sy, smin = mx ? sy : sx;
  // Sample offsets are id = 1, 2, 4, ... along the major axis.  slope*id =
  // m*drecip*id = (m*drecip)*id exactly (scaling by a power of two), likewise
  // id*zslope, so both start from m*|drecip| and (tz-oz)*|drecip| and are
  // bit-identical to the reference's products (siting.cpp:91).
  const float r = rtab[ad];
  const float slope = fmul(i2f(am), r), zslope = fmul(i2f(ev + c.ctz), r);
  // every staged sample is tested: a blocked target's lane would idle until
  // its warp's other lanes finish anyway
  int vis = 1;
  if constexpr (kNear > 0) vis = near_samples<kNear>(ad, slope, zslope, c.foz, c.ob2, smaj, smin);
  if constexpr (kFar) {
    if (ad > (1 << kNear) && vis) {
      const int P = a.pitch;
      const int gmaj = mx ? (dx < 0 ? -P : P) : (dy < 0 ? -1 : 1);
      const int gmin = mx ? (dy < 0 ? -1 : 1) : (dx < 0 ? -P : P);
      for (int id = 1 << kNear; id < ad; id <<= 1) {
        const float fid = i2f(id);
        const float f = __fmaf_rn(slope, fid, 0x1.fffffep-2f);
        const float h = __fmaf_rn(zslope, fid, c.foz);
        if (i2f(__ldg(a.dem + (c.gbase + id * gmaj + f2i(f) * gmin))) > h) return 0;
      }
    }
  }
  return vis;
}

// The tile's (cell, target) items: L = blockDim/T^2 consecutive threads share
// a cell (T = 16: 4) and take every L-th of its targets, so a thread keeps one
// cell for the whole pass (no per-item bookkeeping) and a warp's lanes run the
// same number of targets; the L partial counts are summed by shuffles.
template <int kNear, bool kFar, bool kInterior>
__device__ __forceinline__ void vix_tile_work(const VixArgs &a, const uint16_t *halo, int tx0,
                                              int ty0, int hx0, int hy0, const uint2 *jump,
                                              const float *rtab, const uint8_t *vtab) {
  const int T = a.tile, ncell = T * T;
  const int L = max(1, (int)blockDim.x / ncell);  // a power of two: tiles are 16, 32, 64
  const int per_pass = blockDim.x / L;
  const float span = fmul(fadd(i2f(2 * a.roi), 0.99999f), 0x1p-32f);  // of doubled draws
  const unsigned long long span2 = f2_pack(span, span);
  const int roi2 = a.roi * a.roi;
  const int W2 = 2 * a.halo_w;
  const int sub = threadIdx.x & (L - 1);
  const uint32_t win = smem_u32(halo);
  for (int c0 = 0; c0 < ncell; c0 += per_pass) {
    const int cell = c0 + threadIdx.x / L;
    const int lx = cell / T, ly = cell - lx * T;
    VixCell c;
    c.ox = tx0 + lx;
    c.oy = ty0 + ly;
    const bool in = cell < ncell && c.ox < a.n && c.oy < a.n;
    int acc = 0;
    if (in) {
      const int at = (c.ox - hx0) * a.halo_w + (c.oy - hy0);
      const int oz = halo[at] + a.oht;
      c.ob2 = win + 2u * (uint32_t)at;
      c.ctz = a.tht - oz;
      c.foz = i2f(oz);
      c.seed = (uint32_t)(c.ox * a.n + c.oy);  // the cell index (siting.cpp:150, r = tid)
      c.gbase = c.ox * a.pitch + c.oy;
#pragma unroll 1  // unrolled, the copies crowd the 32 registers (4096^2: 7.24 vs 7.02 ms)
      for (int t = sub; t < a.ntests; t += L)
        acc += vix_target<kNear, kFar, kInterior>(a, c, W2, roi2, span2, jump[t], rtab);
    }
    for (int o = 1; o < L; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (in && sub == 0) a.vix[c.ox * a.n + c.oy] = vtab[acc];
  }
}

// One T x T tile of cells: `map` is the window's tensor map, `tile` the
// tile's index (row-major over tiles_per_row^2), `sm` the CTA's dynamic
// shared memory (vix_smem_bytes), `mbar` the window's mbarrier (shared
// memory).  Every thread of the CTA calls it.
template <int kForm>
__device__ __forceinline__ void vix_tile(const CUtensorMap *map, const VixArgs &a, int tile,
                                         unsigned char *sm, uint64_t *mbar) {
  const int T = a.tile;
  const int tx0 = (tile / a.tiles_per_row) * T;
  const int ty0 = (tile % a.tiles_per_row) * T;
  const int hx0 = tx0 - a.halo;
  const int hy0 = (ty0 - a.halo) & ~7;  // TMA inner coordinate: 16-byte aligned
  size_t off = 0;
  uint16_t *halo = reinterpret_cast<uint16_t *>(sm);
  const uint32_t halo_bytes = (uint32_t)a.nboxes * a.box_rows * a.halo_w * 2u;
  off += halo_bytes + 16;  // (the per-tile kernel's mbarrier)
  uint2 *jump = reinterpret_cast<uint2 *>(sm + off);
  off += (size_t)a.ntests * 8;
  float *rtab = reinterpret_cast<float *>(sm + off);
  off += (size_t)(a.roi + 1) * 4;
  uint8_t *vtab = sm + off;

  if (threadIdx.x == 0) {
    mbar_init(mbar, 1);
    mbar_expect_tx(mbar, halo_bytes);
    for (int b = 0; b < a.nboxes; b++)
      tma_load_window(halo + (size_t)b * a.box_rows * a.halo_w, map, hy0, hx0 + b * a.box_rows,
                      mbar);
  }
  for (int i = threadIdx.x; i < a.ntests; i += blockDim.x)  // doubled draws (vix_target)
    jump[i] = make_uint2(2u * a.jump[2 * i], 2u * a.jump[2 * i + 1]);
  for (int i = threadIdx.x; i <= a.roi; i += blockDim.x) rtab[i] = a.rtab[i];
  for (int i = threadIdx.x; i <= a.ntests; i += blockDim.x) vtab[i] = a.vtab[i];
  __syncthreads();

  // targets lie within roi of their cell (after the fold, |dx|,|dy| <= roi)
  const bool interior = tx0 >= a.roi && ty0 >= a.roi && tx0 + T + a.roi <= a.n &&
                        ty0 + T + a.roi <= a.n;
  if (!mbar_wait(mbar, 0)) {
    if (threadIdx.x == 0) atomicOr(a.err, kErrTmaTimeout);
    return;
  }
  auto work = [&](auto near) {
    constexpr int kNear = decltype(near)::value;
    constexpr bool kFar = kForm == kFarForm || kForm == kBareForm;
    if (interior)
      vix_tile_work<kNear, kFar, true>(a, halo, tx0, ty0, hx0, hy0, jump, rtab, vtab);
    else
      vix_tile_work<kNear, kFar, false>(a, halo, tx0, ty0, hx0, hy0, jump, rtab, vtab);
  };
  if constexpr (kForm == kBareForm) {
    work(std::integral_constant<int, 0>());
  } else if constexpr (kForm == kFarForm) {
    work(std::integral_constant<int, kFarNear>());
  } else if constexpr (kForm == kSmallForm) {
    if (a.roi <= 2)
      work(std::integral_constant<int, 1>());
    else
      work(std::integral_constant<int, 3>());
  } else {  // the fewest samples that reach offsets below roi
    if (a.roi <= 32)
      work(std::integral_constant<int, 5>());
    else if (a.roi <= 64)
      work(std::integral_constant<int, 6>());
    else if (a.roi <= 128)
      work(std::integral_constant<int, 7>());
    else
      work(std::integral_constant<int, 8>());
  }
}

template <int kForm>
__global__ void __launch_bounds__(1024, 2) vix_kernel(const __grid_constant__ CUtensorMap map,
                                                     const VixArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  const uint32_t halo_bytes = (uint32_t)a.nboxes * a.box_rows * a.halo_w * 2u;
  vix_tile<kForm>(&map, a, blockIdx.x, sm, reinterpret_cast<uint64_t *>(sm + halo_bytes));
}

// ---- VIX of many jobs in one launch (batched form) ---------------------------
// One grid covers the (job, tile) items of many jobs, so a job's last tiles
// overlap the next job's first ones instead of each job ending a grid of its
// own.  The job table travels as the kernel's parameters, and a CTA finds its
// job from its index: every value derived from the table is then the same in
// all threads and is read from the constant bank, as in the one-job kernel.

struct VixQJob {
  CUtensorMap map;  // window map
  VixArgs a;
  unsigned first;   // grid index of the job's first tile
};

struct VixQTable {
  VixQJob jobs[kStageQueueMaxJobs];
  int njobs;
};
static_assert(sizeof(VixQTable) <= 32000, "kernel parameters are limited to 32 KB");

// One CTA per (job, tile) item, all of one form: one kernel per form keeps each within
// 32 registers a thread.
template <int kForm>
__global__ void __launch_bounds__(1024, 2) vixq_kernel(const __grid_constant__ VixQTable tab) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t mbar;
  const unsigned it = blockIdx.x;
  int lo = 0, hi = tab.njobs - 1;  // the last job whose first tile is at or before `it`
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tab.jobs[mid].first <= it)
      lo = mid;
    else
      hi = mid - 1;
  }
  const VixQJob &J = tab.jobs[lo];
  vix_tile<kForm>(&J.map, J.a, (int)(it - J.first), sm, &mbar);
}

int round8(int v) { return (v + 7) & ~7; }

// Samples of the near window of the far form: offsets 1..64, so the window
// reaches kFarHalo cells around the tile.
constexpr int kFarHalo = 1 << (kFarNear - 1);
// Targets a cell up to which not even that window pays: the tile alone is staged (us at
// radius 120, 1 and 2 targets: 1000^2 26.7 and 30.8 with
// the window, 20.8 and 26.8 without).
constexpr int kBareTests = 2;

// Two 1024-thread CTAs share an SM when each takes at most half of its 228 KB
// shared memory (at most 32 registers a thread); the second CTA fills the
// issue slots that the first leaves while its warps drain at the end of a tile.
constexpr size_t kVixTwoCtaSmem = 112 * 1024;
constexpr size_t kVixMaxSmem = 220 * 1024;

struct HaloGeom {
  int w, box_rows, nboxes;
  size_t bytes() const { return (size_t)nboxes * box_rows * w * 2; }
};

// mbarrier, jump table, reciprocals, VIX bytes
size_t tables_tail_bytes(int roi, int ntests) {
  return 16 + (size_t)ntests * 8 + (size_t)(roi + 1) * 4 + ntests + 1;
}

int vix_form(const VixPlan &p, int roi) {
  if (p.use_smem) return roi <= kSmallRoi ? kSmallForm : kStagedForm;
  return p.bare ? kBareForm : kFarForm;
}

int plan_halo(const VixPlan &p, int roi) { return p.use_smem ? roi : p.bare ? 0 : kFarHalo; }

// The window of a tile: its columns start at a multiple of 8 at or before the
// halo's first (tiles start at multiples of 16).
HaloGeom halo_geom(const VixPlan &p, int roi, int ntests) {
  const int halo = plan_halo(p, roi), h = p.tile + 2 * halo;
  HaloGeom g;
  g.w = round8(h + (-halo & 7));
  g.nboxes = (h + 255) / 256;
  // boxes after the first start on 128 bytes
  g.box_rows = g.nboxes == 1 ? h : round8((h + g.nboxes - 1) / g.nboxes);
  // A row pitch of an odd multiple of 4 words starts nearby rows in distinct
  // banks (2048^2, roi 100: 387 M -> 310 M shared-memory wavefronts), unless
  // the wider rows cost the second CTA of an SM.
  HaloGeom o = g;
  o.w |= 8;
  const size_t tail = tables_tail_bytes(roi, ntests);
  return g.bytes() + tail <= kVixTwoCtaSmem && o.bytes() + tail > kVixTwoCtaSmem ? g : o;
}

}  // namespace

size_t vix_table_bytes(int roi, int ntests) {
  return (((size_t)ntests * 8 + (size_t)(roi + 1) * 4 + ntests + 1) + 15) & ~(size_t)15;
}

void vix_fill_tables(void *host_buf, int roi, int ntests) {
  uint32_t *jump = static_cast<uint32_t *>(host_buf);
  const uint32_t a = 1103515245u, c = 12345u;
  uint32_t A = a, C = c;  // map of 1 step
  for (int t = 0; t < ntests; t++) {
    jump[2 * t] = A;  // map of 2t+1 steps
    jump[2 * t + 1] = C;
    A = a * (a * A);  // advance by two steps
    C = a * (a * C + c) + c;
  }
  float *rtab = reinterpret_cast<float *>(jump + 2 * ntests);
  rtab[0] = 0.f;
  for (int d = 1; d <= roi; d++) rtab[d] = (float)(1.0 / d);  // siting.cpp:91
  uint8_t *vtab = reinterpret_cast<uint8_t *>(rtab + roi + 1);
  for (int v = 0; v <= ntests; v++) {
    const float f = (float)v / ntests;  // siting.cpp:186-189
    const int q = (int)(f * 255.999f);
    vtab[v] = (uint8_t)(q < 255 ? q : 255);
  }
}

size_t vix_smem_bytes(const VixPlan &p, int roi, int ntests) {
  return tables_tail_bytes(roi, ntests) + halo_geom(p, roi, ntests).bytes();
}

// 32x32 tiles (one cell a thread) with the whole halo staged are fastest where
// two CTAs share an SM, then 16x16 (four threads a cell), whose halo takes
// longer to load for a quarter of the cells: 2048^2, roi 96, staged 16x16 takes
// 0.32 ms + 12.2 us a target, 32x32 with the near window alone 0.04 ms + 16.1
// us, so few targets take the far form (16x16 over it at 64 and 72 targets: 1024^2, radius
// 100, 1.00, 0.97; 2001^2, 105, 1.01, 0.99; 3000^2, 110, 1.01, 0.99).  64x64 tiles (four cells a thread)
// never won.  A grid of 32x32 tiles that is not two waves of the SMs' CTA
// pairs leaves SMs idle: 16x16 tiles then (us at 32 and 16, 256^2 roi 20: 23,
// 15; 400^2 roi 200: 100, 69; 700^2 roi 200: 198, 176; 1000^2 roi 50: 187, 207),
// unless the targets are so few that four threads a cell and four halos for one cost
// more, an eighth of the tiles (roi 45: 300^2, 8 targets 14.6, 16.8, 16 18.6, 19.7, 32
// 27.3, 26.0; 700^2, 16 46.9, 57.1, 32 77.6, 79.6, 64 142, 128).
VixPlan vix_default_plan(int nrows, int roi, int ntests, int sm_count) {
  const int t32 = (nrows + 31) / 32;
  const bool few = t32 * t32 < 4 * sm_count && 8 * ntests >= t32 * t32;
  const VixPlan s32{32, 1024, true, false}, s16{16, 1024, true, false};
  if (!few && vix_smem_bytes(s32, roi, ntests) <= kVixTwoCtaSmem) return s32;
  if ((few || ntests >= 72) && vix_smem_bytes(s16, roi, ntests) <= kVixTwoCtaSmem) return s16;
  return VixPlan{few ? 16 : 32, 1024, false, ntests <= kBareTests};
}

VixPlan vix_plan_for(int nrows, int roi, int ntests, int tile, int smem, int sm_count) {
  VixPlan p = vix_default_plan(nrows, roi, ntests, sm_count);
  if (tile == 16 || tile == 32 || tile == 64) {
    p.tile = tile;
    p.use_smem = smem != 0;
    p.bare = false;
    if (p.use_smem &&
        (halo_geom(p, roi, ntests).w > 2048 || vix_smem_bytes(p, roi, ntests) > kVixMaxSmem))
      p.use_smem = false;
  } else if (smem == 0) {
    p.use_smem = false;
  }
  return p;
}

namespace {

// Kernel arguments and halo map of one job; false if the map cannot be made.
bool vix_args(const DemView &dem, int roi, int oht, int tht, int ntests, uint8_t *vix,
              const void *d_tables, const VixPlan &plan, int *d_err, VixArgs *out,
              CUtensorMap *map) {
  // the radii whose tables of 8 bytes an entry fit a CTA
  if ((size_t)roi * 8 + (size_t)ntests * 9 + 5200 > 227 * 1024) return false;
  VixArgs a{};
  a.dem = dem.data;
  a.pitch = dem.pitch;
  a.n = dem.nrows;
  a.roi = roi;
  a.oht = oht;
  a.tht = tht;
  a.ntests = ntests;
  a.vix = vix;
  a.tile = plan.tile;
  a.tiles_per_row = ceil_div(dem.nrows, plan.tile);
  a.jump = static_cast<const uint32_t *>(d_tables);
  a.rtab = reinterpret_cast<const float *>(a.jump + 2 * ntests);
  a.vtab = reinterpret_cast<const uint8_t *>(a.rtab + roi + 1);
  a.err = d_err;
  a.halo = plan_halo(plan, roi);
  const HaloGeom g = halo_geom(plan, roi, ntests);
  a.halo_w = g.w;
  a.box_rows = g.box_rows;
  a.nboxes = g.nboxes;
  *out = a;
  return make_dem_tensor_map(map, dem, g.w, g.box_rows);
}

}  // namespace

cudaError_t launch_vix(const DemView &dem, int roi, int oht, int tht, int ntests, uint8_t *vix,
                       const void *d_tables, const VixPlan &plan, int *d_err, cudaStream_t st) {
  VixArgs a;
  CUtensorMap map;
  if (!vix_args(dem, roi, oht, tht, ntests, vix, d_tables, plan, d_err, &a, &map))
    return cudaErrorInvalidValue;
  const size_t shm = vix_smem_bytes(plan, roi, ntests);
  const int grid = a.tiles_per_row * a.tiles_per_row;
  const int form = vix_form(plan, roi);
  auto kern = form == kStagedForm  ? vix_kernel<kStagedForm>
              : form == kSmallForm ? vix_kernel<kSmallForm>
              : form == kFarForm   ? vix_kernel<kFarForm>
                                   : vix_kernel<kBareForm>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
  if (e != cudaSuccess) return e;
  kern<<<grid, plan.threads, shm, st>>>(map, a);
  return cudaGetLastError();
}

cudaError_t launch_vix_queue(const StageJob *jobs, int njobs, cudaStream_t st) {
  // one launch for the jobs of each form, at most kStageQueueMaxJobs jobs a launch
  static thread_local VixQTable tab;  // 20 KB: not on the host stack
  for (int kind = 0; kind < kForms; kind++) {
    int j = 0;
    while (j < njobs) {
      tab.njobs = 0;
      size_t shm = 0;
      unsigned total = 0;
      for (; j < njobs && tab.njobs < kStageQueueMaxJobs; j++) {
        const StageJob &J = jobs[j];
        VixQJob &q = tab.jobs[tab.njobs];
        memset(&q, 0, sizeof(q));
        if (vix_form(J.vplan, J.roi) != kind) continue;
        if (!vix_args(J.dem, J.roi, J.oht, J.tht, J.ntests, J.vix, J.vix_tables, J.vplan, J.err,
                      &q.a, &q.map))
          return cudaErrorInvalidValue;
        q.first = total;
        shm = std::max(shm, vix_smem_bytes(J.vplan, J.roi, J.ntests));
        total += (unsigned)(q.a.tiles_per_row * q.a.tiles_per_row);
        tab.njobs++;
      }
      if (!tab.njobs) continue;
      auto kern = kind == kStagedForm  ? vixq_kernel<kStagedForm>
                  : kind == kSmallForm ? vixq_kernel<kSmallForm>
                  : kind == kFarForm   ? vixq_kernel<kFarForm>
                                       : vixq_kernel<kBareForm>;
      cudaError_t e =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
      if (e != cudaSuccess) return e;
      kern<<<total, 1024, shm, st>>>(tab);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace siting
