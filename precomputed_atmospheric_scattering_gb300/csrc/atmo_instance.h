// atmo_instance.h -- one atmosphere instance as the kernels see it, and the
// work lists that let a single launch cover many instances (batched rebuilds
// of uneven LUT shapes and order counts).
#ifndef ATMO_INSTANCE_H_
#define ATMO_INSTANCE_H_

#include "atmo_device.cuh"

namespace atmo {

// Device buffers of one instance.  All LUTs are float4 RGBA, x fastest, in the
// reference's texture layouts (atmosphere/model.cc:747-766, :872-897).
struct Instance {
  Consts c;
  Shape s;
  Tables tab;
  float4* T;        // transmittance, W_T x H_T
  float4* Tau;      // optical depth -ln(T) of the same texels (internal)
  float4* I;        // irradiance accumulator, W_I x H_I
  float4* dI;       // delta irradiance
  float4* dI2;      // second delta irradiance (odd indirect orders), or nullptr: dI only
  float4* dR;       // delta Rayleigh; also delta multiple scattering (model.cc:897)
  float4* dM;       // delta Mie
  float4* dJ;       // delta scattering density
  float4* S;        // scattering accumulator (RGB + single-Mie red in alpha if combined)
  float4* M;        // single-Mie accumulator, nullptr when combined
  void* S_half;     // half-precision scattering output (half_precision only)
  void* M_half;     // half-precision single-Mie output (half_precision, not combined)
  int combined;     // combine_scattering_textures
  int blend;        // accumulate into I / S / M (wavelength groups after the first)
};

// The delta irradiance of indirect order k (0: the direct pass).  With two
// buffers the indirect pass of order k + 1 writes the other one while the
// density pass of order k + 2 reads this one, so the two can run at once.
ATMO_HD float4* DeltaIrradiance(const Instance& in, int k) {
  return (k & 1) && in.dI2 ? in.dI2 : in.dI;
}

// A launch covers `count` instances; instance inst[q] owns the tiles
// [start[q], start[q+1]).  Both arrays live in device memory.
struct WorkList {
  const int* inst;
  const int* start;
  int count;
  int kinds;   // the instances' KernelKinds bits
};

constexpr int kSmCount = 152;   // of a GB300

// The multiple-scattering kernel of a LUT shape, a bit: 1, the mu_s columns of
// a nu node in one register per lane (MU_S <= 32); 2, in two (MU_S 33 to 64);
// 4, lines in shared memory.  The nodes win unless many lanes idle: kernel 4
// packs a block's threads with columns of up to 4 rows, so that it is the
// nodes' 32 / MU_S x MU_S lanes of 32 against its rows x W of 256.  With three
// nodes nearly every column has clamped nu at both ends, three tasks in all.
// 4 instances of 32 x 128 rows, MU_S x NU, kernel 4 / nodes, ms: 8 x 8 0.287 /
// 0.244, 11 x 8 (22 lanes) 0.438 / 0.360, 19 x 8 0.768 / 0.672, 20 x 4 (20
// lanes, W = 80) 0.364 / 0.391, 32 x 8 0.985 / 0.725, 32 x 3 0.434 / 0.487;
// 33 x 8 1.84 / 1.31, 64 x 8 2.39 / 1.36, 64 x 4 1.018 / 0.803, 40 x 2 0.383 /
// 0.367, 33 x 4 0.751 / 0.773, 33 x 5 0.834 / 0.918, 64 x 3 0.823 / 1.004.
ATMO_HD int MultipleKind(const Shape& s) {
  if (s.snu == 3) return 4;
  if (s.smus <= 32) return 32 / s.smus * s.smus >= 22 || s.sw() > 128 ? 1 : 4;
  return s.smus <= 64 && (s.sw() > 256 || (s.smus >= 40 && s.snu % 2 == 0)) ? 2 : 4;
}

// The scattering-density kernel of a LUT shape above order 2, a bit: arcs, 4
// or 8 nu nodes per warp, or a table lookup per direction.  A warp of the arcs
// is a long chain that needs blocks enough to fill the chip, slabs of (mu,
// mu_s) texels; its lanes are 32 mu rows, of which some idle in the last group
// of an odd MU; and up to 12 nodes the groups of 8 have idle ones, unless they
// are 5 to 8.  One and four instances, lookups / arcs of 4 / of 8, us, by
// slabs x NU: 8192 x 8 35 / 51 / 68 and 96 / 68 / 68; 12288 x 3 47 / 37 / 43, x
// 6 51 / 45 / 59 and 137 / 104 / 80, x 9 90 / 53 / 72 and 209 / 137 / 184;
// 16384 x 8 53 / 51 / 68 and 162 / 127 / 98, x 14 102 / 94 / 94 and 328 / 320 /
// 285; 24576 x 8 96 / 68 / 68 and 252 / 174 / 172; 32768 x 9 154 / 127 / 107
// and 471 / 342 / 354, x 14 190 / 178 / 148 and 632 / 585 / 503; 131072 x 8 281
// / 225 / 184 and 1058 / 800 / 606; MU = 100 (100 lanes of 128): 51200 x 12
// four 705 / 768 / 809, x 16 279 / 340 / 311 and 924 / 1234 / 1026.
constexpr int kDensityArcs4 = 8, kDensityArcs8 = 16, kDensityLookups = 32;
ATMO_HD int DensityKind(const Shape& s) {
  const long long slabs = (long long)s.sr * s.smu * s.smus;
  if (s.snu > 16 || s.iw > 512 || slabs < 12288) return kDensityLookups;
  if (s.snu > 10 && 8 * s.smu < 7 * ((s.smu + 31) / 32 * 32)) return kDensityLookups;
  if (s.snu <= 4 || (s.snu > 8 && s.snu <= 12)) return kDensityArcs4;
  return s.snu > 12 || slabs > 16384 ? kDensityArcs8 : kDensityArcs4;
}

// The single-scattering kernel of a LUT shape, a bit: one, two or four texel
// columns of a row per thread.  Two share a sample's loads and hide each
// other's latency (256 columns, 16 instances: 2.97 ms against 3.20 with one);
// a row of up to 128 columns has only one for each thread (64 columns, one
// instance: 57 us, with two 76), and a row of wide transmittance lines, or of a
// LUT of few rows, wants 256 threads to build the lines (204 columns, lines of
// 339: 100 us against 150; 80 rows of 252 columns: 29 us against 31).  Of 69 shapes
// of 24 to 1024 columns one loses against 16-byte line entries built row by row:
// 442 rows of 64 x 12 columns take 6% longer (18% less on average).
constexpr int kSingleOne = 64, kSingleTwo = 128, kSingleTwoWide = 256, kSingleFour = 512;
constexpr int kSingleOneWide = 1024;   // with kSingleOne: needs 256 threads
ATMO_HD int SingleKind(const Shape& s) {
  if (s.sw() <= 256)
    return s.sw() <= 128 || s.tw > 256 || s.sr * s.smu < 304 ? kSingleOne : kSingleTwo;
  return s.sw() <= 512 ? kSingleTwoWide : kSingleFour;
}
// The bits of a pass's kernels; of `kinds`, as many as the pass launches.
constexpr int kMultipleKinds = 1 | 2 | 4;
constexpr int kDensityKinds = kDensityArcs4 | kDensityArcs8 | kDensityLookups;
constexpr int kSingleKinds = kSingleOne | kSingleTwo | kSingleTwoWide | kSingleFour;
ATMO_HD int KernelKinds(const Shape& s) {
  return MultipleKind(s) | DensityKind(s) | SingleKind(s) |
         (s.sw() > 128 && SingleKind(s) == kSingleOne ? kSingleOneWide : 0);
}

#ifdef __CUDACC__
// Finds the work-list entry holding `tile` (binary search over start[]).
__device__ __forceinline__ int FindEntry(const WorkList& wl, int tile, int* local) {
  int lo = 0, hi = wl.count - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(wl.start + mid) <= tile) lo = mid; else hi = mid - 1;
  }
  *local = tile - __ldg(wl.start + lo);
  return __ldg(wl.inst + lo);
}
#endif

// Threads per block and texels per tile of each kernel (host and device).
constexpr int kTransmittanceLanes = 16;                 // lanes per texel
constexpr int kTransmittanceThreads = 256;
constexpr int kTransmittanceTexelsPerTile = kTransmittanceThreads / kTransmittanceLanes;
constexpr int kHorizonTexelsPerTile = 32 / kTransmittanceLanes;   // one warp's
ATMO_HD int HorizonTiles(const Shape& s) {
  return (s.th + kHorizonTexelsPerTile - 1) / kHorizonTexelsPerTile;
}
constexpr int kTexelThreads = 128;                      // per-texel kernels
constexpr int kIndirectThreads = 128;                   // one warp per texel
constexpr int kIndirectTexelsPerTile = kIndirectThreads / 32;
constexpr int kTableThreads = 128;

}  // namespace atmo

#endif  // ATMO_INSTANCE_H_
