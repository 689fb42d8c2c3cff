// atmo_fast.cu -- fast-path kernels: the slab-restructured scattering density
// (the dominant pass, functions.glsl:1163-1260), the row-restructured single
// and multiple scattering (:650-730, :1285-1330; described where they start
// below), the FP16 output conversion and the FP32 FMA throughput probe.
//
// Scattering density, restructured.  For a texel at r-slice k and mu_s column
// c, every incoming-radiance lookup of ComputeScatteringDensity is made at the
// texel's own r and mu_s, whose texture coordinates land on the centres of
// slice k and column c (the texel mapping and the lookup mapping are inverse
// to each other), while mu = cos(theta_l) takes one of 16 values shared by
// all texels of the slice and only nu varies with the direction.  A block
// therefore owns the slab (k, c) -- the NU x MU texels with that r and mu_s --
// and stages in shared memory, per theta row l and nu node n, the previous
// order's radiance bilinearly interpolated in mu: L[l][n].  The quadrilinear
// lookup of a direction reduces to a lerp between L[l][n0] and L[l][n0 + 1].
// The ground term reads the bottom row of the irradiance LUT (the ground
// point is at r = Rb, on row 0's centre), also staged in shared memory.
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "atmo_kernels.h"
#include "atmo_passes.cuh"

namespace atmo {

constexpr int kDensityFastThreads = 256;


// Piecewise-linear functions staged in shared memory.  A row of N node
// values L[0..N-1] (node coordinate v in [0, N - 1]) is stored as N + 1
// entries, each the line a + b s of one interval in the unit coordinate
// s = (v + 0.5) / N: entry 0 is L[0] (v < 0), entry N is L[N - 1] (v >
// N - 1), entry e in between the segment [e - 1, e] (b = the slope times N).
// A lookup takes s from a saturating FMA, which clamps it to [0, 1] and maps
// a NaN to 0, then the entry from a second FMA: s N + 1.5 x 2^23, rounded to
// nearest, leaves round(v + 0.5), in [0, N], in the sum's low mantissa bits
// (a v on a node may take either neighbouring entry; both give the node's
// value).  The sum's bit pattern, times the entry size, plus a row offset
// that cancels the constant's exponent bits (mod 2^32), is the entry's
// shared-memory address: no index can leave the row, and the value is one
// FMA per channel.  The intercept's cancellation costs at most ~n ulp of the
// node values (n < 128).
constexpr float kRoundMagic = 12582912.0f;
constexpr uint32_t kRoundMagicBits = 0x4B400000u;

// One entry: a.xyz, b.x | b.y, b.z, -, - at order 2; above order 2 (packed)
// a.xy, b.xy | a.z, b.z, -, -, the x, y channels as aligned register pairs
// for the packed FP32x2 FMA.
constexpr int kNodeBytes = 32;
// One order-2 entry, the Rayleigh and the Mie lines in 48 bytes:
// aR.xyz, bR.x | bR.yz, aM.xy | aM.z, bM.xyz.  The 48-byte stride also puts
// the 8 entries of a 16-bank span on disjoint banks.
constexpr int kPairBytes = 48;

// Three channels as a register pair (x, y) and a scalar (z) for the packed
// FP32x2 instructions (per component the same IEEE operations as fmaf and
// fadd, so the sums are bit-identical to the scalar ones).  Above order 2 the
// packed FMAs and adds of the lookups and sums save ~3% of the kernel's time.
// At order 2 they do not pay, although they save 11% of the instructions: a
// packed FMA holds the FMA pipe for two slots or more (9.8 ms per launch
// against 9.0), only the packed products are free.
struct P3 {
  float2 xy;
  float z;
};
__device__ __forceinline__ float2 Dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ P3 ToP3(F3 a) { return P3{make_float2(a.x, a.y), a.z}; }
__device__ __forceinline__ F3 ToF3(P3 a) { return F3{a.xy.x, a.xy.y, a.z}; }
__device__ __forceinline__ F3 ToF3(F3 a) { return a; }
__device__ __forceinline__ P3 Fma(P3 a, P3 b, P3 c) {
  return P3{__ffma2_rn(a.xy, b.xy, c.xy), fmaf(a.z, b.z, c.z)};
}
__device__ __forceinline__ P3 Add(P3 a, P3 b) { return P3{__fadd2_rn(a.xy, b.xy), a.z + b.z}; }

// Approximate reciprocal square root, square root and division that flush
// subnormal operands to zero (the PTX .approx.ftz forms).  The non-flushing
// forms that rsqrtf, sqrtf under --prec-sqrt=false and __fdividef compile to
// add a range check and a rescaling of subnormal operands to every call.
// Every operand given to these below is zero, a normal number or negative
// (where both forms return NaN); on normal operands of the ranges used here
// the two forms agree bit for bit (16.7 M operands per range compared on a
// GB300).  Single and multiple scattering take 4.5% and 3.8% less time; their
// LUTs are not bit-identical to the non-flushing build's (the code around the
// calls is scheduled and contracted differently) and meet the same bounds.
__device__ __forceinline__ float RsqrtFtz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float SqrtFtz(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float DivFtz(float a, float b) {
  float y;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// a b + c clamped to [0, 1], NaN to 0 (one FMA with the .sat modifier).
__device__ __forceinline__ float FmaSat(float a, float b, float c) {
  float d;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

#ifdef ATMO_DEVICE_CHECKS
// The checked build's test of a table lookup: the `bytes` at shared address
// a lie within the block's dynamic shared memory, else the lookup reads its
// first bytes.
extern __shared__ float4 atmo_fast_dynamic_smem[];
__device__ __forceinline__ uint32_t CheckedShared(uint32_t a, int bytes) {
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(atmo_fast_dynamic_smem);
  uint32_t size;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(size));
  return base + (uint32_t)ATMO_CHECKED_INDEX(kCheckSharedLookup, a - base,
                                             (long long)size - bytes + 1);
}
#endif

template <int kOffset>
__device__ __forceinline__ float4 LoadShared4(uint32_t addr) {
#ifdef ATMO_DEVICE_CHECKS
  addr = CheckedShared(addr + kOffset, 16) - kOffset;
#endif
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr), "n"(kOffset));
  return v;
}
template <int kOffset>
__device__ __forceinline__ F3 LoadShared3(uint32_t addr) {
#ifdef ATMO_DEVICE_CHECKS
  addr = CheckedShared(addr + kOffset, 12) - kOffset;
#endif
  F3 v;
  asm volatile("ld.shared.f32 %0, [%3+%4];\n\tld.shared.f32 %1, [%3+%5];\n\t"
               "ld.shared.f32 %2, [%3+%6];"
               : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z)
               : "r"(addr), "n"(kOffset), "n"(kOffset + 4), "n"(kOffset + 8));
  return v;
}
template <int kOffset>
__device__ __forceinline__ float2 LoadShared2(uint32_t addr) {
#ifdef ATMO_DEVICE_CHECKS
  addr = CheckedShared(addr + kOffset, 8) - kOffset;
#endif
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(addr), "n"(kOffset));
  return v;
}
// The line a + b s of entry e (0 <= e <= N) of a row of N node values v[].
__device__ __forceinline__ void EntryLine(const float4* v, int e, int N, F3* a, F3* b) {
  if (e == 0 || e == N) {
    const float4 p = v[e == 0 ? 0 : N - 1];
    *a = F3{p.x, p.y, p.z};
    *b = f3(0.0f);
    return;
  }
  const float4 p = v[e - 1], q = v[e];
  const F3 d{q.x - p.x, q.y - p.y, q.z - p.z};
  const float c = 0.5f - float(e);   // -(n + 0.5) for the segment n = e - 1
  *a = fma3(d, c, F3{p.x, p.y, p.z});
  *b = d * float(N);
}
template <bool kPacked>
__device__ __forceinline__ void StoreLine(float4* entry, F3 a, F3 b) {
  if (kPacked) {
    entry[0] = make_float4(a.x, a.y, b.x, b.y);
    entry[1] = make_float4(a.z, b.z, 0.0f, 0.0f);
  } else {
    entry[0] = make_float4(a.x, a.y, a.z, b.x);
    entry[1] = make_float4(b.y, b.z, 0.0f, 0.0f);
  }
}
// Entry e (0 <= e <= N) of a row of N node values v[0..N-1].
template <bool kPacked>
__device__ __forceinline__ void StoreEntry(float4* entry, const float4* v, int e, int N) {
  F3 a, b;
  EntryLine(v, e, N, &a, &b);
  StoreLine<kPacked>(entry, a, b);
}
// Entry e of a row of N Rayleigh values r[] and Mie values m[] (order 2).
__device__ __forceinline__ void StorePairEntry(float4* entry, const float4* r, const float4* m,
                                               int e, int N) {
  float4 a[2], b[2];
  StoreEntry<false>(a, r, e, N);
  StoreEntry<false>(b, m, e, N);
  entry[0] = a[0];
  entry[1] = make_float4(a[1].x, a[1].y, b[0].x, b[0].y);
  entry[2] = make_float4(b[0].z, b[0].w, b[1].x, b[1].y);
}
// The staged function at the unit coordinate s, t = fmaf(s, N, kRoundMagic),
// of the table whose entries (kStride bytes apart, the function's at byte
// kOffset) start at row_adj + kRoundMagicBits kStride.
template <int kStride, int kOffset>
__device__ __forceinline__ F3 EvalNodes(float s, float t, uint32_t row_adj) {
  const uint32_t a = (uint32_t)__float_as_int(t) * (uint32_t)kStride + row_adj;
  const float4 p = LoadShared4<kOffset>(a);
  const float2 q = LoadShared2<kOffset + 16>(a);
  return F3{fmaf(s, p.w, p.x), fmaf(s, q.x, p.y), fmaf(s, q.y, p.z)};
}
// The line of the packed entry at shared address a, at s.
__device__ __forceinline__ P3 PackedLine(float s, uint32_t a) {
  const float4 p = LoadShared4<0>(a);
  const float2 q = LoadShared2<16>(a);
  return P3{__ffma2_rn(Dup(s), make_float2(p.z, p.w), make_float2(p.x, p.y)), fmaf(s, q.y, q.x)};
}
// EvalNodes for a packed table of kNodeBytes entries.
__device__ __forceinline__ P3 EvalNodesPacked(float s, float t, uint32_t row_adj) {
  return PackedLine(s, (uint32_t)__float_as_int(t) * (uint32_t)kNodeBytes + row_adj);
}
// Both lines of an order-2 entry (kPairBytes apart).
__device__ __forceinline__ void EvalPair(float s, float t, uint32_t row_adj, F3* ray, F3* mie) {
  const uint32_t a = (uint32_t)__float_as_int(t) * (uint32_t)kPairBytes + row_adj;
  const float4 p = LoadShared4<0>(a), q = LoadShared4<16>(a), r = LoadShared4<32>(a);
  *ray = F3{fmaf(s, p.w, p.x), fmaf(s, q.x, p.y), fmaf(s, q.y, p.z)};
  *mie = F3{fmaf(s, r.y, q.z), fmaf(s, r.z, q.w), fmaf(s, r.w, r.x)};
}
// magic: kRoundMagic, as a run-time value.  With the constant in sight the
// compiler merges it with the loads' offsets into terms too large for a load's
// immediate and adds each to the address: one more instruction per load (3 of
// 34 per sample at order 2, whose 16-instance launch took 9.08 ms, now 8.47).
__device__ __forceinline__ uint32_t RowAdjust(uint32_t base, int stride, float magic) {
  return base - (uint32_t)__float_as_int(magic) * (uint32_t)stride;
}

// Ground rows above order 2.  On a theta row whose directions hit the ground
// the incoming radiance is the sky line (entry i, in s) plus tg times the
// irradiance line (entry j, in the ground coordinate x = gs s + go), and on
// each (i, j) pair their sum is one line in s.  A merged table of (NU + 1) x J
// entries per row (J = the ground entries the row can reach) turns the ground
// lookup into a second index: x and its entry come from the same saturating
// and rounding FMAs as the separate lookup, monotone in s, so the entries
// reached lie between those of s = 0 and s = 1 and no index leaves the table.
// Rows are merged in theta order while their tables fit the budget; the
// others keep the separate lookups.
struct MergeRow {
  float gs, go;       // x = gs s + go (the same values build and read the table)
  uint32_t adj;       // address adjustment of the row's table
  uint32_t jstride;   // J x kNodeBytes; 0 when the row is not merged
};
// Above order 2 a block is limited to 2 per SM by its registers, so its
// shared memory may grow to ~99 KB (opted in above the default 48 KB) at no
// cost in occupancy.
constexpr int kDensityMaxSmem = 99 * 1024;

// Shared memory of one block, bytes, without the merged tables: [16][NU + 1]
// entries (the previous order interpolated in mu at the slab's r and mu_s;
// at order 2 a Rayleigh and a Mie line each), the bottom row of the
// irradiance LUT as [IW + 1] entries, a float4 staging value per node, and
// above order 2 the merge rows' descriptors and the merged entry count.
__host__ __device__ inline int DensityBaseSmem(const Shape& s, int order) {
  const int species = order == 2 ? 2 : 1;
  const int nodes = kDensityThetaSamples * s.snu;
  const int entries = kDensityThetaSamples * (s.snu + 1);
  return entries * (order == 2 ? kPairBytes : kNodeBytes) + (s.iw + 1) * kNodeBytes +
         (species * nodes + s.iw) * 16 +
         (order == 2 ? 0 : kDensityThetaSamples * (int)(sizeof(MergeRow) + sizeof(int4)) + 16);
}
// The merged tables a block of the instance may need above order 2, bytes:
// the largest r-slice's sum over its ground rows of (NU + 1) J entries, with
// J bounded from the ray's distance to the ground (the FP64 geometry of the
// set-up tables at the slice's r and cos(theta_l), plus a margin for the
// rounding of both ends).  Only a budget: rows that do not fit it keep the
// separate sky and ground lookups.
int DensityMergeNeed(const Shape& s, const Consts& c) {
  const double Rb = c.dRb, H = c.dH, pi = 3.14159265358979323846;
  const double k1 = double(s.snu - 1) / (2.0 * s.snu), kg = double(s.iw - 1) / (2.0 * s.iw);
  int worst = 0;
  for (int k = 0; k < s.sr; ++k) {
    const double rho = H * k / double(s.sr > 1 ? s.sr - 1 : 1);
    const double r = std::sqrt(rho * rho + Rb * Rb);
    int entries = 0;
    for (int l = 0; l < kDensityThetaSamples; ++l) {
      const double mu = std::cos((l + 0.5) * pi / kDensityThetaSamples);
      const double disc = r * r * (mu * mu - 1.0) + Rb * Rb;
      if (mu >= 0.0 || disc < 0.0) continue;
      const double gs = kg * (-r * mu - std::sqrt(disc)) / (Rb * k1);
      const int J = std::min((int)std::floor(gs * s.iw) + 3, s.iw + 1);
      entries += (s.snu + 1) * J;
    }
    worst = std::max(worst, entries);
  }
  return worst * kNodeBytes;
}
// Shapes whose order-2 tables (the larger) fit the default 48 KB per block;
// the others take the plain density kernel.
bool DensityFastFits(const Shape& s) { return DensityBaseSmem(s, 2) <= 48 * 1024; }

// Texels of one mu row that a thread integrates together: they share the
// outgoing direction's phase functions (4 at every order: at order 2, 128
// registers and 2 blocks per SM beat 2 texels at 80 registers and 3 blocks
// by ~3%).
template <bool kOrder2>
__host__ __device__ constexpr int DensityTexelsPerTask() { return 4; }

// A block's tasks (a mu row and up to 4 of its texels each) go to its threads
// in rounds of 256.  The tasks of the last round, where they are at most half
// as many (in whole warps), are split into parts of the 16 theta rows, whose
// sums are added in order through shared memory: a slab of half the
// reference's size has 64 tasks, which kept 2 of a block's 8 warps busy (order
// 2, one such instance 86 -> 49 us, 8 of them 545 -> 293; 70 shapes of 16
// to 250 mu rows and 3 to 15 nodes: 19% less time).
__host__ __device__ inline int DensityTasks(const Shape& s) { return s.smu * ((s.snu + 3) / 4); }
__host__ __device__ inline int DensityLastRound(const Shape& s) {
  return DensityTasks(s) % kDensityFastThreads;
}
__host__ __device__ inline int DensityParts(const Shape& s, int order) {
  const int last = DensityLastRound(s), warps = (last + 31) / 32;
  if (last == 0 || warps > kDensityFastThreads / 64) return 1;
  const int parts = kDensityFastThreads / 32 / warps;
  return DensityBaseSmem(s, order) + parts * last * 4 * (int)sizeof(F3) <= 48 * 1024 ? parts : 1;
}
// The parts' sums, bytes (a multiple of 16).
__host__ __device__ inline int DensityPartSmem(const Shape& s, int order) {
  const int parts = DensityParts(s, order);
  return parts > 1 ? parts * DensityLastRound(s) * 4 * (int)sizeof(F3) : 0;
}

// The outgoing direction's phase functions and the scattering coefficients
// fold into one weight per channel and direction, shared by the task's 4
// texels (one mu row: one altitude), so a texel keeps one sum.
template <bool kOrder2>
struct DensityTask {
  static constexpr int kN = DensityTexelsPerTask<kOrder2>();
  using V = std::conditional_t<kOrder2, F3, P3>;   // packed above order 2
  float sx[kN], sy[kN];   // the sun's x, y
  V sum[kN];              // sums of L (a_R P_R(nu2) + a_M P_M(nu2)) dw
};

// Ground rows at order 2: the irradiance seen along a theta row is linear in
// s on nearly every row (the directions reach one irradiance interval), or has
// one kink; then it needs no lookup, and its sum over the two sides of a phi
// pair no more than their s: base + slope (s0 + s1) + bend (max(s0 - kink, 0)
// + max(s1 - kink, 0)) (base twice the line's).  More intervals: lookups.
// The lookups were 18% of the kernel's shared-memory wavefronts and 6 of 38
// instructions per sample; without them the 16-instance launch at the
// reference's shape takes 9.08 ms instead of 10.31.
enum GroundForm { kNoGround, kGroundLine, kGroundKink, kGroundLookup };
struct __align__(16) GroundRow {
  F3 base;
  int form;
  F3 slope;
  float kink;
  F3 bend;
  float pad;
};

// The 32 phi samples of theta row l for the texels of one task.  Everything
// is in the unit coordinate s = 1/2 + k1 nu1 (k1 = (NU - 1) / (2 NU)) of the
// staged rows: A is s's part 1/2 + k1 mu_s cos(theta_l), hs = k1 sin(theta_l)
// scales the direction's cos(phi), sin(phi), so a side's coordinate is one
// FMA with the sun's sx or sy and the ground lookup's coordinate another
// (g_scale, g_off map s to the irradiance row's unit coordinate); order 2
// recovers nu1 = (s - 1/2) / k1 for its phase functions.  war, wam: the
// scattering coefficients at the texel times the phase constants and dw.
// kMerged (ground rows above order 2): the row's merged table (MergeRow)
// replaces the sky and ground lookups.
template <bool kOrder2, int kForm, bool kMerged = false>
__device__ __forceinline__ void DensityThetaRow(DensityTask<kOrder2>& task,
                                                const Consts& c, float A, float hs, float B,
                                                float oxs, F3 war, F3 wam, float fnu,
                                                float inv_k1, float magic, uint32_t row_adj, F3 tg,
                                                float g_scale, float g_off, float fiw,
                                                uint32_t ir_adj, uint32_t jstride = 0,
                                                uint32_t madj = 0,
                                                const GroundRow* ground = nullptr) {
  constexpr bool kGround = kForm == kGroundLookup;
  static_assert(!kMerged || (kGround && !kOrder2), "merged tables: ground rows above order 2");
  [[maybe_unused]] F3 g_base = f3(0.0f), g_slope = f3(0.0f), g_bend = f3(0.0f);
  [[maybe_unused]] float g_kink = 0.0f;
  if constexpr (kForm == kGroundLine || kForm == kGroundKink) {
    g_base = ground->base;
    g_slope = ground->slope;
    if constexpr (kForm == kGroundKink) {
      g_bend = ground->bend;
      g_kink = ground->kink;
    }
  }
  constexpr int kDensityTexelsPerTask = DensityTexelsPerTask<kOrder2>();
  [[maybe_unused]] const float m2g = c.m2g, g2p1 = c.g2p1;
  // phi and 2 pi - phi share cos(phi), hence nu2 and the phase functions of
  // the outgoing direction; nu1 differs by the sign of sy sin(phi).  Unrolled
  // 4 times above order 2, twice at order 2 (8.27 ms per 16-instance launch
  // against 8.47; 4 times overflows the instruction cache: 9.38).
#pragma unroll(kOrder2 ? 2 : 4)
  for (int m = 0; m < kDensityPhiSamples / 2; ++m) {
    const float2 cs = c_density_phi[m];
    // Phase functions at nu2 (functions.glsl:739-747, :1245-1254), folded
    // with the scattering coefficients into one weight per channel.
    const float nu2 = fmaf(oxs, cs.x, B);
    const float q2 = fmaf(nu2, nu2, 1.0f);
    // 1 + g^2 - 2 g nu2 >= (1 - g)^2: zero or normal for |g| < 1.
    const float rs = RsqrtFtz(fmaf(m2g, nu2, g2p1));
    const F3 wf = fma3(wam, q2 * (rs * rs * rs), war * q2);
    const float hc = cs.x * hs, hn = cs.y * hs;
#pragma unroll
    for (int q = 0; q < kDensityTexelsPerTask; ++q) {
      // The unit coordinate of nu1: bu +- sy sin(theta) sin(phi) / 2.
      const float bu = fmaf(task.sx[q], hc, A);
      const float2 u2 =
          make_float2(FmaSat(hn, task.sy[q], bu), FmaSat(-hn, task.sy[q], bu));
      if constexpr (kOrder2) {
        // Single scattering with its phase functions at nu1 (:998-1004):
        // (1 + nu1^2) (R 3/(16 pi) + M k_M / (1 + g^2 - 2 g nu1)^(3/2)),
        // with the constant factors staged into the tables.
        const float n0 = fmaf(u2.x, inv_k1, -0.5f * inv_k1);
        const float n1 = fmaf(u2.y, inv_k1, -0.5f * inv_k1);
        const float2 r1 = make_float2(RsqrtFtz(fmaf(m2g, n0, g2p1)), RsqrtFtz(fmaf(m2g, n1, g2p1)));
        const float2 r3 = __fmul2_rn(__fmul2_rn(r1, r1), r1);
        F3 Ls;
        if constexpr (kForm == kGroundLine || kForm == kGroundKink) {
          Ls = fma3(g_slope, u2.x + u2.y, g_base);
          if constexpr (kForm == kGroundKink)
            Ls = fma3(g_bend, fmaxf(u2.x - g_kink, 0.0f) + fmaxf(u2.y - g_kink, 0.0f), Ls);
        }
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const float u = side == 0 ? u2.x : u2.y, nu1 = side == 0 ? n0 : n1;
          F3 L, M;
          EvalPair(u, fmaf(u, fnu, magic), row_adj, &L, &M);
          const F3 L1 = fma3(M, side == 0 ? r3.x : r3.y, L);
          const float q1 = fmaf(nu1, nu1, 1.0f);
          Ls = side == 0 && (kForm == kNoGround || kGround) ? L1 * q1 : fma3(L1, q1, Ls);
          if (kGround) {
            // Ground bounce: the ground point is at radius Rb, so the cosine
            // of its normal with the sun is (r mu_s + dist nu1) / Rb; the
            // irradiance lookup at r = Rb reads row 0 of the LUT.
            const float x = FmaSat(u, g_scale, g_off);
            Ls = fma3(tg, EvalNodes<kNodeBytes, 0>(x, fmaf(x, fiw, magic), ir_adj), Ls);
          }
        }
        task.sum[q] = fma3(Ls, wf, task.sum[q]);
      } else {
        // Ls is seeded with the first side's radiance (an explicit 0 + x
        // would cost an add per channel: IEEE keeps it).
        P3 Ls;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const float u = side == 0 ? u2.x : u2.y, t = fmaf(u, fnu, magic);
          if constexpr (kMerged) {
            // Entry (i, j) of the merged table: one line in s for sky + ground.
            const float x = FmaSat(u, g_scale, g_off);
            const uint32_t a = (uint32_t)__float_as_int(t) * jstride +
                               (uint32_t)__float_as_int(fmaf(x, fiw, magic)) *
                                   (uint32_t)kNodeBytes +
                               madj;
            const P3 L = PackedLine(u, a);
            Ls = side == 0 ? L : Add(Ls, L);
            continue;
          }
          const P3 L = EvalNodesPacked(u, t, row_adj);
          Ls = side == 0 ? L : Add(Ls, L);
          if (kGround) {
            // The ground bounce, as at order 2.
            const float x = FmaSat(u, g_scale, g_off);
            Ls = Fma(ToP3(tg), EvalNodesPacked(x, fmaf(x, fiw, magic), ir_adj), Ls);
          }
        }
        task.sum[q] = Fma(Ls, ToP3(wf), task.sum[q]);
      }
    }
  }
}

template <bool kOrder2>
__global__ void __launch_bounds__(kDensityFastThreads)
k_density_fast(const Instance* __restrict__ insts, WorkList wl, int order, int smem_bytes,
               float magic) {
  extern __shared__ float4 smem[];
  constexpr int kSpecies = kOrder2 ? 2 : 1;
  constexpr int kStride = kOrder2 ? kPairBytes : kNodeBytes;
  constexpr int kDensityTexelsPerTask = DensityTexelsPerTask<kOrder2>();
  int local;
  const Instance& in = insts[FindEntry(wl, blockIdx.x, &local)];
  if (!kOrder2 && DensityKind(in.s) != kDensityLookups) return;
  const Shape s = in.s;
  const int NU = s.snu, W = s.sw();
  const int k = local / s.smus, col = local % s.smus;
  const int nodes = kDensityThetaSamples * NU;
  const int row_entries = NU + 1;
  float4* E = smem;                                            // [16][NU + 1] entries
  float4* G = E + kDensityThetaSamples * row_entries * (kStride / 16);
  float4* V = G + (s.iw + 1) * (kNodeBytes / 16);              // [species][16][NU], [IW] values
  constexpr int kSmemOrder = kOrder2 ? 2 : 3;
  F3* part_sums = reinterpret_cast<F3*>(V + kSpecies * nodes + s.iw);
  // Above order 2: the merge rows, their table layout (offset, J, j0, size in
  // entries; size 0 when not merged) and the merged tables.
  MergeRow* meta = reinterpret_cast<MergeRow*>(V + kSpecies * nodes + s.iw +
                                               DensityPartSmem(s, kSmemOrder) / 16);
  int4* build = reinterpret_cast<int4*>(meta + kDensityThetaSamples);
  int& merged_entries = *reinterpret_cast<int*>(build + kDensityThetaSamples);
  float4* X = reinterpret_cast<float4*>(build + kDensityThetaSamples + 1);
  const DensityRow* drows = in.tab.drows + k * kDensityThetaSamples;
  const Consts& c = in.c;
  const TexelCol cc = in.tab.cols[col];
  const float fnu = float(NU), fiw = float(s.iw);
  // s = 1/2 + k1 nu1 on the sky rows, 1/2 + kg mu_g on the irradiance row.
  const float k1 = float(NU - 1) / (2.0f * fnu), kg = float(s.iw - 1) / (2.0f * fiw);
  const float inv_k1 = 1.0f / k1, inv_rb = 1.0f / c.Rb;

  // Node values: the previous order (Rayleigh or multiple, then Mie at order
  // 2) at column n MU_S + col of slice k, bilinear in mu; then the irradiance.
  const int staged = kSpecies * nodes + s.iw;
  for (int e = threadIdx.x; e < staged; e += blockDim.x) {
    float4 v;
    if (e < kSpecies * nodes) {
      const int sp = e / nodes, ne = e - sp * nodes;
      const int l = ne / NU, n = ne - l * NU;
      const float Y = drows[l].u_mu * float(s.smu) - 0.5f;
      const float fy = floorf(Y);
      const float wy = Y - fy;
      const int y0 = ClampIdx((int)fy, s.smu), y1 = ClampIdx((int)fy + 1, s.smu);
      const float4* src =
          (kOrder2 && sp == 1 ? in.dM : in.dR) + k * s.smu * W + n * s.smus + col;
#ifdef ATMO_DEVICE_CHECKS
      const long long o = src - (kOrder2 && sp == 1 ? in.dM : in.dR), nS = s.s_texels();
      const float4 a = __ldg(src - o + ATMO_CHECKED_INDEX(kCheckDensityStage, o + y0 * W, nS));
      const float4 b = __ldg(src - o + ATMO_CHECKED_INDEX(kCheckDensityStage, o + y1 * W, nS));
#else
      const float4 a = __ldg(src + y0 * W), b = __ldg(src + y1 * W);
#endif
      // At order 2 the single-scattering tables carry their phase constants.
      const float scale = kOrder2 ? (sp == 1 ? in.c.mie_k : in.c.ray_k) : 1.0f;
      v = make_float4(fmaf(wy, b.x - a.x, a.x) * scale, fmaf(wy, b.y - a.y, a.y) * scale,
                      fmaf(wy, b.z - a.z, a.z) * scale, 0.0f);
    } else {
      v = __ldg(DeltaIrradiance(in, order - 2) + (e - kSpecies * nodes));
    }
    V[e] = v;
  }
  if (!kOrder2 && threadIdx.x < kDensityThetaSamples) {
    // Row l's ground coordinate and the ground entries j0..j1 it can reach.
    const int l = threadIdx.x;
    const DensityRow dr = drows[l];
    MergeRow mr{0.0f, 0.0f, 0u, 0u};
    int4 b = make_int4(0, 0, 0, 0);
    if (dr.ground) {
      // The ground point's mu_g = (r mu_s + dist nu1) / Rb: its irradiance
      // coordinate 1/2 + kg mu_g is w0 + kg dist (s - 1/2) / (k1 Rb).
      const float w0 = fmaf(in.tab.rows[k * s.smu].r * cc.mu_s * inv_rb, kg, 0.5f);
      mr.gs = kg * dr.dist_ground * inv_rb * inv_k1;
      mr.go = fmaf(-0.5f, mr.gs, w0);
      const int j0 = __float_as_int(fmaf(FmaSat(0.0f, mr.gs, mr.go), fiw, kRoundMagic)) -
                     (int)kRoundMagicBits;
      const int j1 = __float_as_int(fmaf(FmaSat(1.0f, mr.gs, mr.go), fiw, kRoundMagic)) -
                     (int)kRoundMagicBits;
      if (j1 >= j0) b = make_int4(0, j1 - j0 + 1, j0, (NU + 1) * (j1 - j0 + 1));
    }
    meta[l] = mr;
    build[l] = b;
  }
  __syncthreads();
  if (!kOrder2 && threadIdx.x == 0) {
    // Table offsets, rows in theta order while they fit the budget.
    // The budget: the launch's shared memory beyond this instance's tables.
    const int budget =
        max(smem_bytes - DensityBaseSmem(s, 3) - DensityPartSmem(s, 3), 0) / kNodeBytes;
    const uint32_t xbase = (uint32_t)__cvta_generic_to_shared(X);
    int off = 0;
    for (int l = 0; l < kDensityThetaSamples; ++l) {
      int4 b = build[l];
      if (b.w > 0 && off + b.w <= budget) {
        b.x = off;
        const uint32_t js = (uint32_t)(b.y * kNodeBytes);
        meta[l].jstride = js;
        // Entry (i, j) at X + off + i J + (j - j0), addressed from the two
        // rounding sums (magic + i, magic + j).
        meta[l].adj = xbase + (uint32_t)(off * kNodeBytes) - kRoundMagicBits * js -
                      (kRoundMagicBits + (uint32_t)b.z) * (uint32_t)kNodeBytes;
        off += b.w;
      } else {
        b.w = 0;
      }
      build[l] = b;
    }
    merged_entries = off;
  }
  __syncthreads();
  const int sky_entries = kDensityThetaSamples * row_entries;
  const int base_entries = sky_entries + s.iw + 1;
  const int total_entries = base_entries + (kOrder2 ? 0 : merged_entries);
  for (int e = threadIdx.x; e < total_entries; e += blockDim.x) {
    if (e < sky_entries) {
      const int l = e / row_entries, i = e - l * row_entries;
      if (kOrder2) {
        StorePairEntry(E + e * (kPairBytes / 16), V + l * NU, V + nodes + l * NU, i, NU);
      } else {
        StoreEntry<true>(E + e * (kNodeBytes / 16), V + l * NU, i, NU);
      }
    } else if (e < base_entries) {
      const int i = e - sky_entries;
      StoreEntry<!kOrder2>(G + i * (kNodeBytes / 16), V + kSpecies * nodes, i, s.iw);
    } else if (!kOrder2) {
      // Merged entry (i, j) of row l: sky line + tg (ground line at gs s + go).
      const int m = e - base_entries;
      int l = 0;
      while (l < kDensityThetaSamples - 1 && !(build[l].w > 0 && m < build[l].x + build[l].w)) ++l;
      const int4 b = build[l];
      const int idx = m - b.x, i = idx / b.y, j = b.z + (idx - i * b.y);
      F3 sa, sb, ga, gb;
      EntryLine(V + l * NU, i, NU, &sa, &sb);
      EntryLine(V + nodes, j, s.iw, &ga, &gb);
      const F3 tg = f3(drows[l].t_ground);
      const MergeRow mr = meta[l];
      StoreLine<true>(X + m * (kNodeBytes / 16), fma3(tg, fma3(gb, mr.go, ga), sa),
                fma3(tg, gb * mr.gs, sb));
    }
  }
  __syncthreads();

  // Order 2: the ground rows' forms, in place of the node values.
  GroundRow* grounds = reinterpret_cast<GroundRow*>(V);
  if (kOrder2 && threadIdx.x < kDensityThetaSamples) {
    const DensityRow dr = drows[threadIdx.x];
    GroundRow g;
    g.base = g.slope = g.bend = f3(0.0f);
    g.kink = g.pad = 0.0f;
    g.form = dr.ground ? kGroundLookup : kNoGround;
    if (dr.ground) {
      // The irradiance entries reached from s = 1/2 + k1 (mu_s cos(theta) -+
      // sin_s sin(theta)).
      const float gs = kg * dr.dist_ground * inv_rb * inv_k1;
      const float go = fmaf(-0.5f, gs, fmaf(in.tab.rows[k * s.smu].r * cc.mu_s * inv_rb, kg, 0.5f));
      const float mid = fmaf(cc.mu_s * dr.cos_t, k1, 0.5f), half = k1 * dr.sin_t * cc.sin_s;
      const int j0 = __float_as_int(fmaf(FmaSat(mid - half, gs, go), fiw, kRoundMagic)) -
                     (int)kRoundMagicBits;
      const int j1 = __float_as_int(fmaf(FmaSat(mid + half, gs, go), fiw, kRoundMagic)) -
                     (int)kRoundMagicBits;
      if (j1 <= j0 + 1) {
        const float4* e0 = G + j0 * (kNodeBytes / 16);
        const float4* e1 = G + j1 * (kNodeBytes / 16);
        const F3 tg = f3(dr.t_ground);
        const F3 a{e0[0].x, e0[0].y, e0[0].z}, b{e0[0].w, e0[1].x, e0[1].y};
        g.base = tg * fma3(b, go, a) * 2.0f;
        g.slope = tg * b * gs;
        g.form = kGroundLine;
        if (j1 > j0) {
          // Entries j0 and j0 + 1 meet at node j0: (j0 + 1/2) / IW.
          g.form = kGroundKink;
          g.bend = tg * (F3{e1[0].w, e1[1].x, e1[1].y} - b) * gs;
          g.kink = ((float(j0) + 0.5f) / fiw - go) / gs;
        }
      }
    }
    grounds[threadIdx.x] = g;
  }
  if (kOrder2) __syncthreads();

  const float dtdp = (kPiF / 16.0f) * (kPiF / 16.0f);
  const uint32_t e_base = (uint32_t)__cvta_generic_to_shared(E);
  const uint32_t ir_adj = RowAdjust((uint32_t)__cvta_generic_to_shared(G), kNodeBytes, magic);
  const int tasks = DensityTasks(s), last = DensityLastRound(s);
  const int parts_last = DensityParts(s, kSmemOrder);
  for (int first = 0; first < tasks; first += kDensityFastThreads) {
    const int parts = tasks - first == last ? parts_last : 1;
    const int part = parts > 1 ? (int)threadIdx.x / ((last + 31) & ~31) : 0;
    const int id = (int)threadIdx.x - part * ((last + 31) & ~31), ti = first + id;
    if (part >= parts || ti >= tasks) break;
    const int j = ti % s.smu, n0 = (ti / s.smu) * kDensityTexelsPerTask;
    const TexelRow row = in.tab.rows[k * s.smu + j];
    DensityTask<kOrder2> task;
#pragma unroll
    for (int q = 0; q < kDensityTexelsPerTask; ++q) {
      const TexelAngles ang = MakeAngles(s, row, cc, min(n0 + q, NU - 1));
      task.sx[q] = ang.sx;
      task.sy[q] = ang.sy;
      task.sum[q] = typename DensityTask<kOrder2>::V{};
    }
    // The scattering coefficients at the texel, with the phase constants.
    const F3 a_r = c.rayleigh * (ProfileDensity(c.prof_r, row.h) * c.ray_k);
    const F3 a_m = c.mie_sca * (ProfileDensity(c.prof_m, row.h) * c.mie_k);
    // Order 2: the ground point's mu_g = (r mu_s + dist nu1) / Rb; its
    // irradiance coordinate 1/2 + kg mu_g is w0 + kg dist nu1 / Rb.
    const float w0 = fmaf(row.r * cc.mu_s * inv_rb, kg, 0.5f);
    const int l_end = (part + 1) * kDensityThetaSamples / parts;
    for (int l = part * kDensityThetaSamples / parts; l < l_end; ++l) {
      const DensityRow dr = drows[l];
      const float B = row.mu * dr.cos_t;
      const float oxs = row.omega_x * dr.sin_t;
      const float dw = dtdp * dr.sin_t;
      // In the unit coordinate of nu1 (see DensityThetaRow).
      const float A = fmaf(cc.mu_s * dr.cos_t, k1, 0.5f);
      const float hs = k1 * dr.sin_t;
      const uint32_t row_adj =
          RowAdjust(e_base + (uint32_t)(l * row_entries * kStride), kStride, magic);
      if constexpr (kOrder2) {
        const GroundRow* g = grounds + l;
        if (g->form == kGroundLine) {
          DensityThetaRow<kOrder2, kGroundLine>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu,
                                                inv_k1, magic, row_adj, f3(0.0f), 0.0f, 0.0f, fiw, ir_adj,
                                                0, 0, g);
        } else if (g->form == kGroundKink) {
          DensityThetaRow<kOrder2, kGroundKink>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu,
                                                inv_k1, magic, row_adj, f3(0.0f), 0.0f, 0.0f, fiw, ir_adj,
                                                0, 0, g);
        } else if (g->form == kGroundLookup) {
          // The ground point's irradiance coordinate from s = 1/2 + k1 nu1:
          // w0 + kg dist (s - 1/2) / (k1 Rb).
          const float gs = kg * dr.dist_ground * inv_rb * inv_k1;
          const float go = fmaf(-0.5f, gs, w0);
          DensityThetaRow<kOrder2, kGroundLookup>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu,
                                                  inv_k1, magic, row_adj, f3(dr.t_ground), gs, go, fiw,
                                                  ir_adj);
        } else {
          DensityThetaRow<kOrder2, kNoGround>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu,
                                              inv_k1, magic, row_adj, f3(0.0f), 0.0f, 0.0f, fiw, ir_adj);
        }
      } else if (dr.ground) {
        const MergeRow mr = meta[l];
        if (mr.jstride != 0) {
          DensityThetaRow<kOrder2, kGroundLookup, true>(
              task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu, inv_k1, magic, row_adj, f3(0.0f), mr.gs,
              mr.go, fiw, ir_adj, mr.jstride, mr.adj);
        } else {
          DensityThetaRow<kOrder2, kGroundLookup>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu,
                                                  inv_k1, magic, row_adj, f3(dr.t_ground), mr.gs, mr.go,
                                                  fiw, ir_adj);
        }
      } else {
        DensityThetaRow<kOrder2, kNoGround>(task, c, A, hs, B, oxs, a_r * dw, a_m * dw, fnu, inv_k1,
                                            magic, row_adj, f3(0.0f), 0.0f, 0.0f, fiw, ir_adj);
      }
    }
#pragma unroll
    for (int q = 0; q < kDensityTexelsPerTask; ++q) {
      const F3 J = ToF3(task.sum[q]);
      if (parts > 1) {
        part_sums[(part * last + id) * kDensityTexelsPerTask + q] = J;
      } else if (n0 + q < NU) {
        in.dJ[(k * s.smu + j) * W + (n0 + q) * s.smus + col] = to4(J, 1.0f);
      }
    }
  }
  if (parts_last == 1) return;
  __syncthreads();
  for (int e = threadIdx.x; e < last * kDensityTexelsPerTask; e += kDensityFastThreads) {
    const int ti = tasks - last + e / kDensityTexelsPerTask;
    const int j = ti % s.smu, n = ti / s.smu * kDensityTexelsPerTask + e % kDensityTexelsPerTask;
    F3 J = part_sums[e];
    for (int part = 1; part < parts_last; ++part)
      J += part_sums[part * last * kDensityTexelsPerTask + e];
    if (n < NU) in.dJ[(k * s.smu + j) * W + n * s.smus + col] = to4(J, 1.0f);
  }
}

// ---------------------------------------------------------------------------
// Scattering density above order 2, by arcs.
//
// A texel of the slab (k, c) is its row's mu and the azimuth alpha of its sun
// about the zenith.  On theta row l the incoming radiance is a function of
// x = cos(phi - alpha) alone, piecewise linear in x with a kink at each nu
// node (and, on ground rows, at each irradiance node) in range: a base line
// plus delta_e max(x - kappa_e, 0) per kink.  The outgoing phase functions
// P(phi_m) depend on the row and theta only.  A texel's sum over the 32
// directions of a theta row is therefore, per kink, the sum of P (x - kappa)
// over the directions with |phi - alpha| < psi = acos(kappa): a contiguous
// arc, whose sums of P, P cos(phi) and P sin(phi) are differences of two
// prefix sums (x = cos(alpha) cos(phi) + sin(alpha) sin(phi)).  Four kinks
// (the reference's NU = 8) replace 32 lookups.  A direction on an arc's end
// has x = kappa and contributes nothing, so the rounding of the end does not
// matter.
//
// A block owns 32 mu rows of a slice k, one per lane, and 8 items of (mu_s
// column c, up to kNq nu nodes), one per warp: the kinks are the warp's own
// (no divergence), the prefix sums the lane's own (no bank conflict at any
// index).  The prefix sums start at phi = pi, opposite the forward peak of
// the Mie phase function, so that arcs on either side of the peak are
// differences of small numbers.
//
// Bound by the L1 data pipe at 77%: a kink costs a texel six 8-byte reads of
// the sums.  16 instances at the reference's shape 4.53 -> 2.30 ms per launch
// (91 M warp instructions per instance instead of 262 M), 16 at half its
// sizes 0.563 -> 0.158, one high-resolution instance (NU 16: 9 kinks) 4.44 ->
// 4.01.  Two blocks of 8 warps per SM overlap one block's set-up of a theta
// row with the other's arcs; one block of 16 with two tables measured 2.53,
// 16-byte reads of two sums 2.81, 4 nodes per warp 2.94.
// ---------------------------------------------------------------------------
constexpr int kArcWarps = 8;
constexpr int kArcMaxSmem = 113 * 1024;   // two blocks per SM
constexpr int kArcThreads = 32 * kArcWarps;
constexpr int kArcHalf = kDensityPhiSamples / 2;    // phi samples of a half circle
constexpr int kArcEntries = 3 * kArcHalf + 1;       // ends phi = -pi .. 2 pi
constexpr int kArcEntryBytes = 32 * 8;              // (Rayleigh, Mie) of 32 lanes
constexpr int kArcSumBytes = kArcEntries * kArcEntryBytes;
constexpr int kArcTableBytes = 3 * kArcSumBytes;    // P, P cos(phi), P sin(phi)
constexpr int kArcPhaseBytes = kArcHalf * kArcEntryBytes;

// One kink: kappa, the slope change per channel times the Rayleigh and the
// Mie scattering coefficient, and the arc ends' index offsets -psi and +psi
// (16 fraction bits, the table's base included).
struct __align__(16) ArcKink {
  float4 r;    // Rayleigh, kappa
  float4 m;    // Mie, -
  int2 ends;
  int2 pad;
};

__host__ __device__ inline int ArcNodes(const Shape& s) {
  return DensityKind(s) == kDensityArcs4 ? 4 : 8;
}
__host__ __device__ inline int ArcGroups(const Shape& s) {
  const int nq = ArcNodes(s), items = s.smus * ((s.snu + nq - 1) / nq);
  return (items + kArcWarps - 1) / kArcWarps;
}
int DensityFastTiles(const Shape& s, int order) {
  if (order == 2 || DensityKind(s) == kDensityLookups) return s.sr * s.smus;
  return s.sr * ((s.smu + 31) / 32) * ArcGroups(s);
}
// The table and two phase buffers, each warp's nodes and kinks, the
// irradiance row.
__host__ __device__ inline int DensityArcSmem(const Shape& s) {
  return 256 + kArcTableBytes + 2 * kArcPhaseBytes +
         kArcWarps * (kDensityThetaSamples * s.snu * 16 + 32 * (int)sizeof(ArcKink)) + s.iw * 16;
}

int DensityFastSmem(const Shape& s, const Consts& c, int order) {
  const int base = DensityBaseSmem(s, order) + DensityPartSmem(s, order);
  if (order == 2) return base;
  if (DensityKind(s) != kDensityLookups) return DensityArcSmem(s);
  const int room = kDensityMaxSmem - base;
  const int merge = std::min(DensityMergeNeed(s, c), room > 0 ? room : 0);
  return base + merge / kNodeBytes * kNodeBytes;
}

__device__ __forceinline__ float2 Sub2(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}

template <int kNq>
__global__ void __launch_bounds__(kArcThreads, 2)
k_density_arcs(const Instance* __restrict__ insts, WorkList wl, int order) {
  extern __shared__ float4 smem[];
  int local;
  const Instance& in = insts[FindEntry(wl, blockIdx.x, &local)];
  if (DensityKind(in.s) != (kNq == 4 ? kDensityArcs4 : kDensityArcs8)) return;
  const Shape s = in.s;
  const Consts& c = in.c;
  const int NU = s.snu, W = s.sw(), lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  const int chunks = (NU + kNq - 1) / kNq, groups = ArcGroups(s), jtiles = (s.smu + 31) / 32;
  const int k = local / (groups * jtiles), rest = local - k * groups * jtiles;
  const int jt = rest / groups, item = (rest - jt * groups) * kArcWarps + warp;
  const bool active = item < s.smus * chunks;
  const int col = active ? item / chunks : 0;
  const int n0 = active ? (item - col * chunks) * kNq : 0;
  const int j = jt * 32 + lane;

  const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t tab0 = (smem0 + 255u) & ~255u;
  char* tab = reinterpret_cast<char*>(smem) + (tab0 - smem0);
  float2* phase = reinterpret_cast<float2*>(tab + kArcTableBytes);   // [2][16][32]
  float4* nodes = reinterpret_cast<float4*>(tab + kArcTableBytes + 2 * kArcPhaseBytes);
  const float4* V = nodes + warp * kDensityThetaSamples * NU;            // the warp's [16][NU]
  float4* irr = nodes + kArcWarps * kDensityThetaSamples * NU;
  ArcKink* kinks = reinterpret_cast<ArcKink*>(irr + s.iw) + warp * 32;   // the warp's [32]

  const DensityRow* drows = in.tab.drows + k * kDensityThetaSamples;
  const TexelRow row = in.tab.rows[k * s.smu + min(j, s.smu - 1)];
  const TexelCol cc = in.tab.cols[col];
  // The previous order at each warp's column of slice k, interpolated in mu at
  // the theta samples, per nu node (neighbouring threads load neighbouring
  // columns); the bottom row of the irradiance.
  const int total = s.smus * chunks, item0 = item - warp;
  for (int e = threadIdx.x; e < kArcWarps * kDensityThetaSamples * NU; e += kArcThreads) {
    const int w = e % kArcWarps, ln = e / kArcWarps, l = ln / NU, n = ln - l * NU;
    if (item0 + w >= total) continue;
    const float Y = drows[l].u_mu * float(s.smu) - 0.5f, fy = floorf(Y), wy = Y - fy;
    const int y0 = ClampIdx((int)fy, s.smu), y1 = ClampIdx((int)fy + 1, s.smu);
    const int o = k * s.smu * W + n * s.smus + (item0 + w) / chunks;
    [[maybe_unused]] const long long nS = s.s_texels();
    const float4 a = __ldg(ATMO_CHECKED_PTR(kCheckDensityStage, in.dR, o, y0 * W, nS));
    const float4 b = __ldg(ATMO_CHECKED_PTR(kCheckDensityStage, in.dR, o, y1 * W, nS));
    nodes[w * kDensityThetaSamples * NU + ln] =
        make_float4(fmaf(wy, b.x - a.x, a.x), fmaf(wy, b.y - a.y, a.y),
                    fmaf(wy, b.z - a.z, a.z), 0.0f);
  }
  for (int e = threadIdx.x; e < s.iw; e += kArcThreads)
    irr[e] = __ldg(DeltaIrradiance(in, order - 2) + e);

  // The lane's texels: cos(alpha), sin(alpha), and alpha as an index of the
  // tables' ends (16 fraction bits, plus 1/2 to round, from phi = -pi).
  float ca[kNq], sa[kNq];
  int ia[kNq];
  const float inv_sin = cc.sin_s > 0.0f ? 1.0f / cc.sin_s : 0.0f;
#pragma unroll
  for (int q = 0; q < kNq; ++q) {
    const TexelAngles ang = MakeAngles(s, row, cc, min(n0 + q, NU - 1));
    ca[q] = ang.sx * inv_sin;
    sa[q] = ang.sy * inv_sin;
    const float a = atan2f(ang.sy, ang.sx) * (float(kArcHalf) / kPiF);
    ia[q] = min(max(__float2int_rn((a + 0.5f) * 65536.0f), 0x8000),
                (kArcHalf << 16) + 0x8000) + (kArcHalf << 16);
  }
  F3 acc[kNq];
#pragma unroll
  for (int q = 0; q < kNq; ++q) acc[q] = f3(0.0f);
  // The scattering coefficients at the slice, with the phase constants.
  const F3 a_r = c.rayleigh * (ProfileDensity(c.prof_r, row.h) * c.ray_k);
  const F3 a_m = c.mie_sca * (ProfileDensity(c.prof_m, row.h) * c.mie_k);

  const float row_r = in.tab.rows[k * s.smu].r;
  const float dtdp = (kPiF / 16.0f) * (kPiF / 16.0f);
  // The outgoing phase functions of the lane's row at the 16 phi samples of a
  // half circle on theta row l, times the solid angle.
  auto build_phase = [&](int l) {
    const float ct = drows[l].cos_t, st = drows[l].sin_t;
    const float B = row.mu * ct, ox = row.omega_x * st, dw = dtdp * st;
    for (int m = warp; m < kArcHalf; m += kArcWarps) {
      const float nu2 = fmaf(ox, c_density_phi[m].x, B);
      const float q2 = fmaf(nu2, nu2, 1.0f) * dw;
      // 1 + g^2 - 2 g nu2 >= (1 - g)^2: zero or normal for |g| < 1.
      const float rs = RsqrtFtz(fmaf(c.m2g, nu2, c.g2p1));
      phase[((l & 1) * kArcHalf + m) * 32 + lane] = make_float2(q2, q2 * (rs * rs * rs));
    }
  };
  // The prefix sums of theta row l: of P, P cos(phi) and P sin(phi) from phi
  // up to pi (negative past it), at the ends b Delta, 2 pi - b Delta and
  // -b Delta.  With T(b) the half circle's sum of the samples b and after (P
  // is even), the even sums are T(b), -T(b) and T(0) plus the samples before
  // b; the odd one is T(b) at all three.  Tasks 0 and 1: the even sums' first
  // two; 2 and 3: their third; 4: the odd sum.
  auto build_table = [&](int l, int task) {
    const float2* p = phase + (l & 1) * kArcHalf * 32 + lane;
    const int kind = task == 4 ? 2 : task & 1;
    float2* t = reinterpret_cast<float2*>(tab + kind * kArcSumBytes) + lane;
    float2 T = make_float2(0.0f, 0.0f);
    auto add = [&](int m) {
      const float f = kind == 0 ? 1.0f : kind == 1 ? c_density_phi[m].x : c_density_phi[m].y;
      T = __ffma2_rn(Dup(f), p[m * 32], T);
    };
    if (task == 2 || task == 3) {
#pragma unroll
      for (int m = kArcHalf - 1; m >= 0; --m) add(m);
      t[kArcHalf * 32] = T;
#pragma unroll
      for (int b = 1; b <= kArcHalf; ++b) {
        add(b - 1);
        t[(kArcHalf - b) * 32] = T;
      }
      return;
    }
#pragma unroll
    for (int b = kArcHalf; b >= 0; --b) {
      if (b < kArcHalf) add(b);
      if (task == 4) {
        t[(kArcHalf + b) * 32] = T;
        t[(kArcHalf - b) * 32] = T;
        t[(3 * kArcHalf - b) * 32] = T;
      } else {
        if (b > 0) t[(kArcHalf + b) * 32] = T;
        t[(3 * kArcHalf - b) * 32] = make_float2(-T.x, -T.y);
      }
    }
  };

  const uint32_t lane8 = (uint32_t)lane * 8u;
  const float nodes_half = 0.5f * float(NU - 1), irr_half = 0.5f * float(s.iw - 1);
  const float inv_rb = 1.0f / c.Rb;
  const int sky = NU - 2;   // inner nu nodes
  // Theta row l's node coordinates v = v0 + h x (sky) and w = w0 + hw x
  // (irradiance), the candidate kinks (the inner nu nodes, then the inner
  // irradiance nodes that may be in range: those before i0 lie below it), and
  // the base segments, complete once every candidate has been looked at.
  float v0, h, w0, hw;
  int i0, candidates, sky_seg, ground_seg, count;
  auto next_row = [&](int l) {
    const DensityRow& dr = drows[l];
    v0 = fmaf(cc.mu_s * dr.cos_t, nodes_half, nodes_half);
    h = dr.sin_t * cc.sin_s * nodes_half;
    w0 = fmaf(fmaf(dr.dist_ground, dr.cos_t, row_r) * cc.mu_s * inv_rb, irr_half, irr_half);
    hw = dr.dist_ground * dr.sin_t * cc.sin_s * inv_rb * irr_half;
    i0 = max((int)floorf(w0 - hw), 1);
    candidates =
        sky + (dr.ground ? max(min((int)ceilf(w0 + hw), s.iw - 2) - i0 + 1, 0) : 0);
    sky_seg = 0;
    ground_seg = min(i0 - 1, s.iw - 2);
  };
  // The kinks among the 32 candidates from `first`.
  auto list_kinks = [&](int l, int first) {
    const int cand = first + lane;
    const bool is_sky = cand < sky, valid = cand < candidates;
    const int node = valid ? (is_sky ? cand + 1 : i0 + cand - sky) : 1;
    const float scale = is_sky ? h : hw;
    const float kappa = (float(node) - (is_sky ? v0 : w0)) / scale;
    // Nodes below the range set the base segment; a zero scale gives none in
    // range.
    const bool below = valid && !(kappa > -1.0f), inside = valid && kappa > -1.0f && kappa < 1.0f;
    sky_seg += __popc(__ballot_sync(0xffffffffu, below && is_sky));
    ground_seg += __popc(__ballot_sync(0xffffffffu, below && !is_sky));
    const unsigned in_range = __ballot_sync(0xffffffffu, inside);
    __syncwarp();
    if (inside) {
      const float4* v = is_sky ? V + l * NU + node : irr + node;
      const float4 va = v[-1], vb = v[0], vc = v[1];
      F3 d = F3{(vc.x - vb.x) - (vb.x - va.x), (vc.y - vb.y) - (vb.y - va.y),
                (vc.z - vb.z) - (vb.z - va.z)} * scale;
      if (!is_sky) d = d * f3(drows[l].t_ground);
      const int p = __float2int_rn(acosf(kappa) * (float(kArcHalf) * 65536.0f / kPiF));
      const int b = (int)(tab0 >> 8) << 16;
      ArcKink& kn = kinks[__popc(in_range & ((1u << lane) - 1u))];
      kn.r = to4(d * a_r, kappa);
      kn.m = to4(d * a_m, 0.0f);
      kn.ends = make_int2(b - p, b + p);
    }
    __syncwarp();
    count = __popc(in_range);
  };

  build_phase(0);
  build_phase(1);
  __syncthreads();
  F3 base0 = f3(0.0f), base1 = f3(0.0f);   // the base lines' sums: constant, cos(alpha) part
#pragma unroll 1
  for (int l = 0; l < kDensityThetaSamples; ++l) {
    // Five warps have a part of the table to build.
    for (int task = (warp + 3 * l) % kArcWarps; task < 5; task += kArcWarps) build_table(l, task);
    next_row(l);
    if (active) list_kinks(l, 0);
    __syncthreads();
    if (l + 2 < kDensityThetaSamples) build_phase(l + 2);
    if (active) {
      for (int first = 0;;) {
        for (int e = 0; e < count; ++e) {
          const float4 kr = kinks[e].r, km = kinks[e].m;
          const int2 ends = kinks[e].ends;
          // Four texels' sums are loaded at a time, ahead of their use: 2.30 ms
          // per 16-instance launch against 2.43 in the compiler's own order.
          constexpr int kG = 4;
#pragma unroll
          for (int q0 = 0; q0 < kNq; q0 += kG) {
            float2 lo[kG][3], hi[kG][3];
#pragma unroll
            for (int u = 0; u < kG; ++u) {
              const uint32_t a0 = __byte_perm((uint32_t)(ia[q0 + u] + ends.x), lane8, 0x5324);
              const uint32_t a1 = __byte_perm((uint32_t)(ia[q0 + u] + ends.y), lane8, 0x5324);
              lo[u][0] = LoadShared2<0>(a0);
              hi[u][0] = LoadShared2<0>(a1);
              lo[u][1] = LoadShared2<kArcSumBytes>(a0);
              hi[u][1] = LoadShared2<kArcSumBytes>(a1);
              lo[u][2] = LoadShared2<2 * kArcSumBytes>(a0);
              hi[u][2] = LoadShared2<2 * kArcSumBytes>(a1);
            }
#pragma unroll
            for (int u = 0; u < kG; ++u) {
              const int q = q0 + u;
              const float2 d0 = Sub2(lo[u][0], hi[u][0]);
              const float2 dc = Sub2(lo[u][1], hi[u][1]);
              const float2 ds = Sub2(lo[u][2], hi[u][2]);
              const float gr = fmaf(-kr.w, d0.x, fmaf(sa[q], ds.x, ca[q] * dc.x));
              const float gm = fmaf(-kr.w, d0.y, fmaf(sa[q], ds.y, ca[q] * dc.y));
              acc[q] = fma3(F3{km.x, km.y, km.z}, gm, fma3(F3{kr.x, kr.y, kr.z}, gr, acc[q]));
            }
          }
        }
        first += 32;
        if (first >= candidates) break;
        list_kinks(l, first);
      }
      // The base line R0 + R1 x over the whole circle.
      F3 r0, r1;
      {
        const float4 a = V[l * NU + sky_seg], b = V[l * NU + sky_seg + 1];
        const F3 d{b.x - a.x, b.y - a.y, b.z - a.z};
        r0 = fma3(d, v0 - float(sky_seg), F3{a.x, a.y, a.z});
        r1 = d * h;
      }
      if (drows[l].ground) {
        const F3 tg = f3(drows[l].t_ground);
        const float4 a = irr[ground_seg], b = irr[ground_seg + 1];
        const F3 d{b.x - a.x, b.y - a.y, b.z - a.z};
        r0 = fma3(tg, fma3(d, w0 - float(ground_seg), F3{a.x, a.y, a.z}), r0);
        r1 = fma3(tg, d * hw, r1);
      }
      const uint32_t full = tab0 + kArcHalf * kArcEntryBytes + lane8;   // phi = 0
      const float2 t0 = LoadShared2<0>(full), tc = LoadShared2<kArcSumBytes>(full);
      base0 = fma3(r0, fma3(a_m, t0.y, a_r * t0.x), base0);
      base1 = fma3(r1, fma3(a_m, tc.y, a_r * tc.x), base1);
    }
    __syncthreads();
  }
  if (!active || j >= s.smu) return;
  // The full circle is twice the half circle's sums.
#pragma unroll
  for (int q = 0; q < kNq; ++q) {
    if (n0 + q < NU) {
      const F3 J = fma3(fma3(base1, ca[q], base0), 2.0f, acc[q]);
      in.dJ[(k * s.smu + j) * W + (n0 + q) * s.smus + col] = to4(J, 1.0f);
    }
  }
}

// Lets k_density_fast<false> take kDensityMaxSmem (once per device; every
// later call is a lock-free check).  Called before a CUDA graph capture and
// by the launcher.
cudaError_t PrepareDensityFast() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(k_density_fast<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kDensityMaxSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_density_arcs<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kArcMaxSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_density_arcs<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kArcMaxSmem);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

cudaError_t LaunchDensityFast(const Instance* insts, WorkList wl, int tiles, int order,
                              int smem_bytes, cudaStream_t st) {
  // smem_bytes: the largest DensityFastSmem of the work list's instances.
  const size_t bytes = (size_t)smem_bytes;
  if (order == 2) {
    k_density_fast<true><<<tiles, kDensityFastThreads, bytes, st>>>(insts, wl, order, smem_bytes,
                                                                      kRoundMagic);
  } else {
    if (smem_bytes > 48 * 1024) {
      const cudaError_t e = PrepareDensityFast();
      if (e != cudaSuccess) return e;
    }
    // Each kernel returns at the others' instances.
    if (wl.kinds & kDensityArcs8)
      k_density_arcs<8><<<tiles, kArcThreads, bytes, st>>>(insts, wl, order);
    if (wl.kinds & kDensityArcs4)
      k_density_arcs<4><<<tiles, kArcThreads, bytes, st>>>(insts, wl, order);
    if (wl.kinds & kDensityLookups) {
      const int fast_bytes = std::min(smem_bytes, kDensityMaxSmem);
      k_density_fast<false><<<tiles, kDensityFastThreads, (size_t)fast_bytes, st>>>(
          insts, wl, order, fast_bytes, kRoundMagic);
    }
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Multiple scattering, restructured (functions.glsl:1268-1308).
//
// Every quantity of a quadrature sample but mu_s depends only on the texel's
// row (r-slice k, mu-row j): the sample's r and mu, hence the (y, z) position
// of its 4D lookup, and the transmittance from the texel to the sample.  A
// block owns whole rows; it computes their samples once (RaySample), then,
// per sample, interpolates the density LUT in (mu, r) at the sample into a
// line of W = NU x MU_S columns in shared memory.  A texel's lookup reduces to
// its own mu_s mapping and a bilinear (mu_s, nu) interpolation of 4 columns
// of that line.  Lines are built G samples at a time, double-buffered, so a
// stage needs one barrier.
// ---------------------------------------------------------------------------
constexpr int kMultipleFastThreads = 256;
constexpr int kMultipleFastMaxCols = 4;   // texel columns per thread (W <= 1024)
constexpr int kRaySamples = kMultipleScatteringSamples + 1;

struct __align__(16) RaySample {
  // Element offsets of the four LUT rows around the sample, the (k, j) = (r,
  // mu) row with even k and j first, then odd j, odd k, both odd: of two
  // samples' rows, those they share have the same place.
  int r00, r01, r10, r11;
  float w00, w01, w10, w11;  // their bilinear weights in (mu, r)
  float tx, ty, tz;          // transmittance texel -> sample x dx x trapezoid weight
  float rb_inv_r, rb_d;      // Rb / r and Rb d / r at the sample
  int fresh;                 // a bit for each row that the next sample changes
  float d;                   // distance from the texel's point along its ray
  float inv_r;               // 1 / r at the sample
};

struct MultipleFastDims {
  int rows;    // LUT rows per block
  int group;   // samples per line stage
};
// Rows per block and samples per line stage: the tuned values of the shape,
// else as many rows (up to 4) as fill 256 threads and two line buffers of
// group x rows x W float4 within 32 KB.
__host__ __device__ inline MultipleFastDims MultipleDims(const Shape& s) {
  const int W = s.sw();
  int rows = kMultipleFastThreads / W;
  rows = rows < 1 ? 1 : (rows > 4 ? 4 : rows);
  if (s.tune[0] > 0) rows = s.tune[0];
  int group = 32768 / (2 * 16 * rows * W);
  group = group < 1 ? 1 : (group > 4 ? 4 : group);
  if (s.tune[1] > 0) group = s.tune[1];
  return MultipleFastDims{rows, group};
}
// The LUT row that logical row i of the multiple-scattering blocks takes.
__device__ __forceinline__ int RowAt(const Tables& tab, int i) {
  return tab.row_order ? __ldg(tab.row_order + i) : i;
}

// Sample i of the ray of LUT row `rowi` (the per-sample part of
// MultipleScatteringTexel that does not depend on mu_s or nu).
__device__ RaySample MakeRaySample(const Instance& in, int rowi, int i) {
  const Consts& c = in.c;
  const Shape& s = in.s;
  const TexelRow row = in.tab.rows[rowi];
  const bool ground = row.ground != 0;
  const float dx = row.d / float(kMultipleScatteringSamples);
  const float d = float(i) * dx;
  const float e = float(kMultipleScatteringSamples - i) * dx;
  const RadialPoint p = PointFromRho2(c, RayRho2(row, d, e));
  const float u_mu = UMuFromDistance(c, s, p, e, ground);
  const float u_r = TexCoord(s, kMapSR, p.rho / c.H);
  const TStart start = MakeTStart(c, s, in.T, in.Tau, row.rho, row.r,
                                  ground ? -row.rmu : row.rmu, row.delta);
  const F3 t = SegmentTransmittance(c, s, in.T, in.Tau, row.rmu, row.delta, p, d, ground, start);
  const float w = (i == 0 || i == kMultipleScatteringSamples) ? 0.5f : 1.0f;
  const float Y = u_mu * float(s.smu) - 0.5f, Z = u_r * float(s.sr) - 0.5f;
  const float fy = floorf(Y), fz = floorf(Z);
  const float b = Y - fy, cz = Z - fz;
  const int j0 = ClampIdx((int)fy, s.smu), j1 = ClampIdx((int)fy + 1, s.smu);
  const int k0 = ClampIdx((int)fz, s.sr), k1 = ClampIdx((int)fz + 1, s.sr);
  const int W = s.sw();
  RaySample rs;
  const bool oj = j0 & 1, ok = k0 & 1;
  const int je = oj ? j1 : j0, jo = oj ? j0 : j1, ke = ok ? k1 : k0, ko = ok ? k0 : k1;
  const float bo = oj ? 1.0f - b : b, be = oj ? b : 1.0f - b;
  const float co = ok ? 1.0f - cz : cz, ce = ok ? cz : 1.0f - cz;
  rs.r00 = (ke * s.smu + je) * W;
  rs.r01 = (ke * s.smu + jo) * W;
  rs.r10 = (ko * s.smu + je) * W;
  rs.r11 = (ko * s.smu + jo) * W;
  rs.w00 = be * ce;
  rs.w01 = bo * ce;
  rs.w10 = be * co;
  rs.w11 = bo * co;
  const float dw = dx * w;
  rs.tx = t.x * dw;
  rs.ty = t.y * dw;
  rs.tz = t.z * dw;
  rs.d = d;
  rs.inv_r = 1.0f / p.r;
  rs.rb_inv_r = c.Rb / p.r;
  rs.rb_d = rs.rb_inv_r * d;
  rs.fresh = 0;
  return rs;
}

// UMuSFromMuS with the mapping's constant divisions replaced by products
// (inv_range = 1 / (d_max - d_min), inv_A = 1 / A) and the others approximate
// (<= 2 ulp): for samples along a ray, whose mu_s is not a texel's own.
__device__ __forceinline__ float UMuSFromMuSAlongRay(const Consts& c, const Shape& s, float mu_s,
                                                     float inv_range, float inv_A) {
  const float H2 = c.H * c.H;
  const float rmus = c.Rb * mu_s;
  // H^2 + (Rb mu_s)^2 >= H^2 and rmus + sq >= H > 0: normal.  The last
  // quotient's numerator is zero or in [ulp(1), 1], its denominator in
  // [1, 2].
  const float sq = SqrtFtz(fmaf(rmus, rmus, H2));
  const float d = rmus > 0.0f ? DivFtz(H2, rmus + sq) : sq - rmus;
  const float a = (d - (c.Rt - c.Rb)) * inv_range;
  return TexCoord(s, kMapSMUS, DivFtz(fmaxf(fmaf(-a, inv_A, 1.0f), 0.0f), 1.0f + a));
}

// The element at offset + x of a LUT row of a line build.
#define ATMO_LINE_PTR(base, offset, x, n) ATMO_CHECKED_PTR(kCheckLineLoad, base, offset, x, n)

// A read-only global load predicated on p: v keeps its value when p is 0.
// The predicate keeps the line build free of branches, so a sample's loads
// still issue as early as the unconditional ones.
__device__ __forceinline__ void LoadIf(float4& v, const float4* ptr, int p) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
      "@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "l"(ptr), "r"(p));
}

template <int kCols>
__device__ __forceinline__ void MultipleFastBlock(const Instance& in, int local, float4* smem) {
  const Shape s = in.s;
  const Consts& c = in.c;
  const MultipleFastDims dims = MultipleDims(s);
  const int W = s.sw(), R = dims.rows, G = dims.group;
  const int rows_total = s.sr * s.smu;
  [[maybe_unused]] const long long nS = s.s_texels();   // checked build
  const int row0 = local * R;
  RaySample* samp = reinterpret_cast<RaySample*>(smem);                 // [R][kRaySamples]
  float4* line = smem + R * kRaySamples * (int)(sizeof(RaySample) / 16);   // [2][G][R][W]

  for (int e = threadIdx.x; e < R * kRaySamples; e += kMultipleFastThreads) {
    const int rr = e / kRaySamples, i = e - rr * kRaySamples;
    if (row0 + rr < rows_total) samp[e] = MakeRaySample(in, RowAt(in.tab, row0 + rr), i);
  }

  // This thread's row within the tile and its texel columns x_t + 256 m.
  const int rr = kCols == 1 ? (int)threadIdx.x / W : 0;
  const int x_t = kCols == 1 ? (int)threadIdx.x - rr * W : (int)threadIdx.x;
  const bool active = rr < R && row0 + rr < rows_total;
  const int rowi = active ? RowAt(in.tab, row0 + rr) : 0;
  const float smus_f = float(s.smus);
  const int nmax = W - 1;
  const float inv_range = 1.0f / (c.H - (c.Rt - c.Rb));
  const float inv_A = 1.0f / c.mus_A;
  float rmu_s[kCols], nu[kCols], lnu[kCols];
  int xb[kCols];
  F3 acc[kCols];
  if (active) {
    const TexelRow row = in.tab.rows[rowi];
#pragma unroll
    for (int m = 0; m < kCols; ++m) {
      const int x = min(x_t + m * kMultipleFastThreads, nmax);
      const int n = x / s.smus, col = x - n * s.smus;
      const TexelAngles ang = MakeAngles(s, row, in.tab.cols[col], n);
      rmu_s[m] = row.r * ang.mu_s;
      nu[m] = ang.nu;
      // A texel whose nu is not clamped sits on its own nu node n: the
      // reference's FP64 coordinate (nu + 1) / 2 (NU - 1) is n to ~1e-16, so
      // the neighbouring node's weight is taken as 0 and its taps skipped.
      const float tex_coord_x = (ang.nu + 1.0f) * 0.5f * float(s.snu - 1);
      const float tex_x = ang.on_node ? float(n) : floorf(tex_coord_x);
      lnu[m] = ang.on_node ? 0.0f : tex_coord_x - tex_x;
      xb[m] = (int)tex_x * s.smus;   // the node's block (see MakeLookup)
      acc[m] = f3(0.0f);
    }
  }
  __syncthreads();

  const int line_stride = G * R * W;
  const int stages = (kRaySamples + G - 1) / G;
  for (int stage = 0; stage < stages; ++stage) {
    float4* buf = line + (stage & 1) * line_stride;
    const int first = stage * G;
    const int count = min(G, kRaySamples - first);
    if (active && kCols == 1) {
      // Consecutive samples of a ray lie in the same (mu, r) cell of the
      // delta-density LUT for 38% of the samples at the reference's shape:
      // their four rows, already in registers, are not loaded again (r00 and
      // r11 fix all four).  Predicated loads rather than a branch: a branch
      // around the loads measured slower than four loads per sample.  The
      // values, hence the LUTs, are the same as with four loads per sample.
      // The thread's column of the LUT, of its line and of its row's samples,
      // addressed once (row offsets are then 32-bit adds to a 64-bit base:
      // 7% fewer instructions than forming each address, 1.7% less time).
      int o00 = -1, o11 = -1;
      float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a, p = a, q = a;
      const float4* col = in.dJ + x_t;
      float4* out_col = buf + rr * W + x_t;
      const RaySample* srow = samp + rr * kRaySamples + first;
      for (int g = 0; g < count; ++g) {
        const RaySample& sm = srow[g];
        const int fresh = (sm.r00 != o00) | (sm.r11 != o11);
        LoadIf(a, ATMO_LINE_PTR(col, sm.r00, 0, nS - x_t), fresh);
        LoadIf(b, ATMO_LINE_PTR(col, sm.r01, 0, nS - x_t), fresh);
        LoadIf(p, ATMO_LINE_PTR(col, sm.r10, 0, nS - x_t), fresh);
        LoadIf(q, ATMO_LINE_PTR(col, sm.r11, 0, nS - x_t), fresh);
        o00 = sm.r00;
        o11 = sm.r11;
        out_col[g * R * W] = make_float4(
            fmaf(q.x, sm.w11, fmaf(p.x, sm.w10, fmaf(b.x, sm.w01, a.x * sm.w00))),
            fmaf(q.y, sm.w11, fmaf(p.y, sm.w10, fmaf(b.y, sm.w01, a.y * sm.w00))),
            fmaf(q.z, sm.w11, fmaf(p.z, sm.w10, fmaf(b.z, sm.w01, a.z * sm.w00))), 0.0f);
      }
    } else if (active) {
      for (int g = 0; g < count; ++g) {
        const RaySample& sm = samp[rr * kRaySamples + first + g];
        float4* out = buf + (g * R + rr) * W;
#pragma unroll
        for (int m = 0; m < kCols; ++m) {
          const int x = x_t + m * kMultipleFastThreads;
          if (kCols > 1 && x >= W) break;
          const float4 a = __ldg(ATMO_LINE_PTR(in.dJ, sm.r00, x, nS));
          const float4 b = __ldg(ATMO_LINE_PTR(in.dJ, sm.r01, x, nS));
          const float4 p = __ldg(ATMO_LINE_PTR(in.dJ, sm.r10, x, nS));
          const float4 q = __ldg(ATMO_LINE_PTR(in.dJ, sm.r11, x, nS));
          out[x] = make_float4(
              fmaf(q.x, sm.w11, fmaf(p.x, sm.w10, fmaf(b.x, sm.w01, a.x * sm.w00))),
              fmaf(q.y, sm.w11, fmaf(p.y, sm.w10, fmaf(b.y, sm.w01, a.y * sm.w00))),
              fmaf(q.z, sm.w11, fmaf(p.z, sm.w10, fmaf(b.z, sm.w01, a.z * sm.w00))), 0.0f);
        }
      }
    }
    __syncthreads();
    if (active) {
      const RaySample* srow = samp + rr * kRaySamples + first;
      const float4* lrow = buf + rr * W;
      for (int g = 0; g < count; ++g) {
        const RaySample& sm = srow[g];
        const float4* L = lrow + g * R * W;
#pragma unroll
        for (int m = 0; m < kCols; ++m) {
          if (kCols > 1 && x_t + m * kMultipleFastThreads >= W) break;
          const float mu_s_i = clampf(fmaf(sm.d, nu[m], rmu_s[m]) * sm.inv_r, -1.0f, 1.0f);
          const float x0 =
              fmaf(UMuSFromMuSAlongRay(c, s, mu_s_i, inv_range, inv_A), smus_f, -0.5f);
          const float fx = floorf(x0);
          const float a = x0 - fx;
          const int i0 = xb[m] + (int)fx;
          const int c0 = min(max(i0, 0), nmax), c1 = min(max(i0 + 1, 0), nmax);
          const int c2 = min(max(i0 + s.smus, 0), nmax), c3 = min(max(i0 + s.smus + 1, 0), nmax);
          const float l1 = lnu[m], l0 = 1.0f - l1;
          const float v0 = (1.0f - a) * l0, v1 = a * l0;
          const float4 t0 = L[ATMO_CHECKED_INDEX(kCheckLineTap, c0, W)];
          const float4 t1 = L[ATMO_CHECKED_INDEX(kCheckLineTap, c1, W)];
          F3 S{fmaf(t1.x, v1, t0.x * v0), fmaf(t1.y, v1, t0.y * v0),
               fmaf(t1.z, v1, t0.z * v0)};
          if (l1 != 0.0f) {
            const float v2 = (1.0f - a) * l1, v3 = a * l1;
            const float4 t2 = L[ATMO_CHECKED_INDEX(kCheckLineTap, c2, W)];
            const float4 t3 = L[ATMO_CHECKED_INDEX(kCheckLineTap, c3, W)];
            S = F3{fmaf(t3.x, v3, fmaf(t2.x, v2, S.x)), fmaf(t3.y, v3, fmaf(t2.y, v2, S.y)),
                   fmaf(t3.z, v3, fmaf(t2.z, v2, S.z))};
          }
          acc[m] = fma3(S, F3{sm.tx, sm.ty, sm.tz}, acc[m]);
        }
      }
    }
  }

  if (!active) return;
#pragma unroll
  for (int m = 0; m < kCols; ++m) {
    const int x = x_t + m * kMultipleFastThreads;
    if (kCols > 1 && x >= W) break;
    const int texel = (int)ATMO_CHECKED_INDEX(kCheckOutput, rowi * W + x, nS);
    in.dR[texel] = to4(acc[m], 1.0f);   // delta multiple aliases delta Rayleigh
    const F3 add = MatVec(c.lum, acc[m]) * (1.0f / RayleighPhase(c, nu[m]));
    const float4 o = in.S[texel];
    in.S[texel] = make_float4(o.x + add.x, o.y + add.y, o.z + add.z, o.w);
  }
}

// ---------------------------------------------------------------------------
// Multiple scattering by nu nodes (MultipleKind 1 and 2): no shared line.
//
// The columns of one nu node's block are the MU_S <= 64 mu_s columns of that
// node, so a warp can hold a sample's interpolated line of one node (two
// columns per lane above MU_S = 32) or of several nodes (32 / MU_S) in
// registers: a lane interpolates its own columns from the four delta-density
// rows, and a texel's two mu_s taps are shuffles.  A warp then marches the 51
// samples of a row on its own, with no line in shared memory and no barrier
// per line stage.
//
// A texel whose nu is not clamped sits on its own node, so its taps are in
// its own warp.  The texels of a row and column whose nu is clamped share the
// clamped value (one below, one above the physical range), which lies between
// two nodes n0, n0 + 1: those two nodes' warps each march that nu through
// their own node's line, weighted with the node's lerp weight, and the two
// parts are added through shared memory at the end.  A column thus gives its
// warp up to three of the tasks {its own texel, the low and the high clamped
// nu}, 1.2 on average at the reference's shape.  Any lane can march any task,
// so the warp packs them: 1.5 marches of 32 tasks per node, where a lane that
// marches its own columns' tasks needs 1.7.
//
// Bound by the L1 data pipe (78%) and instruction issue (74%) together, 27
// wavefronts and 99 instructions per warp and sample, against 45 and 135 of
// the lines in shared memory, whose stores, taps and clamps it does without.
// Of a sample's four rows those it shares with the last one stay in
// registers.  Per 16-instance launch at the reference's shape 4.13 (lines in
// shared memory) -> 3.25 (nodes) -> 3.08 (packed tasks) -> 2.95 (four items
// per warp, handed out) -> 2.76 ms (shared rows kept); one high-resolution
// instance 4.40 -> 3.43 -> 3.08 -> 3.03 -> 2.72 ms.
// ---------------------------------------------------------------------------
constexpr int kNodeWarps = kMultipleFastThreads / 32;
constexpr int kNodeSamples = kRaySamples + 1;   // the last one twice
__host__ __device__ inline bool MultipleByNodes(const Shape& s) { return MultipleKind(s) < 4; }
// Nu nodes held by one warp, and warp items (of that many nodes) per row.
__host__ __device__ inline int NodesPerWarp(const Shape& s) {
  return s.smus <= 32 ? 32 / s.smus : 1;
}
__host__ __device__ inline int NodeItemsPerRow(const Shape& s) {
  const int per = NodesPerWarp(s);
  return (s.snu + per - 1) / per;
}
// Rows per block: as many (up to 4) as give its 8 warps one item each, or four
// where that leaves a full wave of blocks (4 per SM).  Four items
// per warp shorten the blocks' idle time (their sample tables are built by 51
// threads per row, and the items differ): 2.82 ms per 16-instance launch at
// the reference's shape against 2.91 with two; smaller LUTs want the shorter
// blocks.
__host__ __device__ inline int NodeRows(const Shape& s) {
  const int items = NodeItemsPerRow(s);
  const bool many = (long long)s.sr * s.smu * items >= 4LL * kNodeWarps * 4 * kSmCount;
  const int rows = (many ? 4 : 1) * kNodeWarps / items;
  return rows < 1 ? 1 : (rows > 4 ? 4 : rows);
}

// LoadIf of two neighbouring texels (32-byte aligned).
__device__ __forceinline__ void LoadTwoIf(float4& a, float4& b, const float4* ptr, int p) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %9, 0;\n\t"
      "@q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
      : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w), "+f"(b.x), "+f"(b.y), "+f"(b.z), "+f"(b.w)
      : "l"(ptr), "r"(p));
}

// A lane's columns of one LUT row: one, two with a 256-bit load (kPair: the
// columns are 32-byte aligned), or two loads (second: the offset of the
// second column, 0 where the lane has one).
template <int kCols>
struct NodeRow {
  float4 v[kCols];
};
template <int kCols, bool kPair>
__device__ __forceinline__ void LoadRowIf(NodeRow<kCols>& row, const float4* col, int offset,
                                          int second, [[maybe_unused]] long long n, int p) {
  if constexpr (kCols == 1) {
    LoadIf(row.v[0], ATMO_LINE_PTR(col, offset, 0, n), p);
  } else if constexpr (kPair) {
    LoadTwoIf(row.v[0], row.v[1], ATMO_LINE_PTR(col, offset, 0, n - 1), p);
  } else {
    LoadIf(row.v[0], ATMO_LINE_PTR(col, offset, 0, n), p);
    LoadIf(row.v[1], ATMO_LINE_PTR(col, offset, second, n), p);
  }
}

__device__ __forceinline__ F3 Shuffle3(F3 v, int lane) {
  return F3{__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane),
            __shfl_sync(0xffffffffu, v.z, lane)};
}

// acc + the line at x of the mu_s range of a node.  magic: kRoundMagic plus
// the node's first lane; the FMA rounded down leaves the lower tap's lane in
// the sum's low bits (a shuffle's lane counts modulo 32: at x = 1 the upper
// tap, of weight 0, may be any lane).
template <int kCols>
__device__ __forceinline__ F3 TapLine(const F3 (&line)[kCols], float x, float n1, float magic,
                                      F3 acc) {
  const float t = __fmaf_rd(x, n1, magic);
  const float w1 = fmaf(x, n1, magic - t), w0 = 1.0f - w1;
  const int i0 = __float_as_int(t);
  if constexpr (kCols == 1) {
    const F3 t0 = Shuffle3(line[0], i0), t1 = Shuffle3(line[0], i0 + 1);
    return fma3(t1, w1, fma3(t0, w0, acc));
  } else {
    // Columns 2 l, 2 l + 1 in lane l: the taps i0, i0 + 1 are one even and
    // one odd column.
    const bool odd = i0 & 1;
    const F3 te = Shuffle3(line[0], (i0 + 1) >> 1), to = Shuffle3(line[1], i0 >> 1);
    return fma3(to, odd ? w0 : w1, fma3(te, odd ? w1 : w0, acc));
  }
}

// Marches the row's samples: acc[t] += the line's value at the mu_s and nu of
// the lane's task t, times the sample's transmittance and weight.
template <int kCols, int kTasks, bool kPair, bool kSub>
__device__ __forceinline__ void MarchNodes(const RaySample* samp, const float4* col, int second,
                                           long long n, const SunMap& map,
                                           const float (&magic)[kSub ? kTasks : 1],
                                           const float (&rmu_s)[kTasks],
                                           const float (&nu)[kTasks], F3 (&acc)[kTasks]) {
  NodeRow<kCols> a, b, p, q;
#pragma unroll
  for (int m = 0; m < kCols; ++m)
    a.v[m] = b.v[m] = p.v[m] = q.v[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int4 r = *reinterpret_cast<const int4*>(&samp[0].r00);
  LoadRowIf<kCols, kPair>(a, col, r.x, second, n, 1);
  LoadRowIf<kCols, kPair>(b, col, r.y, second, n, 1);
  LoadRowIf<kCols, kPair>(p, col, r.z, second, n, 1);
  LoadRowIf<kCols, kPair>(q, col, r.w, second, n, 1);
#pragma unroll 1
  for (int i = 0; i < kRaySamples; ++i) {
    const float4 w = *reinterpret_cast<const float4*>(&samp[i].w00);
    const float4 t = *reinterpret_cast<const float4*>(&samp[i].tx);
    const float2 rb_fresh = *reinterpret_cast<const float2*>(&samp[i].rb_d);
    const int fresh = __float_as_int(rb_fresh.y);
    F3 line[kCols];
#pragma unroll
    for (int m = 0; m < kCols; ++m) {
      line[m] = fma3(f3(q.v[m]), w.w,
                     fma3(f3(p.v[m]), w.z, fma3(f3(b.v[m]), w.y, f3(a.v[m]) * w.x))) *
                F3{t.x, t.y, t.z};
    }
    // The next sample's rows are loaded while this one's taps are made, but
    // for those it shares with this one (sample 51 is sample 50 again).  One
    // column per lane skips them all with a branch where there is nothing to
    // load (2.76 ms per 16-instance launch against 2.82; two columns per lane
    // 2.80 against 2.79).
    if (kCols == 2 || fresh) {
      const int4 r1 = *reinterpret_cast<const int4*>(&samp[i + 1].r00);
      LoadRowIf<kCols, kPair>(a, col, r1.x, second, n, fresh & 1);
      LoadRowIf<kCols, kPair>(b, col, r1.y, second, n, fresh & 2);
      LoadRowIf<kCols, kPair>(p, col, r1.z, second, n, fresh & 4);
      LoadRowIf<kCols, kPair>(q, col, r1.w, second, n, fresh & 8);
    }
    // Rb mu_s at the sample: (r mu_s + d nu) Rb / r_i.
#pragma unroll
    for (int k = 0; k < kTasks; ++k) {
      const float x = SunCoordinate(map, fmaf(nu[k], rb_fresh.x, rmu_s[k] * t.w));
      acc[k] = TapLine<kCols>(line, x, map.n1, magic[kSub ? k : 0], acc[k]);
    }
  }
}

// The nu of a texel and whether it sits on its own node (MakeAngles).  Not
// inlined: the lanes that march a clamped nu and the texels that take the sum
// must agree on which texels are clamped, to the bit.
struct NodeNu {
  float nu;
  int side;   // -1 on the texel's own node, 0 clamped from below, 1 from above
};
__device__ __noinline__ NodeNu TexelNu(const Instance& in, int rowi, int col, int n) {
  const TexelAngles a = MakeAngles(in.s, in.tab.rows[rowi], in.tab.cols[col], n);
  return NodeNu{a.nu, a.on_node ? -1 : a.raised ? 0 : 1};
}

// Adds a texel's result to the LUTs (functions.glsl:1369-1383).
__device__ __forceinline__ void StoreMultiple(const Instance& in, int texel, F3 sum, float nu) {
  [[maybe_unused]] const long long nS = in.s.s_texels();
  texel = (int)ATMO_CHECKED_INDEX(kCheckOutput, texel, nS);
  in.dR[texel] = to4(sum, 1.0f);   // delta multiple aliases delta Rayleigh
  const F3 add = MatVec(in.c.lum, sum) * (1.0f / RayleighPhase(in.c, nu));
  const float4 o = in.S[texel];
  in.S[texel] = make_float4(o.x + add.x, o.y + add.y, o.z + add.z, o.w);
}

// A task of a warp: the nu to march, and where its result goes: the lane and
// column (lane x kCols + m) x 256 + 1 for the texel itself, 2 + 2 side + half
// for a part of a clamped nu.
struct NodeTask {
  float nu;
  int code;
};

template <int kCols, bool kPair, bool kSub>
__device__ __forceinline__ void MultipleNodesBlock(const Instance& in, int local, float4* smem) {
  const Shape s = in.s;
  const Consts& c = in.c;
  const int W = s.sw(), R = NodeRows(s), per = NodesPerWarp(s), items = NodeItemsPerRow(s);
  const int rows_total = s.sr * s.smu, row0 = local * R;
  [[maybe_unused]] const long long nS = s.s_texels();   // checked build
  RaySample* samp = reinterpret_cast<RaySample*>(smem);                        // [R][52]
  float4* edge = smem + R * kNodeSamples * (int)(sizeof(RaySample) / 16);       // [R][2][2][MU_S]
  const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  NodeTask* tasks = reinterpret_cast<NodeTask*>(edge + R * 4 * s.smus) +      // [8][3][32 kCols]
                    warp * 96 * kCols;
  __shared__ int next;   // the first item no warp has taken
  if (threadIdx.x == 0) next = kNodeWarps;

  for (int e = threadIdx.x; e < R * kNodeSamples; e += kMultipleFastThreads) {
    const int rr = e / kNodeSamples, i = min(e - rr * kNodeSamples, kRaySamples - 1);
    if (row0 + rr < rows_total) samp[e] = MakeRaySample(in, RowAt(in.tab, row0 + rr), i);
  }
  for (int e = threadIdx.x; e < R * 4 * s.smus; e += kMultipleFastThreads)
    edge[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();
  for (int e = threadIdx.x; e < R * kNodeSamples - 1; e += kMultipleFastThreads) {
    const int4 u = *reinterpret_cast<const int4*>(&samp[e].r00);
    const int4 v = *reinterpret_cast<const int4*>(&samp[e + 1].r00);
    samp[e].fresh = (u.x != v.x) | (u.y != v.y) << 1 | (u.z != v.z) << 2 | (u.w != v.w) << 3;
  }
  __syncthreads();

  const SunMap map = MakeSunMap(c, s);
  const float nodes1 = float(s.snu - 1);
  // The items go to the warps as these finish, the innermost nodes (the most
  // work) first.
  for (int item = warp; item < R * items;) {
    const int rr = item % R, o = item / R;
    const int slot = (items - 1) / 2 + (o & 1 ? (o + 1) / 2 : -(o / 2));
    if (lane == 0) item = atomicAdd(&next, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (row0 + rr >= rows_total) continue;
    const int rowi = RowAt(in.tab, row0 + rr);
    const int sub = kSub ? lane / s.smus : 0;
    const int n = slot * per + sub;
    const int col0 = kCols == 1 ? lane - sub * s.smus : 2 * lane;
    const int cols = sub < per && n < s.snu ? min(max(s.smus - col0, 0), kCols) : 0;
    // Lanes without a texel march column 0 of node 0 and keep nothing.
    const int second = cols == 2 ? 1 : 0;
    const float4* col = in.dJ + (cols > 0 ? n * s.smus + col0 : 0);
    // The tasks of the warp's columns, packed: any lane can march any of them,
    // as the taps are shuffles.
    int count = 0;
    auto add = [&](bool any, int m, int use, float nu) {
      const unsigned mask = __ballot_sync(0xffffffffu, any);
      if (any)
        tasks[count + __popc(mask & ((1u << lane) - 1u))] =
            NodeTask{nu, (lane * kCols + m) << 8 | use};
      count += __popc(mask);
    };
#pragma unroll
    for (int m = 0; m < kCols; ++m) {
      const int colm = m < cols ? col0 + m : 0;
      const NodeNu own = TexelNu(in, rowi, colm, min(n, s.snu - 1));
      add(m < cols && own.side < 0, m, 1, own.nu);
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        // Some texel's nu is clamped at an end where the end node's own is.
        const NodeNu end = TexelNu(in, rowi, colm, side == 0 ? 0 : s.snu - 1);
        const int half = n - (int)floorf((end.nu + 1.0f) * 0.5f * nodes1);
        add(m < cols && end.side == side && (half == 0 || half == 1), m, 2 + 2 * side + half,
            end.nu);
      }
    }
    __syncwarp();
    const RaySample* srow = samp + rr * kNodeSamples;
    auto march = [&](auto per_lane, int first) {
      constexpr int kTasks = decltype(per_lane)::value;
      float magic[kSub ? kTasks : 1], rmu_s[kTasks], nu[kTasks];
      F3 acc[kTasks];
#pragma unroll
      for (int k = 0; k < kTasks; ++k) {
        const int t = first + 32 * k + lane;
        const NodeTask task = t < count ? tasks[t] : NodeTask{0.0f, 0};
        const int at = task.code >> 8, of = kSub ? at / s.smus * s.smus : 0;
        nu[k] = task.nu;
        rmu_s[k] = in.tab.rows[rowi].r * in.tab.cols[at - of].mu_s;
        magic[kSub ? k : 0] = kRoundMagic + float(of);
        acc[k] = f3(0.0f);
      }
      MarchNodes<kCols, kTasks, kPair, kSub>(srow, col, second, nS, map, magic, rmu_s, nu, acc);
#pragma unroll
      for (int k = 0; k < kTasks; ++k) {
        const int t = first + 32 * k + lane;
        if (t >= count) continue;
        const NodeTask task = tasks[t];
        const int at = task.code >> 8, use = task.code & 255;
        if (use == 1) {
          StoreMultiple(in, rowi * W + slot * per * s.smus + at, acc[k], task.nu);
        } else {
          const float x = (task.nu + 1.0f) * 0.5f * nodes1, l1 = x - floorf(x);
          const int of = kSub ? at / s.smus * s.smus : 0;
          edge[(rr * 4 + use - 2) * s.smus + at - of] =
              to4(acc[k] * (use & 1 ? l1 : 1.0f - l1), 0.0f);
        }
      }
    };
    for (int first = 0; first < count;) {
      const int left = count - first;
      if (kCols == 2 && left > 96) {
        march(std::integral_constant<int, 4>(), first);
        first += 128;
      } else if (kCols == 2 && left > 64) {
        march(std::integral_constant<int, 3>(), first);
        first += 96;
      } else if (left > 32) {
        march(std::integral_constant<int, 2>(), first);
        first += 64;
      } else {
        march(std::integral_constant<int, 1>(), first);
        first += 32;
      }
    }
    __syncwarp();
  }
  __syncthreads();

  // The clamped texels: the sum of their two nodes' parts.
  for (int e = threadIdx.x; e < R * W; e += kMultipleFastThreads) {
    const int rr = e / W, x = e - rr * W;
    if (row0 + rr >= rows_total) break;
    const int rowi = RowAt(in.tab, row0 + rr);
    const int n = x / s.smus, colx = x - n * s.smus;
    const NodeNu ang = TexelNu(in, rowi, colx, n);
    if (ang.side < 0) continue;
    const float4 u = edge[(rr * 4 + 2 * ang.side) * s.smus + colx];
    const float4 v = edge[(rr * 4 + 2 * ang.side + 1) * s.smus + colx];
    StoreMultiple(in, rowi * W + x, F3{u.x + v.x, u.y + v.y, u.z + v.z}, ang.nu);
  }
}

// MultipleKind 1 (kCols 1; 64 registers, 4 blocks per SM) and 2 (kCols 2;
// 128 registers, 2 blocks per SM: 3 at 80 registers spill and run 1% slower).
// An instance is always marched by the same kernel, whatever shapes share its
// launch: the blocks of the other instances return at once.
template <int kCols>
__global__ void __launch_bounds__(kMultipleFastThreads, kCols == 1 ? 4 : 2)
k_multiple_nodes(const Instance* __restrict__ insts, WorkList wl) {
  extern __shared__ float4 smem[];
  int local;
  const Instance& in = insts[FindEntry(wl, blockIdx.x, &local)];
  if (MultipleKind(in.s) != kCols) return;
  if (kCols == 2 && in.s.smus % 2 == 0 && ((size_t)in.dJ & 31) == 0) {
    MultipleNodesBlock<kCols, kCols == 2, false>(in, local, smem);
  } else if (kCols == 1 && in.s.smus <= 16) {
    MultipleNodesBlock<kCols, false, kCols == 1>(in, local, smem);
  } else {
    MultipleNodesBlock<kCols, false, false>(in, local, smem);
  }
}

__global__ void __launch_bounds__(kMultipleFastThreads, 4)
k_multiple_fast(const Instance* __restrict__ insts, WorkList wl) {
  extern __shared__ float4 smem[];
  int local;
  const Instance& in = insts[FindEntry(wl, blockIdx.x, &local)];
  if (MultipleKind(in.s) != 4) return;
  if (in.s.sw() <= kMultipleFastThreads) {
    MultipleFastBlock<1>(in, local, smem);
  } else {
    MultipleFastBlock<kMultipleFastMaxCols>(in, local, smem);
  }
}

bool MultipleFastFits(const Shape& s) {
  return MultipleByNodes(s) || s.sw() <= kMultipleFastThreads * kMultipleFastMaxCols;
}
int MultipleFastTiles(const Shape& s) {
  const int rows = MultipleByNodes(s) ? NodeRows(s) : MultipleDims(s).rows;
  return (s.sr * s.smu + rows - 1) / rows;
}
static int MultipleLinesSmem(const Shape& s) {
  const MultipleFastDims d = MultipleDims(s);
  return d.rows * kRaySamples * (int)sizeof(RaySample) + 2 * d.group * d.rows * s.sw() * 16;
}
int MultipleFastSmem(const Shape& s) {
  if (!MultipleByNodes(s)) return MultipleLinesSmem(s);
  return NodeRows(s) * (kNodeSamples * (int)sizeof(RaySample) + 4 * s.smus * 16) +
         kNodeWarps * 96 * MultipleKind(s) * (int)sizeof(NodeTask);
}

cudaError_t LaunchMultipleFast(const Instance* insts, WorkList wl, int tiles, int smem_bytes,
                               cudaStream_t st) {
  // smem_bytes: the largest MultipleFastSmem of the work list's instances.
  const size_t bytes = (size_t)smem_bytes;
  if (wl.kinds & 1) k_multiple_nodes<1><<<tiles, kMultipleFastThreads, bytes, st>>>(insts, wl);
  if (wl.kinds & 2) k_multiple_nodes<2><<<tiles, kMultipleFastThreads, bytes, st>>>(insts, wl);
  if (wl.kinds & 4) k_multiple_fast<<<tiles, kMultipleFastThreads, bytes, st>>>(insts, wl);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Single scattering, restructured (functions.glsl:650-730, :933-945).
//
// As for multiple scattering, a sample's r, altitude, densities and the
// transmittance from the texel to it depend on the texel's row only; the
// transmittance from the sample to the sun depends on mu_s at the sample,
// hence on the texel's column.  Its LUT lookup happens at the sample's
// (rho, r): a fixed pair of transmittance LUT rows.  Per sample the block
// interpolates those two rows into a line of W_T columns in shared memory; a
// texel computes the x_mu of its sun direction and reads 2 line entries.
//
// Bound by the L1 data pipe (91% busy before the following, 37 wavefronts per
// warp and sample): the lines' rows, the sample's constants and the taps.  So
// an entry is three floats (a tap is three conflict-free 4-byte loads, where
// 16-byte loads of scattered entries conflict), neighbouring lanes hold the nu
// nodes of one mu_s column (whose taps start at one entry and drift apart
// along the ray, and whose samples are in the planet's shadow together: a
// shadowed sample reads nothing), a thread keeps its line columns of the last
// two rows across samples, and two texel columns of a thread share a sample's
// loads.  Per 16-instance launch at the reference's shape 3.55 -> 2.69 ms, one
// high-resolution instance 2.74 -> 2.60 ms, one of half size 55 -> 35 us; over
// shapes of 64 to 500 line columns and 24 to 1024 texel columns 0 to 45% less.
// ---------------------------------------------------------------------------
constexpr int kSingleSamples = kSingleScatteringSamples + 1;
constexpr int kSingleThreads = 128;   // of a block of a shape of up to 256 columns

struct __align__(16) SunSample {
  float rho, r;              // the sample's rho and r
  float d;                   // distance from the texel's point along its ray
  float inv_2er;             // 1 / (2 r sin(theta_h) alpha_s), sin(theta_h) = Rb / r
  F3 tr;                     // transmittance texel -> sample x Rayleigh density x weight
  float inv_range;           // 1 / (d_max - d_min) of the transmittance mapping
  F3 tm;                     // as tr, Mie
  float pad;
  int t0, t1;                // element offsets of the even and the odd one of the two
  float w0, w1;              //   transmittance LUT rows around rho, and their weights
};

// Rows of a block of `columns` texel columns, and samples per line stage.
__host__ __device__ inline MultipleFastDims SingleDims(const Shape& s, int columns) {
  int rows = columns / s.sw();
  rows = rows < 1 ? 1 : (rows > 4 ? 4 : rows);
  if (s.tune[2] > 0 && (s.tune[2] < rows || columns > kSingleThreads)) rows = s.tune[2];
  int group = 32768 / (2 * 16 * rows * s.tw);
  group = group < 1 ? 1 : (group > 4 ? 4 : group);
  if (s.tune[3] > 0) group = s.tune[3];
  return MultipleFastDims{rows, group};
}
int SingleFastSmem(const Shape& s) {
  const MultipleFastDims d = SingleDims(s, kSingleThreads);
  return d.rows * kSingleSamples * (int)sizeof(SunSample) +
         2 * d.group * d.rows * (s.tw + 1) * (int)sizeof(F3);
}
// The limit of the shapes and tunings taken: blocks of 256 columns, entries of
// 16 bytes (no block needs more).
int SingleFastLimit(const Shape& s) {
  const MultipleFastDims d = SingleDims(s, kMultipleFastThreads);
  return d.rows * kSingleSamples * (int)sizeof(SunSample) + 2 * d.group * d.rows * s.tw * 16;
}
bool SingleFastFits(const Shape& s) {
  return s.sw() <= kMultipleFastThreads * kMultipleFastMaxCols &&
         SingleFastLimit(s) <= 48 * 1024;
}
int SingleFastTiles(const Shape& s) {
  const int rows = SingleDims(s, kSingleThreads).rows;
  return (s.sr * s.smu + rows - 1) / rows;
}

// Whether a (rows, group) block shape is launchable for shape s: one texel
// column per thread needs rows x W <= 256 (wider rows take one row per
// block), and the shared memory of the lines must stay within 48 KB (of the
// shapes without lines too: a tuning is valid or not whichever kernel is taken).
bool FastTuningValid(const Shape& s, bool single, int rows, int group) {
  if (rows < 1 || rows > 4 || group < 1 || group > 8) return false;
  const int W = s.sw();
  if (W > kMultipleFastThreads * kMultipleFastMaxCols) return false;
  if (rows > 1 && rows * W > kMultipleFastThreads) return false;
  Shape t = s;
  t.tune[single ? 2 : 0] = rows;
  t.tune[single ? 3 : 1] = group;
  return (single ? SingleFastLimit(t) : MultipleLinesSmem(t)) <= 48 * 1024;
}

int FastTuningRows(const Shape& s, bool single, int rows) {
  if (!single) return MultipleByNodes(s) ? 0 : rows;
  Shape t = s;
  t.tune[2] = rows;
  return SingleDims(t, kSingleThreads).rows;
}

// Sample i of the ray of LUT row `rowi` (the per-sample part of
// SingleScatteringTexel that does not depend on mu_s or nu).
__device__ SunSample MakeSunSample(const Instance& in, int rowi, int i) {
  const Consts& c = in.c;
  const Shape& s = in.s;
  const TexelRow row = in.tab.rows[rowi];
  const bool ground = row.ground != 0;
  const float dx = row.d / float(kSingleScatteringSamples);
  const float d = float(i) * dx;
  const float e = float(kSingleScatteringSamples - i) * dx;
  const RadialPoint p = PointFromRho2(c, RayRho2(row, d, e));
  const TStart start = MakeTStart(c, s, in.T, in.Tau, row.rho, row.r,
                                  ground ? -row.rmu : row.rmu, row.delta);
  const F3 t = SegmentTransmittance(c, s, in.T, in.Tau, row.rmu, row.delta, p, d, ground, start);
  const float w = (i == 0 || i == kSingleScatteringSamples) ? 0.5f : 1.0f;
  const float Y = p.rho / c.H * float(s.th - 1);
  const float fy = floorf(Y);
  const int j0 = ClampIdx((int)fy, s.th), j1 = ClampIdx((int)fy + 1, s.th);
  SunSample ss;
  const float b = Y - fy;
  const bool odd = j0 & 1;   // j1 is even (or j0 again, of weight b = 0)
  ss.t0 = (odd ? j1 : j0) * s.tw;
  ss.t1 = (odd ? j0 : j1) * s.tw;
  ss.w0 = odd ? b : 1.0f - b;
  ss.w1 = odd ? 1.0f - b : b;
  ss.rho = p.rho;
  ss.r = p.r;
  // 1 / 0 = +inf for a point sun: the smoothstep then becomes a step at 0.
  ss.inv_2er = 1.0f / p.r * (1.0f / (2.0f * (c.Rb / p.r * c.alpha_s)));
  ss.d = d;
  ss.tr = t * (ProfileDensity(c.prof_r, p.h) * w);
  ss.tm = t * (ProfileDensity(c.prof_m, p.h) * w);
  const float d_min = (c.H - p.rho) * (c.H + p.rho) / (c.Rt + p.r);
  ss.inv_range = 1.0f / (p.rho + c.H - d_min);
  ss.pad = 0.0f;
  return ss;
}

// Up to kCols texel columns per thread; kBuild: the line columns a thread keeps
// in registers.  kThreads: of the block, 0 where the launch says how many (any
// number gives the same LUTs).
template <int kCols, int kBuild, int kThreads>
__device__ __forceinline__ void SingleFastBlock(const Instance& in, int local, float4* smem,
                                                float magic) {
  const Shape s = in.s;
  const Consts& c = in.c;
  const MultipleFastDims dims = SingleDims(s, kSingleThreads);
  const int threads = kThreads > 0 ? kThreads : (int)blockDim.x;
  const int W = s.sw(), R = dims.rows, G = dims.group, TW = s.tw;
  const int rows_total = s.sr * s.smu;
  [[maybe_unused]] const long long nT = s.t_texels();   // checked build
  const int row0 = local * R;
  SunSample* samp = reinterpret_cast<SunSample*>(smem);                       // [R][51]
  // [2][G][R][TW + 1] entries of three floats; entry 0 of a line is below its
  // first column, for the tap of weight 0 there.
  float* line = reinterpret_cast<float*>(smem + R * kSingleSamples * (int)(sizeof(SunSample) / 16));
  const int line_floats = 3 * (TW + 1);

  for (int e = threadIdx.x; e < 2 * G * R * 3; e += threads)
    line[e / 3 * line_floats + e % 3] = 0.0f;
  for (int e = threadIdx.x; e < R * kSingleSamples; e += threads) {
    const int rr = e / kSingleSamples, i = e - rr * kSingleSamples;
    if (row0 + rr < rows_total) samp[e] = MakeSunSample(in, row0 + rr, i);
  }

  // Threads per row: a row's columns are x_t, x_t + stride, ...
  const int stride = R == 1 ? threads : W;
  const int rr = (int)threadIdx.x / stride;
  const int x_t = (int)threadIdx.x - rr * stride;
  const int rowi = row0 + rr;
  const bool active = rr < R && rowi < rows_total;
  const int nmax = W - 1;
  float rmu_s[kCols], nu[kCols];
  F3 sum_r[kCols], sum_m[kCols];
  if (active) {
    const TexelRow row = in.tab.rows[rowi];
#pragma unroll
    for (int m = 0; m < kCols; ++m) {
      const int x = min(x_t + m * stride, nmax);
      const int col = x / s.snu, n = x - col * s.snu;
      const TexelAngles ang = MakeAngles(s, row, in.tab.cols[col], n);
      rmu_s[m] = row.r * ang.mu_s;
      nu[m] = ang.nu;
      sum_r[m] = f3(0.0f);
      sum_m[m] = f3(0.0f);
    }
  }
  __syncthreads();

  const float H = c.H, H2 = c.H * c.H;
  const float tw1 = float(TW - 1);
  const uint32_t last = ((uint32_t)TW + (uint32_t)__float_as_int(magic)) * 12u;
  const int line_stride = G * R * line_floats;
  const int stages = (kSingleSamples + G - 1) / G;
  // The block's threads build the lines of its rows side by side, line columns
  // x_b, x_b + per_row, ... of row q_b each.  Where these are at most kBuild, a
  // thread keeps those of the last even and the last odd LUT row in registers:
  // of the rows around consecutive samples of a ray only 0.7 per sample are
  // new at the reference's shape (predicated loads).
  const int per_row = R == 1 ? threads : threads / R;
  const int q_b = R == 1 ? 0 : (int)threadIdx.x / per_row;
  const int x_b = R == 1 ? (int)threadIdx.x : (int)threadIdx.x - q_b * per_row;
  const bool builds = q_b < R && row0 + q_b < rows_total && x_b < TW;
  int o0 = -1, o1 = -1;
  float4 ra[kBuild], rb[kBuild];
#pragma unroll
  for (int k = 0; k < kBuild; ++k) ra[k] = rb[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int stage = 0; stage < stages; ++stage) {
    float* buf = line + (stage & 1) * line_stride;
    const int first = stage * G;
    const int count = min(G, kSingleSamples - first);
    // The two transmittance LUT rows of each sample, interpolated in rho.
    if (builds) {
      const float4* col = in.T + x_b;
      float* out = buf + q_b * line_floats + 3 * (x_b + 1);
      const SunSample* srow = samp + q_b * kSingleSamples + first;
      if (TW <= per_row * kBuild) {
        for (int g = 0; g < count; ++g) {
          const int4 v = *reinterpret_cast<const int4*>(&srow[g].t0);
          const float w0 = __int_as_float(v.z), w1 = __int_as_float(v.w);
#pragma unroll
          for (int k = 0; k < kBuild; ++k) {
            const bool mine = x_b + k * per_row < TW;
            const int xk = mine ? k * per_row : 0;
            LoadIf(ra[k], ATMO_LINE_PTR(col, v.x, xk, nT - x_b), mine && v.x != o0);
            LoadIf(rb[k], ATMO_LINE_PTR(col, v.y, xk, nT - x_b), mine && v.y != o1);
          }
          o0 = v.x;
          o1 = v.y;
#pragma unroll
          for (int k = 0; k < kBuild; ++k) {
            if (x_b + k * per_row < TW) {
              out[3 * k * per_row] = fmaf(w1, rb[k].x, w0 * ra[k].x);
              out[3 * k * per_row + 1] = fmaf(w1, rb[k].y, w0 * ra[k].y);
              out[3 * k * per_row + 2] = fmaf(w1, rb[k].z, w0 * ra[k].z);
            }
          }
          out += R * line_floats;
        }
      } else {
        for (int g = 0; g < count; ++g) {
          const int4 v = *reinterpret_cast<const int4*>(&srow[g].t0);
          const float w0 = __int_as_float(v.z), w1 = __int_as_float(v.w);
          for (int x = 0; x_b + x < TW; x += per_row) {
            const float4 a = __ldg(ATMO_LINE_PTR(col, v.x, x, nT - x_b));
            const float4 b = __ldg(ATMO_LINE_PTR(col, v.y, x, nT - x_b));
            out[3 * x] = fmaf(w1, b.x, w0 * a.x);
            out[3 * x + 1] = fmaf(w1, b.y, w0 * a.y);
            out[3 * x + 2] = fmaf(w1, b.z, w0 * a.z);
          }
          out += R * line_floats;
        }
      }
    }
    __syncthreads();
    if (active) {
      for (int g = 0; g < count; ++g) {
        const SunSample& sm = samp[rr * kSingleSamples + first + g];
        // The line's last column, less the bits of the magic.
        const uint32_t row =
            (uint32_t)__cvta_generic_to_shared(buf + (g * R + rr) * line_floats) + last;
#pragma unroll
        for (int m = 0; m < kCols; ++m) {
          if (x_t + m * stride >= W) break;
          // GetTransmittanceToSun (functions.glsl:552-563) at the sample, with
          // the lookup mapping of TransmittanceCoords.
          const float rmu = clampf(fmaf(sm.d, nu[m], rmu_s[m]), -sm.r, sm.r);
          // smoothstep(-e, e, mu_s - cos(theta_h)), cos(theta_h) = -rho / r.
          const float up = sm.rho + rmu, down = sm.rho - rmu;
          const float st = FmaSat(up, sm.inv_2er, 0.5f);
          // A sample in the planet's shadow adds nothing.
          if (st > 0.0f) {
            // With rho^2 - (r mu)^2 = up down, the distance to the top boundary
            // less its least value is up + up down / (H + sq).  H^2 - up down:
            // zero, or a difference of floats far above FP32's normal range
            // (normal); up and down: zero, or sums of lengths whose exact values
            // are multiples of their operands' ulps (normal); H + sq >= H.
            const float sq = SqrtFtz(fmaxf(fmaf(-up, down, H2), 0.0f));
            const float x = FmaSat(fmaf(up, DivFtz(down, H + sq), up), sm.inv_range, 0.0f);
            const float cell = __fmaf_rd(x, tw1, magic);
            const float gw = fmaf(x, tw1, magic - cell);   // weight of the lower column
            const uint32_t at = row + (uint32_t)__float_as_int(cell) * (uint32_t)-12;
            const F3 lo = LoadShared3<-12>(at), hi = LoadShared3<0>(at);
            const F3 tsun = F3{fmaf(gw, lo.x - hi.x, hi.x), fmaf(gw, lo.y - hi.y, hi.y),
                               fmaf(gw, lo.z - hi.z, hi.z)} * (st * st * fmaf(-2.0f, st, 3.0f));
            sum_r[m] = fma3(tsun, sm.tr, sum_r[m]);
            sum_m[m] = fma3(tsun, sm.tm, sum_m[m]);
          }
        }
      }
    }
  }

  if (!active) return;
  const float dx = in.tab.rows[rowi].d / float(kSingleScatteringSamples);
#pragma unroll
  for (int m = 0; m < kCols; ++m) {
    const int x = x_t + m * stride;
    if (x >= W) break;
    const int col = x / s.snu, n = x - col * s.snu;
    StoreSingleScattering(in, (long long)rowi * W + n * s.smus + col, sum_r[m] * dx * c.solar * c.rayleigh,
                          sum_m[m] * dx * c.solar * c.mie_sca);
  }
}

// A kernel per SingleKind, so that each has the registers it needs.  Blocks per
// SM: kSingleTwo 7 (72 registers; 6 take 1% and 8 take 3% longer),
// kSingleTwoWide 4 (3 take 3% longer over 5 to 15 x 32 to 64 columns),
// kSingleFour 3 (4 spill, and take 2 to 8% longer below 600 rows).
ATMO_HD constexpr int SingleThreads(int kind) {
  return kind == kSingleTwo ? kSingleThreads : kMultipleFastThreads;
}
ATMO_HD constexpr int SingleBlocks(int kind) {
  return kind == kSingleTwo ? 7 : kind == kSingleFour ? 3 : 4;
}
template <int kKind>
__global__ void __launch_bounds__(SingleThreads(kKind), SingleBlocks(kKind))
k_single_fast(const Instance* __restrict__ insts, WorkList wl, float magic) {
  extern __shared__ float4 smem[];
  int local;
  const Instance& in = insts[FindEntry(wl, blockIdx.x, &local)];
  if (SingleKind(in.s) != kKind) return;
  constexpr int kThreads = kKind == kSingleOne ? 0 : SingleThreads(kKind);
  constexpr int kCols = kKind == kSingleOne ? 1 : kKind == kSingleFour ? 4 : 2;
  if (in.s.tw <= kThreads) {
    SingleFastBlock<kCols, 1, kThreads>(in, local, smem, magic);
  } else {
    SingleFastBlock<kCols, 2, kThreads>(in, local, smem, magic);
  }
}

cudaError_t LaunchSingleFast(const Instance* insts, WorkList wl, int tiles, int smem_bytes,
                             cudaStream_t st) {
  // smem_bytes: the largest SingleFastSmem of the work list's instances.
  const size_t bytes = (size_t)smem_bytes;
  if (wl.kinds & kSingleOne) {
    // Where every block of the launch is resident at once (4 per SM), threads
    // without a texel column help with the samples and the lines: one instance
    // of half size (1024 rows of 64 columns) 43 us against 51; 8 of them 260
    // us against 234.  Rows of more than 128 columns need them.
    const bool all = tiles <= 4 * kSmCount || wl.kinds & kSingleOneWide;
    k_single_fast<kSingleOne><<<tiles, all ? kMultipleFastThreads : kSingleThreads, bytes, st>>>(
        insts, wl, kRoundMagic);
  }
  if (wl.kinds & kSingleTwo)
    k_single_fast<kSingleTwo><<<tiles, kSingleThreads, bytes, st>>>(insts, wl, kRoundMagic);
  if (wl.kinds & kSingleTwoWide)
    k_single_fast<kSingleTwoWide>
        <<<tiles, kMultipleFastThreads, bytes, st>>>(insts, wl, kRoundMagic);
  if (wl.kinds & kSingleFour)
    k_single_fast<kSingleFour><<<tiles, kMultipleFastThreads, bytes, st>>>(insts, wl, kRoundMagic);
  return cudaGetLastError();
}

__global__ void k_to_half(const float4* __restrict__ src, __half2* __restrict__ dst, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 v = src[i];
  dst[2 * i] = __floats2half2_rn(v.x, v.y);
  dst[2 * i + 1] = __floats2half2_rn(v.z, v.w);
}

cudaError_t LaunchToHalf(const float4* src, void* dst, long long n, cudaStream_t st) {
  int blocks = (int)((n + 255) / 256);
  k_to_half<<<blocks, 256, 0, st>>>(src, reinterpret_cast<__half2*>(dst), n);
  return cudaGetLastError();
}

// FP32 FMA throughput probe: 8 independent FMA chains per thread.
__global__ void k_fma_probe(float* out, int iters, float a, float b) {
  float x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = threadIdx.x * 1e-3f + i;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = fmaf(x[i], a, b);
  }
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += x[i];
  if (s == 1234.5f) out[blockIdx.x] = s;   // keeps the chains live
}

cudaError_t MeasureFp32Peak(double* tflops) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  float* out = nullptr;
  cudaError_t e = cudaMalloc(&out, sizeof(float) * sms * 8);
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  k_fma_probe<<<blocks, threads>>>(out, iters, 0.999f, 1e-3f);   // warm-up
  cudaEventRecord(t0);
  const int reps = 5;
  for (int r = 0; r < reps; ++r) k_fma_probe<<<blocks, threads>>>(out, iters, 0.999f, 1e-3f);
  cudaEventRecord(t1);
  e = cudaEventSynchronize(t1);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  cudaFree(out);
  double flops = 2.0 * 8.0 * iters * (double)blocks * threads * reps;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return e == cudaSuccess ? cudaGetLastError() : e;
}

ATMO_CHECK_WORD_ACCESSOR(CheckWordFast)

}  // namespace atmo
