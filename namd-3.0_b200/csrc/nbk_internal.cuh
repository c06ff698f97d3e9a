// Device-side types and the FP32 pair math of the B200 nonbonded path.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nbk.h"

namespace nbk {

constexpr int kWarp = 32;
// Forces are accumulated as 64-bit fixed point with 2^32 units per kcal/mol/A.
constexpr float kForceScale = 4294967296.0f;
constexpr double kForceScaleInv = 1.0 / 4294967296.0;
// Energies and virials are accumulated as 64-bit fixed point with 2^30 units.
constexpr double kEnergyScale = 1073741824.0;
constexpr double kEnergyScaleInv = 1.0 / 1073741824.0;

// Slots of the 64-bit accumulator block (energies, virials, counters).
enum AccSlot {
  kAccEVdw = 0,
  kAccEElec = 1,
  kAccESlow = 2,
  kAccVir = 3,       // 9 entries, virial[3*a+b]
  kAccVirSlow = 12,  // 9 entries
  kAccNumExcl = 21,  // number of excluded pairs within the pairlist cutoff
  kAccNumPairs = 22, // pairs evaluated within the cutoff (energy evaluations only)
  kAccCount = 24
};

// Constants of the energy-switched LJ and C1-split PME real-space pair math.
// The switching constants follow CudaComputeNonbonded::getNonbondedCoef
// (src/CudaComputeNonbonded.C:2318-2349): lj0 = c1(rc^2 - 3 rs^2), lj1 = 2 c1,
// lj2 = -12 c1, lj3 = 12 c1 rs^2 with c1 = 1/(rc^2 - rs^2)^3.
struct NbkConst {
  float cutoff2;
  float plcutoff2;
  float rc2;          // == cutoff2, switching upper end
  float rs2;          // switch distance^2
  float lj0, lj1, lj2, lj3;
  float rc3inv;       // 1/rc^3
  float hA, hB;       // (3 - r^2/rc^2)/(2 rc) = hA + hB r^2
  float beta;         // Ewald coefficient
  float beta2Pi;      // 2 beta / sqrt(pi)
  float one14;        // 1 - scale14
  int ljDim;          // LJ table row length
  int switching;      // 0 when switchdist >= cutoff (plain truncated LJ)
  double hAd, hBd;    // hA, hB in FP64 (precise kernel)
  double betad;       // Ewald coefficient in FP64
};

// FP64 copies of the pair-math constants (the corrections kernel's energies and slow virial).
struct NbkConst64 {
  double rc2, rs2, lj0, lj1, lj2, lj3, rc3inv, hA, hB, beta, beta2Pi, one14;
  int switching;
};

// Bounding box of one 32-atom tile: centre and half-widths.
struct BBox {
  float x, y, z, wx, wy, wz;
};

// Per-list patch-pair record (PatchPairRecord, src/CudaTileListKernel.h:24-29).
struct PatchPair {
  int iatomSize, iatomFreeSize, jatomSize, jatomFreeSize;
};

// Sparse-list descriptor built on the host for every (compute, i-tile).
struct ListSeed {
  int icompute;
  int itile;       // i-tile index inside patch 1
  int jcapStart;   // first j-tile slot reserved for this list
  int pad;
};

// Shift of the i atoms, offset . lattice, as the reference's expression
// o.x a + o.y b + o.z c (src/CudaComputeNonbondedKernel.cu:720-722) rounds
// once contracted: the first product fused into the first sum, fma(o.x, a,
// o.y b), then fma(o.z, c, that). Written out as FMAs so that host and device
// agree bit for bit. (With an orthorhombic lattice only one term of each
// component is not 0, and every order gives the same bits.)
__device__ __forceinline__ float3 shiftOf(const float3 o, const float3 a, const float3 b,
                                          const float3 c) {
  float3 s;
  s.x = __fmaf_rn(o.z, c.x, __fmaf_rn(o.x, a.x, __fmul_rn(o.y, b.x)));
  s.y = __fmaf_rn(o.z, c.y, __fmaf_rn(o.x, a.y, __fmul_rn(o.y, b.y)));
  s.z = __fmaf_rn(o.z, c.z, __fmaf_rn(o.x, a.z, __fmul_rn(o.y, b.z)));
  return s;
}

// r^2 of d = xj - xi as the reference's dx*dx + dy*dy + dz*dz
// (src/CudaComputeNonbondedKernel.cu:1225-1230) rounds once contracted the same
// way: fma(dz, dz, fma(dx, dx, dy dy)). Its kernels list a pair whose r^2 is
// 182.249985 in this order and exactly plcutoff^2 = 182.25 in the order
// fma(dz, dz, fma(dy, dy, dx dx)) (a triclinic test cell).
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
  return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// erfc(x) = t P(t) exp(-x^2), t = 1/(1 + p x): Hastings' rational form (the
// form of Abramowitz & Stegun 7.1.26) with a degree-7 P whose coefficients
// were fitted by least squares on [0, 4] (oracle/fit_erfc.py; max relative error
// 1.6e-8). `ex` is exp(-x^2), shared with the force's Gaussian term.
constexpr float kErfcP = 4.067848869e-01f;
constexpr float kErfcC0 = 8.043135869e-02f, kErfcC1 = -4.030445941e-01f,
                kErfcC2 = 6.621032108e-01f, kErfcC3 = -3.509793830e-01f,
                kErfcC4 = 3.971568035e-01f, kErfcC5 = 1.455091497e-01f,
                kErfcC6 = 2.400594718e-01f, kErfcC7 = 2.287639988e-01f;
__device__ __forceinline__ float erfcShared(const float x, const float ex) {
  const float t = __fdividef(1.0f, fmaf(kErfcP, x, 1.0f));
  float q = kErfcC0;
  q = fmaf(q, t, kErfcC1);
  q = fmaf(q, t, kErfcC2);
  q = fmaf(q, t, kErfcC3);
  q = fmaf(q, t, kErfcC4);
  q = fmaf(q, t, kErfcC5);
  q = fmaf(q, t, kErfcC6);
  q = fmaf(q, t, kErfcC7);
  return t * q * ex;
}

// ---- two pairs at once with sm_100's packed FP32 instructions --------------
// fma/mul/add .f32x2 issue two IEEE-rounded FP32 operations per instruction,
// so every element below is rounded exactly as the scalar form would be;
// only the number of issued instructions halves.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// Shared-memory accesses by 32-bit address (a base held in a register and an
// immediate offset), so that the pair loop forms no addresses.
__device__ __forceinline__ unsigned sharedAddr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ float4 ldShared4(const unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ int ldShared1(const unsigned a) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 ldShared2(const unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}

// Programmatic dependent launch: waits until the kernel before this one in the
// stream has finished (nothing to wait for in an ordinary launch), and lets the
// kernel after this one be scheduled before this one has finished.
__device__ __forceinline__ void waitForPredecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void admitSuccessor() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// PTX approximate reciprocal, base-2 exponential and reciprocal square root
// (rcp/ex2/rsqrt.approx.ftz.f32). The inputs here are normal numbers (r^2 is
// at least the square of the shortest pair distance, 2^(gaussK r^2) lies in
// (2^-15, 1], 1 + p beta r lies in [1, 3]), where the ftz forms equal the
// non-ftz ones.
__device__ __forceinline__ float rcpApprox(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2Approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrtApprox(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// PTX rsqrt.approx.ftz.f64: relative error below 2^-20 for normal inputs
// (measured 2^-20.1 over [0.5, 200] on B200); callers refine it.
__device__ __forceinline__ double rsqrtApprox64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// Constants of the packed pair math (makePacked, nbk_consts.cu); those that a
// packed instruction reads are held twice. With d = min(rc^2 - r^2, D), D =
// rc^2 - rs^2 and c1 = 1/D^3 the switch is S = c1 d^2 (3 D - 2 d) and (dS/dr)/r
// = 12 c1 d (d - D) = T, so -6 S = d (T - 6 c1 D d). Without switching d = D =
// 1 for every pair, which gives S = 1 and T = 0 exactly.
struct PackedConst {
  float2 dA, dB, hA;    // -12 c1 D, 12 c1, -6 c1 D
  float2 rc3inv;
  float rc2, dMax;      // rc^2 (huge without switching), D
  // the slow force factor: from its table (rows > 0), row k = (c0, c1, c2, c3)
  // in w = s - k D, or from the erfc form
  const float4* tab;
  int tabRows;
  float tabStep, tabInvStep;
  float2 nBeta2Pi;      // -2 beta / sqrt(pi)
  float pBeta, gaussK;  // erfcShared's p times beta; exp(-beta^2 r^2) = 2^(gaussK r^2)
};
// The fit's error relative to the factor's largest value (at r = 0), and the
// rows a table may have (16 KB of shared memory). At 3e-8 the fit is an order
// below the rounding of the erfc form ((1 - erfc term) r^-3 cancels at short
// range), and the benchmark's parameters give 94 rows.
constexpr double kForceTableTol = 3e-8;
constexpr int kForceTableMaxRows = 1024;

// The table in shared memory, as a lane of the force kernel reads it: copies
// interleaved row by row, so that with 8 of them the lanes of a quarter warp
// read from 8 different bank groups whatever rows they want. A row's address
// is base + bits(1.5 2^23 + row) * stride.
struct ForceTable {
  unsigned base, stride;
  float step, invStep, sMax;
};
constexpr float kRowMagic = 12582912.0f;        // 1.5 2^23
constexpr unsigned kRowMagicBits = 0x4B400000u;

// FP32 pair math for two pairs (x and y elements); nB = -B. F, FS = (dE/dr)/r
// of LJ + fast electrostatics and of the slow (PME real-space remainder)
// electrostatics; the caller applies F_i += F (x_j - x_i), F_j -= F (x_j - x_i).
//   LJ      E = (A r^-12 - B r^-6) S(r^2), S = 1 below rs, Hermite switch above
//   fast    E = qq (1/r - (3 - r^2/rc^2)/(2 rc))
//   slow    E = qq ((3 - r^2/rc^2)/(2 rc) + (erfc(beta r) - 1)/r)
// (src/CudaComputeNonbondedInteractions.h:37-159 states the same forms.) Only
// the LJ energy is formed here (doVdwEnergy; e6 = -6 E): the electrostatic
// energies and the slow virial are formed in FP64 by the precise kernel
// (nbk_force.cu). Callers replace the results of an element that is no
// interacting pair (they may be anything, but their r^2 is clamped into the
// table). LJ is taken as r^-6 [(2 A r^-6 - B) (-6 S/r^2) + (A r^-6 -
// B) (dS/dr)/r], which needs the fewest operations. The slow factor (dE/dr)/r =
// qq K(s) comes from the cubic table of K (kTable; 20 issue slots against 34 of
// the erfc form, whose rcp and ex2 it saves, and a smaller error), or, when the
// tolerance needs more rows than the table may have, from the erfc form: with
// x = beta r, t = 1/(1 + p x) and e = exp(-x^2) = 2^(gaussK r^2), erfc = t P(t)
// e and the force factor erfc + (2 beta/sqrt(pi)) r e = (t P(t) + (2
// beta/sqrt(pi)) r) e; the bracket is formed with its sign turned.
template <bool doVdwEnergy, bool doSlow, bool kTable>
__device__ __forceinline__ void pairForce2(const float2 r2, const float2 qq, const float2 A,
                                           const float2 nB, const PackedConst& c,
                                           const ForceTable& T, float2& f, float2& fs, float2& e6) {
  const float2 rinv = make_float2(rsqrtApprox(r2.x), rsqrtApprox(r2.y));
  const float2 rinv2 = mul2(rinv, rinv);
  const float2 rinv3 = mul2(rinv, rinv2);
  const float2 rinv6 = mul2(rinv3, rinv3);
  // scalar: A and B of the two pairs come from two table entries
  const float2 ab6 = make_float2(fmaf(A.x, rinv6.x, nB.x), fmaf(A.y, rinv6.y, nB.y));
  const float2 ab12 = make_float2(fmaf(A.x, rinv6.x, ab6.x), fmaf(A.y, rinv6.y, ab6.y));
  const float2 d = make_float2(fminf(c.rc2 - r2.x, c.dMax), fminf(c.rc2 - r2.y, c.dMax));
  const float2 ds = mul2(d, fma2(c.dB, d, c.dA));
  const float2 s6 = mul2(d, fma2(c.hA, d, ds));
  const float2 lj = fma2(ab12, mul2(rinv2, s6), mul2(ab6, ds));
  f = fma2(lj, rinv6, mul2(qq, add2(c.rc3inv, neg2(rinv3))));
  if (doVdwEnergy) e6 = mul2(mul2(ab6, rinv6), s6);
  if (doSlow && kTable) {
    // row = nearest integer to s/D, in the low bits of t
    const float2 s = make_float2(fminf(r2.x, T.sMax), fminf(r2.y, T.sMax));
    const float2 t = fma2(s, f2(T.invStep), f2(kRowMagic));
    const float2 w = fma2(add2(t, f2(-kRowMagic)), f2(-T.step), s);
    const float4 a = ldShared4(T.base + __float_as_uint(t.x) * T.stride);
    const float4 b = ldShared4(T.base + __float_as_uint(t.y) * T.stride);
    const float2 k = make_float2(fmaf(fmaf(fmaf(a.w, w.x, a.z), w.x, a.y), w.x, a.x),
                                 fmaf(fmaf(fmaf(b.w, w.y, b.z), w.y, b.y), w.y, b.x));
    fs = mul2(qq, k);
  } else if (doSlow) {
    const float2 r = mul2(r2, rinv);
    const float2 t = make_float2(rcpApprox(fmaf(c.pBeta, r.x, 1.0f)),
                                 rcpApprox(fmaf(c.pBeta, r.y, 1.0f)));
    const float2 ex = make_float2(ex2Approx(r2.x * c.gaussK), ex2Approx(r2.y * c.gaussK));
    float2 q = f2(-kErfcC0);
    q = fma2(q, t, f2(-kErfcC1));
    q = fma2(q, t, f2(-kErfcC2));
    q = fma2(q, t, f2(-kErfcC3));
    q = fma2(q, t, f2(-kErfcC4));
    q = fma2(q, t, f2(-kErfcC5));
    q = fma2(q, t, f2(-kErfcC6));
    q = fma2(q, t, f2(-kErfcC7));
    const float2 nCorr = fma2(c.nBeta2Pi, r, mul2(t, q));
    fs = mul2(qq, fma2(fma2(nCorr, ex, f2(1.0f)), rinv3, neg2(c.rc3inv)));
  } else {
    fs = f2(0.0f);
  }
}

// ---- the FP64 slow-term table ------------------------------------------------
// The slow electrostatic energy per unit qq, phi_s(s) = h(s) - erf(beta sqrt(s))/sqrt(s)
// with s = r^2 and h(s) = (3 - s/rc^2)/(2 rc), is an entire function of s (the
// 1/r singularities of erfc(beta r)/r and of the fast part cancel), so a
// piecewise polynomial in s represents it closely: with a step D (a power of
// two, at most 32 A^2), row k holds the degree-5 Chebyshev interpolant on s in
// [k D - D/2, k D + D/2] in the monomial basis of w = s - k D (6 coefficients,
// 48 bytes: three 16-byte loads per pair). Its derivative gives the slow force
// factor, (dE/dr)/r = 2 qq phi_s'(s), without the rc^-3 - r^-3 cancellation of
// the FP32 form. Built on the host at handle creation (buildSlowTable) from
// FP64 erf, with D chosen so that the fit is within 1e-12 of the function's
// scale and its derivative within ~1e-9 (94 rows at the benchmark's
// parameters): a systematic error that, even summed over every pair with the
// same sign, stays below 1e-7 of the slow energy.
constexpr double kSlowTableStepMax = 32.0;  // A^2
constexpr int kSlowTableDeg = 5;
constexpr int kSlowTableDeg1 = kSlowTableDeg + 1;  // coefficients per row
constexpr int kSlowTableRow = 6;  // doubles per row of the global copy
constexpr double kSlowTableTol = 1e-12;  // fit error, relative to max |phi_s| + 1/rc

// Puts the 32 x 32 bits of a tile held as rows (lane i: bit j) into block order
// (lane l: bit 8 J + 4 e + I <-> i = 8 I + (l & 7), j = 8 J + (4 e ^ (l & 4)) +
// (l >> 3), the force kernel's order), or back: the two orders exchange I and
// l >> 3 and swap neighbouring nibbles of lanes with bit 2 set, so the same
// exchange is its own inverse. All lanes call.
__device__ __forceinline__ unsigned blockOrder(const unsigned w, const int lane) {
  unsigned out = 0;
#pragma unroll
  for (int I = 0; I < 4; ++I)
    out |= ((__shfl_sync(0xffffffffu, w, 8 * I + (lane & 7)) >> (lane >> 3)) & 0x11111111u) << I;
  return (lane & 4) ? ((out >> 4) & 0x0f0f0f0fu) | ((out & 0x0f0f0f0fu) << 4) : out;
}

// Component k (0..8, row-major 3x3) of a symmetric tensor stored as
// xx, xy, xz, yy, yz, zz.
__device__ __forceinline__ int symIndex(int k) {
  const int a = k / 3, b = k % 3;
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  return lo == 0 ? hi : (lo == 1 ? 2 + hi : 5);
}

__device__ __forceinline__ unsigned long long toFixedForce(float v) {
  return (unsigned long long)__float2ll_rn(v * kForceScale);
}

__device__ __forceinline__ long long toFixedEnergy(double v) {
  return __double2ll_rn(v * kEnergyScale);
}

// The same conversion from FP32: v * 2^30 is exact, so the result equals
// toFixedEnergy((double)v).
__device__ __forceinline__ long long toFixedEnergyF(float v) {
  return __float2ll_rn(v * 1073741824.0f);
}

__device__ __forceinline__ void atomicAddFixed(long long* p, unsigned long long v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(p), v);
}

__device__ __forceinline__ long long warpSumLL(long long v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double warpSumD(double v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- what the tile-list kernels share ------------------------------------------
// The next item of a work counter, drawn by lane 0 for the warp.
__device__ __forceinline__ int drawItem(int* counter, const int lane) {
  int W = 0;
  if (lane == 0) W = atomicAdd(counter, 1);
  return __shfl_sync(0xffffffffu, W, 0);
}

// One reduction step over a pair of lanes (l and l ^ o): every lane keeps one
// of its two values, the lane whose bit o is clear the first, the other the
// second, and adds its partner's share of the one it keeps.
__device__ __forceinline__ float keepHalf(const float first, const float second, const bool bit,
                                          const int o) {
  const float send = bit ? first : second;
  const float keep = bit ? second : first;
  return keep + __shfl_xor_sync(0xffffffffu, send, o);
}

// ---- kernel argument blocks ---------------------------------------------------
struct ForceArgs {
  const nbk_tile_list* lists;
  const int* numListsDev;      // device count (compacted lists) or NULL
  int numListsHost;            // used when numListsDev == NULL
  const int* tileJatomStart;
  nbk_tile_excl* tileExcls;    // block order; read by the force kernel, written by refineKernel
  int* tileJatomOut;           // refineKernel: j-tile starts of the tiles it keeps
  int* listActive;             // refineKernel: number of tiles kept per list
  int* lenHist;                // refineKernel: lists by length 1..maxLen (clamped), or NULL
  int maxLen;
  int* counts;                 // refineKernel: counts[1] += tiles kept
  const PatchPair* patchPairs; // refineKernel
  const float4* xyzq;
  const int* vdwTypes;
  const int* atomIndex;
  const int2* exclIndexMaxDiff;
  const unsigned* exclBits;
  int numExclWords;
  const float2* ljTable;       // [ljDim*ljDim] (A, B) * scaling
  float3 lata, latb, latc;
  NbkConst c;
  PackedConst pk;              // force kernel
  int tabCopies;               // copies of pk.tab in shared memory (set by the launch)
  long long* force;            // SoA [6][stride] fixed point
  int stride;
  long long* acc;              // [kAccCount]
  int* workCounter;            // next work item to hand out (zeroed before the launch)
  int splitLog2;               // force and precise kernel: 2^splitLog2 work items per list
  long long* compF;            // virial: [numComputes][6] i-force sums per compute (0..2 used)
  const double2* slowTable;    // [slowTableRows * kSlowTableRow / 2] phi_s rows (FP64)
  int slowTableRows;
  double slowStep, slowInvStep;  // table step D (a power of two) and 1/D
  bool beyondTables;           // the cutoff exceeds the distance the tables were built for
  unsigned* liveOut;           // [numJtiles][32] interacting-pair words (force kernel writes,
                               // precise kernel reads), block order
  // replicas (batched evaluation; all NULL for a single system)
  const int* compRep;          // [numComputes] replica of each compute
  const float3* repLat;        // [3*numReplicas] lattice vectors a, b, c
  const float2* repLJ;         // [numReplicas][ljDim*ljDim] (A, -B) * scaling
};

}  // namespace nbk
