// Nonbonded force kernel of the B200 path, and the precise energy / virial
// kernel that follows it on energy and virial evaluations.
//
// forceKernel: one warp owns one tile list (32 i atoms of one patch against
// the j tiles of a compute's partner patch), as CudaComputeNonbondedKernel's
// nonbondedForceKernel does (src/CudaComputeNonbondedKernel.cu:629-1644), but:
//   - a tile is taken as 16 blocks of 8 x 8 atoms, one pass of the warp each
//     (two pairs per lane through sm_100's packed FP32 instructions); i and j
//     forces ride in registers and are reduced over lanes per row of blocks
//     and per group of tiles;
//   - blocks without listed pairs are skipped warp-uniformly;
//   - the lists it reads are already refined (masks from refineKernel, in block
//     order); a pairlist step refines, puts the lists in order, then runs this kernel;
//   - per-tile FP32 partial forces are folded into 64-bit fixed point with
//     integer atomics, so the summed forces do not depend on the order in
//     which lists run; the LJ energy is summed in FP32 per group of tiles and
//     folded the same way; the fast virial comes from the fixed-point forces;
//   - on energy and virial evaluations it stores, per tile and lane, which of
//     the lane's pairs interact (the live words).
// preciseKernel: the electrostatic energies and the slow virial in FP64, from
// the live words: per tile, each lane walks a contiguous range of the tile's
// interacting pairs straight from the live words and evaluates them from
// FP64 geometry (see precisePass); its own
// launch runs at higher occupancy than the register- and shared-memory-heavy
// FP32 loop, which hides the FP64 dependency chains.
#include <algorithm>

#include "nbk_internal.cuh"
#include "nbk_launch.h"

namespace nbk {

constexpr int kForceWarps = 4;
// Forces and energies are folded into fixed point once per group of
// kFoldTiles j tiles (groups counted from the start of the list; a list's
// parts hold whole groups), so every sum is independent of the split.
constexpr int kFoldTiles = 4;
// The tiles [first, last] of part `part` of a list.
__device__ __forceinline__ void listPart(const ForceArgs& a, const nbk_tile_list& tl, const int part,
                                         int& first, int& last) {
  const int split = 1 << a.splitLog2;
  const int chunk = (((tl.jtileEnd - tl.jtileStart + split) >> a.splitLog2) + kFoldTiles - 1) &
                    ~(kFoldTiles - 1);
  first = tl.jtileStart + part * chunk;
  last = min(tl.jtileEnd, first + chunk - 1);
}
__device__ __forceinline__ bool groupEnds(const nbk_tile_list& tl, const int jt, const int last) {
  return ((jt - tl.jtileStart + 1) & (kFoldTiles - 1)) == 0 || jt == last;
}
constexpr int kForceThreads = kForceWarps * kWarp;
constexpr size_t kForceTableBytes = 16 * 1024;  // slow force table copies per CTA

// FP64 quantities of the precise pass; after a tile's pass lane q < kNumQ
// holds quantity q: the fast and slow electrostatic energies, then the six
// independent components of the slow virial (xx, xy, xz, yy, yz, zz).
constexpr int kQElec = 0, kQSlow = 1, kQVir = 2, kNumQ = 8;

// virialSlow[3a+b] slots of symmetric component m (xx, xy, xz, yy, yz, zz);
// s1 < 0 for the diagonal.
__device__ __forceinline__ void symSlots(int m, int& s0, int& s1) {
  s0 = m == 0 ? 0 : m == 1 ? 1 : m == 2 ? 2 : m == 3 ? 4 : m == 4 ? 5 : 8;
  s1 = m == 1 ? 3 : m == 2 ? 6 : m == 4 ? 7 : -1;
}

// Adds the force kernel's LJ energy (lane 0) to one replica's accumulators.
template <bool doEnergy>
__device__ __forceinline__ void flushVdw(long long* acc, int lane, long long& accVdw) {
  if (doEnergy && lane == 0 && accVdw != 0) atomicAddFixed(&acc[kAccEVdw], (unsigned long long)accVdw);
  accVdw = 0;
}

// Adds the precise kernel's accumulators to one replica's block: lane
// q < kNumQ its quantity q (accQ), and the warp's pair count.
template <bool doEnergy>
__device__ __forceinline__ void flushPrecise(long long* acc, int lane, long long& accQ, int& npair) {
  if (lane < kNumQ && accQ != 0) {
    if (lane == kQElec) {
      atomicAddFixed(&acc[kAccEElec], (unsigned long long)accQ);
    } else if (lane == kQSlow) {
      atomicAddFixed(&acc[kAccESlow], (unsigned long long)accQ);
    } else {
      int s0, s1;
      symSlots(lane - kQVir, s0, s1);
      atomicAddFixed(&acc[kAccVirSlow + s0], (unsigned long long)accQ);
      if (s1 >= 0) atomicAddFixed(&acc[kAccVirSlow + s1], (unsigned long long)accQ);
    }
  }
  if (doEnergy) {
    int s = npair;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0 && s) atomicAddFixed(&acc[kAccNumPairs], (unsigned long long)s);
  }
  accQ = 0;
  npair = 0;
}

// FP64 geometry of one interacting pair: d = x_j - x_i and the charge product.
struct PairTerms {
  double dx, dy, dz, qq;
};

// The warp's atoms as the precise pass reads them: the list's i atoms in FP64
// (shifted by the exact lattice translation) as two rows of 32 (x, y) and
// (z, q) pairs, and the current j tile as it is stored (FP32 x, y, z, q, exact
// in FP64). A pair reads two 16-byte entries of its i atom and one of its j
// atom: the j reads span the 512 bytes of the row, half of what FP64 rows
// would, and the four conversions to FP64 cost less than the second load. The
// j row is turned: atom j lies at 8 (j & 3) + (j >> 2). Neighbouring lanes walk
// the pairs of neighbouring owners l, whose i atoms differ in l & 7 and whose j
// atoms share l >> 3 and differ in their bit's J and e, so that with both rows
// the lanes of a quarter warp read from different bank groups.
struct Atoms64 {
  double2 ixy[kWarp], izq[kWarp];
  float4 j[kWarp];
};

// One lane's precise-pass sums over the current tile group.
struct LaneSums {
  double eE, eS, w0, w1, w2, w3, w4, w5;
};

// The slow-term table as the precise pass reads it. kCopies > 0: kCopies
// interleaved copies in shared memory (s_slowTab), 16-byte pair n of row k of
// copy c at s_slowTab[(k * P + n) * kCopies + c] with P = kSlowTableDeg1 / 2;
// lane l reads copy l % kCopies, so with 8 copies the 8 lanes of a quarter
// warp (one 16-byte bank group each) never conflict, whatever rows they read;
// fewer copies conflict, at less than reads from the L1 cache cost.
// kCopies == 0: the global copy (kSlowTableRow doubles per row); kBeyond: the
// same, with pairs beyond the table from the formula.
constexpr int kBeyond = -1;
extern __shared__ __align__(16) double2 s_slowTab[];

struct SlowTable {
  const double2* gl;
  unsigned last;
  double step, invStep;
  double sMax;  // centre of the last row
};

// phi_s and phi_s' from the formula, for pairs beyond the table: with E = erf(beta
// r)/r and G = 2 beta/sqrt(pi) e^{-beta^2 s}, E' = (G - E)/(2 s). Out of line: few
// evaluations reach there.
__device__ __noinline__ double2 slowTermsDirect(const NbkConst& c, const double s) {
  const double r = sqrt(s), E = erf(c.betad * r) / r;
  const double G = c.betad * 1.1283791670955126 * exp(-c.betad * c.betad * s);  // 2/sqrt(pi)
  return make_double2(fma(c.hBd, s, c.hAd) - E, c.hBd - (G - E) / (2.0 * s));
}

template <int kCopies>
__device__ __forceinline__ double2 slowPair(const SlowTable& T, const unsigned k, const int n,
                                            const int lane) {
  if constexpr (kCopies > 0) {
    return s_slowTab[(k * (kSlowTableDeg1 / 2) + n) * kCopies + (lane & (kCopies - 1))];
  } else {
    return __ldg(T.gl + (size_t)k * (kSlowTableRow / 2) + n);
  }
}

// The FP64 terms of one interacting pair (qq = 0 contributes exact zeros):
// the fast energy qq (1/r - h(s)) with 1/r from the FP64 approximation
// refined by one Newton step, and from the slow-term table the slow energy
// qq phi_s(s) and the slow virial -2 qq phi_s'(s) d (x) d. The geometry is
// FP64 throughout: the electrostatic totals are small differences of large
// sums (for 9,000 water atoms the fast energy is 4e-5 of the sum of its pair
// terms' magnitudes), so even the unbiased FP32 rounding of r^2 would move
// them by ~3e-6.
template <bool doEnergy, bool doVirial, bool doSlow, int kCopies>
__device__ __forceinline__ void precisePair(const PairTerms& u, const SlowTable& T,
                                            const NbkConst& c, const int lane, LaneSums& L) {
  const double s = fma(u.dz, u.dz, fma(u.dy, u.dy, u.dx * u.dx));
  double p = 0.0, dp = 0.0;
  if (doSlow && kCopies == kBeyond && s > T.sMax) {
    const double2 d = slowTermsDirect(c, s);
    p = d.x;
    dp = d.y;
  } else if (doSlow) {
    // row k = nearest integer to s/D: adding 1.5 * 2^52 rounds s/D (exact, D
    // a power of two) into the low word; k is clamped to the last row (any
    // bit pattern stays in the table) and w = s - k D
    const double magic = 6755399441055744.0;
    const double t = fma(s, T.invStep, magic);
    const unsigned k = min((unsigned)__double2loint(t), T.last);
    // the row number back from t (no conversion); where the clamp acts, s is no
    // pair's and only the row has to exist
    const double wq = fma(-T.step, t - magic, s);
    double cf[kSlowTableDeg1];
#pragma unroll
    for (int n = 0; n < kSlowTableDeg1; n += 2) {
      const double2 v = slowPair<kCopies>(T, k, n / 2, lane);
      cf[n] = v.x;
      cf[n + 1] = v.y;
    }
    // Horner for p(w) and p'(w) together
    p = cf[kSlowTableDeg];
    dp = 0.0;
#pragma unroll
    for (int n = kSlowTableDeg - 1; n >= 0; --n) {
      dp = fma(dp, wq, p);
      p = fma(p, wq, cf[n]);
    }
  }
  if (doEnergy) {
    // y0 (rsqrt.approx.ftz.f64) has relative error below 2^-20; after one
    // Newton step, below 2^-39
    const double y0 = rsqrtApprox64(s);
    const double hs = 0.5 * s;
    const double y = fma(y0, fma(-hs * y0, y0, 0.5), y0);
    L.eE = fma(u.qq, y - fma(c.hBd, s, c.hAd), L.eE);
    if (doSlow) L.eS = fma(u.qq, p, L.eS);
  }
  if (doVirial && doSlow) {
    const double g = (u.qq + u.qq) * dp;  // (dE/dr)/r
    const double gx = -g * u.dx, gy = -g * u.dy, gz = -g * u.dz;
    L.w0 = fma(gx, u.dx, L.w0);
    L.w1 = fma(gx, u.dy, L.w1);
    L.w2 = fma(gx, u.dz, L.w2);
    L.w3 = fma(gy, u.dy, L.w3);
    L.w4 = fma(gy, u.dz, L.w4);
    L.w5 = fma(gz, u.dz, L.w5);
  }
}

// The FP64 pair terms of the pair of owner lane l and bit t (block order) from
// the warp's atoms in shared memory; qq = 0 (exact zeros) when the lane has no pair left and
// repeats its last one, a real interacting pair (so its distance is not 0).
__device__ __forceinline__ void pairTerms(const Atoms64& A, const int l, const int t,
                                          const bool valid, PairTerms& u) {
  const int i = ((t & 3) << 3) | (l & 7);
  const double2 ia = A.ixy[i], ib = A.izq[i];
  // j = ((t & 28) ^ (l & 4)) | (l >> 3), at its place in the turned row
  const float4 jb = A.j[(l & 24) | ((t >> 2) ^ ((l >> 2) & 1))];
  u.dx = (double)jb.x - ia.x;
  u.dy = (double)jb.y - ia.y;
  u.dz = (double)jb.z - ib.x;
  u.qq = valid ? ib.y * (double)jb.w : 0.0;
}

// w without its r lowest set bits (r < popc(w)): the bits from the position p
// of its (r + 1)-th set bit up, p being the largest position with at most r
// set bits below it (a binary search over popc of w's low bits; p + step
// stays below 32).
__device__ __forceinline__ unsigned dropLowBits(const unsigned w, const int r) {
  int p = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1)
    if (__popc(w & ((1u << (p + step)) - 1u)) <= r) p += step;
  return w & (0xffffffffu << p);
}

// One lane's walk over the tile's interacting pairs in lane-major order: the
// owner lane i whose live bits w are not taken yet, and the last pair taken
// (pi, pt).
struct PairWalk {
  int i, pi, pt;
  unsigned w;
};

// Takes the lane's next pair when valid (the lowest bit of w; w is not 0 while
// the lane has pairs left), then, once w is spent, moves on to the next lane
// with live bits (nonEmpty: the lanes whose live word is not 0). Every lane
// runs the shuffle; the source lane is in [0, 31].
__device__ __forceinline__ void walkNext(PairWalk& s, const bool valid, const unsigned live,
                                         const unsigned nonEmpty) {
  if (valid) {
    s.pt = __ffs(s.w) - 1;
    s.pi = s.i;
    s.w &= s.w - 1;
  }
  const int inext = __ffs(nonEmpty & (0xfffffffeu << s.i)) - 1;  // -1: none after i
  const unsigned wn = __shfl_sync(0xffffffffu, live, inext & 31);
  if (valid && s.w == 0u && inext >= 0) {
    s.i = inext;
    s.w = wn;
  }
}

// The precise pass of one tile. live (per lane): bit t set when the pair that
// lane and bit stand for in block order is an interacting pair (mask bit set
// and FP32 r^2 below the cutoff, the classification the FP32 math used). The
// tile's `total` interacting pairs, in lane-major order (by lane, then t), are
// split into 32 contiguous ranges of m = ceil(total / 32): lane k takes pairs
// k m .. k m + m - 1 (the last lanes fewer or none). A lane finds the owner
// of its first pair by a binary search over the lanes' inclusive counts
// (shuffles), skips the owner's lower bits, and then walks the live words bit
// by bit (walkNext), two pairs per iteration (independent dependency
// chains). No queue is written. Each lane's sums take its pairs in a fixed
// order, so they depend only on the tile's live words. A lane without pairs
// repeats the tile's first pair with qq = 0.
template <bool doEnergy, bool doVirial, bool doSlow, int kCopies>
__device__ __forceinline__ void precisePass(const unsigned live, const int lane, const Atoms64& A,
                                            const SlowTable& T, const NbkConst& c, LaneSums& L,
                                            int& npair) {
  const int n = __popc(live);
  if (doEnergy) npair += n;
  int incl = n;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, kWarp - 1);
  if (total == 0) return;  // warp-uniform
  const int m = (total + kWarp - 1) / kWarp;
  const unsigned nonEmpty = __ballot_sync(0xffffffffu, live != 0u);
  int e0 = lane * m;
  const int cnt = min(m, max(0, total - e0));
  if (e0 >= total) e0 = 0;
  // owner of pair e0: the number of lanes whose inclusive count is <= e0
  int owner = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const int v = __shfl_sync(0xffffffffu, incl, owner + step - 1);
    if (v <= e0) owner += step;
  }
  const int ownerExcl = __shfl_sync(0xffffffffu, incl - n, owner);
  const unsigned ownerLive = __shfl_sync(0xffffffffu, live, owner);
  PairWalk s;
  s.i = owner;
  s.w = dropLowBits(ownerLive, e0 - ownerExcl);
  s.pi = owner;
  s.pt = __ffs(s.w) - 1;
  __syncwarp();  // the i rows and this j tile, written by the lanes, are visible
  int k = 0;
  for (; k + 1 < m; k += 2) {  // warp-uniform
    PairTerms u[2];
    walkNext(s, k < cnt, live, nonEmpty);
    pairTerms(A, s.pi, s.pt, k < cnt, u[0]);
    walkNext(s, k + 1 < cnt, live, nonEmpty);
    pairTerms(A, s.pi, s.pt, k + 1 < cnt, u[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) precisePair<doEnergy, doVirial, doSlow, kCopies>(u[h], T, c, lane, L);
  }
  if (k < m) {  // warp-uniform
    PairTerms u;
    walkNext(s, k < cnt, live, nonEmpty);
    pairTerms(A, s.pi, s.pt, k < cnt, u);
    precisePair<doEnergy, doVirial, doSlow, kCopies>(u, T, c, lane, L);
  }
  __syncwarp();  // the j rows are consumed before they are written again
}

// End of a tile group: the lanes' sums are reduced per quantity by a fixed
// butterfly that halves the quantities a lane holds at each step (lanes l and
// l ^ 16 exchange four of their eight, then l ^ 8 two, l ^ 4 one; two more
// steps add within groups of four lanes), so that lane 4q holds the warp's
// total of quantity q; lane q < kNumQ then adds quantity q, in fixed point,
// to accQ, and the sums restart at zero. No shared memory: a transposition
// through it costs more than these 20 shuffles (its reads conflict 16-way).
__device__ __forceinline__ void reduceGroup(const int lane, LaneSums& L, long long& accQ) {
  double v[kNumQ] = {L.eE, L.eS, L.w0, L.w1, L.w2, L.w3, L.w4, L.w5};
  static_assert(kQElec == 0 && kQSlow == 1 && kQVir == 2 && kNumQ == 8, "quantity order");
  // lanes with bit 4 set keep quantities 4..7, the others 0..3
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double send = b4 ? v[k] : v[k + 4];
    const double keep = b4 ? v[k + 4] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double send = b3 ? v[k] : v[k + 2];
    const double keep = b3 ? v[k + 2] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  {
    const double send = b2 ? v[0] : v[1];
    const double keep = b2 ? v[1] : v[0];
    v[0] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  // lane l now holds quantity (l >> 2) summed over the lanes l' with
  // l' & 3 == l & 3; complete the sums within each group of four lanes
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  const double tot = __shfl_sync(0xffffffffu, v[0], 4 * (lane & 7));
  if (lane < kNumQ) accQ += toFixedEnergy(tot);
  L = LaneSums{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
}

// Block order: a 32 x 32 tile is 16 blocks of 8 i atoms by 8 j atoms. Lane
// l = 8 lj + li (li = l & 7, lj = l >> 3) takes, of block (I, J), the pairs of
// i = 8 I + li with j = 8 J + lj and j + 4 (elements x and y of the packed
// math; the other way round in the lanes with bit 2 set), so a block is one pass of the packed loop with every lane
// busy, its j atoms' sums stay in registers over the blocks of a row (the same
// J) and its i atoms' over a group of tiles: the loop has no shuffle. The mask
// words hold bit 8 J + 4 e + I of element e (blockOrder; TileExcl rows are put into this
// order by the refinement and back by the export).
//
// What bounds it: issue slots and the FMA pipe, as before, but on far fewer
// passes. Blocks of 8 x 8 atoms are compact (the atom order bisects down to 8),
// so a pass holds 28.5 interacting pairs of 64 (20k mixed system; 255,843
// passes) where the diagonals j = (l + t) & 31 of the tile held 17.4
// (419,488), and the diagonals' rotation of the j sums (12 shuffles a pass)
// becomes one reduction per row of blocks. Steady steps of the 92,224-atom
// mixed system, by diagonals, when the blocks came, and now (the slow table, i rows
// kept once, overlapped launches): fast + slow forces 392, 290, 267 us, fast forces
// 279, 198, 184, with energies and virials 601, 507, 483 (of which the precise
// kernel is 197); 210 M warp instructions for fast + slow forces when the blocks
// came, 195 M now.
//
// MINB: CTAs per SM the register budget is cut for (4, 5 or 6 -> 128, 96 or
// 80 registers); a.splitLog2: each list's j tiles are shared by 2^splitLog2
// work items (warps), contiguous parts of equal tile count. Both are launch
// choices of the autotuner; results do not depend on them (fixed-point sums
// per tile group).
template <bool doEnergy, bool doVirial, bool doSlow, bool kTable, bool doBatch, int MINB>
__global__ void __launch_bounds__(kForceThreads, MINB)
    forceKernel(const __grid_constant__ ForceArgs a) {
  // the live words feed the precise kernel, which runs on energy evaluations
  // and on virial evaluations with slow forces (it forms the slow virial)
  constexpr bool kLive = doEnergy || (doVirial && doSlow);
  constexpr int kNC = doSlow ? 6 : 3;  // force components: fast x y z, slow x y z
  // the slow force table (kTable; a.tabCopies interleaved copies), then the LJ
  // table [ljDim*ljDim] as (A, -B) (single system)
  extern __shared__ __align__(16) float4 s_tab[];
  // the list's i atoms, shifted: (-x, -y, -z, q), and the byte offset of the
  // type's LJ row. A 16-byte load takes four passes of the shared-memory pipe
  // whatever the lanes share, so the coordinates are not kept twice for the
  // packed instructions.
  __shared__ float4 s_i[kForceWarps][kWarp];
  __shared__ int s_it[kForceWarps][kWarp];
  // the j tile by pairs (j, j + 4) of a row's lanes: entry 4 J + lj holds
  // (x, x', y, y'), (z, z', q, q') and (type, type') as byte offsets in an LJ
  // row; the second copy, for the lanes with bit 2 set, holds j + 4 first
  __shared__ float4 s_j[kForceWarps][2][2][16];
  __shared__ float2 s_jt[kForceWarps][2][16];
  // each lane's i force of the current list part in fixed point, folded in
  // at the end of every tile group, so that the sums do not depend on how a
  // list's tiles are split among warps
  __shared__ long long s_fi[kForceWarps][kNC][kWarp];
  // each lane's LJ energy of the list part in fixed point (s_ev) and of the
  // current tile group in FP32 (s_evg), and the warp's fixed-point LJ total
  // (s_evw, lane 0), kept in shared memory rather than in registers the pair
  // loop needs
  __shared__ long long s_ev[kForceWarps][kWarp];
  __shared__ float s_evg[kForceWarps][kWarp];
  __shared__ long long s_evw[kForceWarps];

  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int li = lane & 7, lj = lane >> 3;
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
  const unsigned adrI = sharedAddr(&s_i[wib][li]), adrIT = sharedAddr(&s_it[wib][li]),
                 adrJ = sharedAddr(&s_j[wib][b2][0][lj]),
                 adrT = sharedAddr(&s_jt[wib][b2][lj]);
  const NbkConst& c = a.c;
  const int dim = c.ljDim;
  const int tabEntries = kTable ? a.pk.tabRows * a.tabCopies : 0;
  const unsigned adrLJ = sharedAddr(s_tab + tabEntries);
  ForceTable T{};
  if (kTable) {
    for (int k = threadIdx.x; k < tabEntries; k += blockDim.x)
      s_tab[k] = a.pk.tab[(unsigned)k / (unsigned)a.tabCopies];
    T.stride = 16u * a.tabCopies;
    T.base = sharedAddr(s_tab + (lane & (a.tabCopies - 1))) - kRowMagicBits * T.stride;
    T.step = a.pk.tabStep;
    T.invStep = a.pk.tabInvStep;
    T.sMax = a.pk.tabStep * (float)(a.pk.tabRows - 1);
  }
  if (!doBatch) {
    float2* s_lj = reinterpret_cast<float2*>(s_tab + tabEntries);
    for (int k = threadIdx.x; k < dim * dim; k += blockDim.x)
      s_lj[k] = make_float2(a.ljTable[k].x, -a.ljTable[k].y);
  }
  if (kTable || !doBatch) __syncthreads();
  // the tables above belong to the handle; what follows needs the cleared
  // buffers and the lists
  waitForPredecessor();
  admitSuccessor();

  const int numLists = a.numListsDev ? *a.numListsDev : a.numListsHost;

  long long accVdw = 0;  // lane 0: LJ energy to flush (batched replica change)
#pragma unroll
  for (int q = 0; q < kNC; ++q) s_fi[wib][q][lane] = 0;
  s_ev[wib][lane] = 0;
  s_evg[wib][lane] = 0.f;
  if (lane == 0) s_evw[wib] = 0;
  int curRep = 0;  // replica whose accumulators the warp is holding

  // lists are handed out one at a time from a global counter, so warps that
  // draw short lists keep working instead of idling at the end
  const int split = 1 << a.splitLog2;
  for (;;) {
    const int W = drawItem(a.workCounter, lane);
    if (W >= numLists * split) break;
    const int part = W & (split - 1);
    const nbk_tile_list tl = a.lists[W >> a.splitLog2];
    int jtFirst, jtLast;
    listPart(a, tl, part, jtFirst, jtLast);
    if (jtLast < jtFirst) continue;  // this part has no tiles (warp-uniform)
    float3 la = a.lata, lb = a.latb, lc = a.latc;
    const char* ljRow = nullptr;  // batched: this replica's LJ table (global)
    if (doBatch) {
      const int rep = __ldg(&a.compRep[tl.icompute]);
      if (rep != curRep) {
        if (lane == 0) {
          accVdw = s_evw[wib];
          s_evw[wib] = 0;
        }
        flushVdw<doEnergy>(a.acc + (size_t)curRep * kAccCount, lane, accVdw);
        curRep = rep;
      }
      la = a.repLat[3 * rep];
      lb = a.repLat[3 * rep + 1];
      lc = a.repLat[3 * rep + 2];
      ljRow = reinterpret_cast<const char*>(a.repLJ + (size_t)rep * dim * dim);
    }
    const float3 off = make_float3(tl.offsetXYZ.x, tl.offsetXYZ.y, tl.offsetXYZ.z);
    const float3 sh = shiftOf(off, la, lb, lc);
    const bool zeroShift = !(dist2(sh.x, sh.y, sh.z) > 0.0f);

    const int iatom = tl.iatomStart + lane;
    {
      const float4 xi = a.xyzq[iatom];
      s_i[wib][lane] = make_float4(-__fadd_rn(xi.x, sh.x), -__fadd_rn(xi.y, sh.y),
                                   -__fadd_rn(xi.z, sh.z), xi.w);
      s_it[wib][lane] = a.vdwTypes[iatom] * dim * 8;
    }

    // this tile group's partial sums of the lane's four i atoms (8 I + li)
    float fi[4][kNC];
#pragma unroll
    for (int I = 0; I < 4; ++I)
#pragma unroll
      for (int q = 0; q < kNC; ++q) fi[I][q] = 0.f;

    // the next tile's mask word and j atom are loaded while the current tile
    // is computed; the j-tile starts come 32 at a time (lane t holds tile
    // jtFirst + 32 b + t) and are handed out by a shuffle
    int jsBlock = 0;
    unsigned maskNext = 0;
    float4 xjNext = make_float4(0.f, 0.f, 0.f, 0.f);
    int tyNext = 0;
    for (int jt = jtFirst; jt <= jtLast; ++jt) {
      const int tb = (jt - jtFirst) & 31;
      if (tb == 0) {
        const int jtl = jt + lane;
        jsBlock = jtl <= jtLast ? a.tileJatomStart[jtl] : 0;
        const int js0 = __shfl_sync(0xffffffffu, jsBlock, 0);
        maskNext = a.tileExcls[jt].excl[lane];
        xjNext = a.xyzq[js0 + lane];
        tyNext = a.vdwTypes[js0 + lane];
      }
      const int jstart = __shfl_sync(0xffffffffu, jsBlock, tb);
      const unsigned mask = maskNext;
      {
        // atom j = lane of the tile: entry 4 (j >> 3) + (j & 3), element (j >> 2) & 1
        const int m = (lane >> 3) * 4 + (lane & 3), e = (lane >> 2) & 1;
#pragma unroll
        for (int copy = 0; copy < 2; ++copy) {
          const int ec = copy ? 1 - e : e;
          float* pa = reinterpret_cast<float*>(&s_j[wib][copy][0][m]) + ec;
          float* pb = reinterpret_cast<float*>(&s_j[wib][copy][1][m]) + ec;
          pa[0] = xjNext.x;
          pa[2] = xjNext.y;
          pb[0] = xjNext.z;
          pb[2] = xjNext.w;
          reinterpret_cast<int*>(&s_jt[wib][copy][m])[ec] = tyNext * 8;
        }
      }
      if (jt < jtLast && tb < 31) {
        const int js1 = __shfl_sync(0xffffffffu, jsBlock, tb + 1);
        maskNext = a.tileExcls[jt + 1].excl[lane];
        xjNext = a.xyzq[js1 + lane];
        tyNext = a.vdwTypes[js1 + lane];
      }
      const unsigned stepMask = __reduce_or_sync(0xffffffffu, mask);
      __syncwarp();
      unsigned live = 0;  // interacting pairs of this lane, block order
      float2 eV2 = f2(0.f);
      // live rows, in order; the j sums of a row wait for a partner row (and,
      // without slow forces, a pair of rows for a partner pair), so that every
      // lane ends up with one j atom of its own
      float held[3], held2[3];
      int Jheld = 0, Jheld2 = 0, rows = 0;
      unsigned todo = stepMask;
#pragma unroll 1
      while (todo) {  // warp-uniform
        const int J8 = (__ffs(todo) - 1) & 24;  // 8 J
        const unsigned rowAny = (todo >> J8) & 0xffu;
        todo &= ~(0xffu << J8);
        const unsigned mrow = mask >> J8;
        const float4 ja = ldShared4(adrJ + J8 * 8), jb = ldShared4(adrJ + 256 + J8 * 8);
        const float2 tj = ldShared2(adrT + J8 * 4);
        const float2 X = make_float2(ja.x, ja.y), Y = make_float2(ja.z, ja.w),
                     Z = make_float2(jb.x, jb.y);
        float2 fj[kNC];
#pragma unroll
        for (int q = 0; q < kNC; ++q) fj[q] = f2(0.f);
        unsigned liveRow = 0;
#pragma unroll
        for (int I = 0; I < 4; ++I) {
          if (!(rowAny & (0x11u << I))) continue;  // warp-uniform
          const float4 xi = ldShared4(adrI + 128 * I);
          const float2 DX = make_float2(X.x + xi.x, X.y + xi.x),
                       DY = make_float2(Y.x + xi.y, Y.y + xi.y),
                       DZ = make_float2(Z.x + xi.z, Z.y + xi.z);
          const float2 R2 = fma2(DZ, DZ, fma2(DX, DX, mul2(DY, DY)));  // dist2's order
          const bool aA = (mrow & (1u << I)) && (R2.x < c.cutoff2);
          const bool aB = (mrow & (0x10u << I)) && (R2.y < c.cutoff2);
          if (!__any_sync(0xffffffffu, aA || aB)) continue;
          if (kLive) liveRow |= (aA ? 1u << I : 0u) | (aB ? 0x10u << I : 0u);
          const int ti = ldShared1(adrIT + 32 * I);
          const int tA = ti + __float_as_int(tj.x), tB = ti + __float_as_int(tj.y);
          const float2 abA = doBatch ? __ldg((const float2*)(ljRow + tA)) : ldShared2(adrLJ + tA);
          const float2 abB = doBatch ? __ldg((const float2*)(ljRow + tB)) : ldShared2(adrLJ + tB);
          const float2 QQ = make_float2(xi.w * jb.z, xi.w * jb.w);
          float2 F, FS, E;
          pairForce2<doEnergy, doSlow, kTable>(R2, QQ, make_float2(abA.x, abB.x),
                                       make_float2(abA.y, abB.y), a.pk, T, F, FS, E);
          // an element that is no interacting pair may hold anything, NaN
          // included: it is replaced by an exact zero
          F = make_float2(aA ? F.x : 0.f, aB ? F.y : 0.f);
          if (doEnergy) eV2 = add2(eV2, make_float2(aA ? E.x : 0.f, aB ? E.y : 0.f));
          fi[I][0] = fmaf(DX.y, F.y, fmaf(DX.x, F.x, fi[I][0]));
          fi[I][1] = fmaf(DY.y, F.y, fmaf(DY.x, F.x, fi[I][1]));
          fi[I][2] = fmaf(DZ.y, F.y, fmaf(DZ.x, F.x, fi[I][2]));
          fj[0] = fma2(DX, F, fj[0]);
          fj[1] = fma2(DY, F, fj[1]);
          fj[2] = fma2(DZ, F, fj[2]);
          if constexpr (doSlow) {
            FS = make_float2(aA ? FS.x : 0.f, aB ? FS.y : 0.f);
            fi[I][3] = fmaf(DX.y, FS.y, fmaf(DX.x, FS.x, fi[I][3]));
            fi[I][4] = fmaf(DY.y, FS.y, fmaf(DY.x, FS.x, fi[I][4]));
            fi[I][5] = fmaf(DZ.y, FS.y, fmaf(DZ.x, FS.x, fi[I][5]));
            fj[3] = fma2(DX, FS, fj[3]);
            fj[4] = fma2(DY, FS, fj[4]);
            fj[5] = fma2(DZ, FS, fj[5]);
          }
        }
        if (kLive) live |= liveRow << J8;
        // the row's j sums over the eight i lanes: lanes l and l ^ 4 hold the
        // two j atoms in turned order, so each keeps its element x; then bit 1
        // tells the fast from the slow force
        float v[3], u[kNC];
#pragma unroll
        for (int q = 0; q < kNC; ++q) u[q] = fj[q].x + __shfl_xor_sync(0xffffffffu, fj[q].y, 4);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if constexpr (doSlow) v[q] = keepHalf(u[q], u[q + 3], b1, 2);
          else v[q] = u[q];
        }
        // the lane bits that are left tell rows apart: bit 0 the rows of a
        // pair (with slow forces), else bit 1 the rows of a pair and bit 0
        // the pairs. A last row without a partner is paired with zeros.
        int Jrow = J8;
        if (!(rows++ & 1)) {
#pragma unroll
          for (int q = 0; q < 3; ++q) held[q] = v[q];
          Jheld = Jrow;
          if (todo) continue;
#pragma unroll
          for (int q = 0; q < 3; ++q) v[q] = 0.f;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) v[q] = keepHalf(held[q], v[q], doSlow ? b0 : b1, doSlow ? 1 : 2);
        Jrow = (doSlow ? b0 : b1) ? Jrow : Jheld;
        if constexpr (!doSlow) {
          if (rows <= 2) {
#pragma unroll
            for (int q = 0; q < 3; ++q) held2[q] = v[q];
            Jheld2 = Jrow;
            if (todo) continue;
#pragma unroll
            for (int q = 0; q < 3; ++q) v[q] = 0.f;
          }
#pragma unroll
          for (int q = 0; q < 3; ++q) v[q] = keepHalf(held2[q], v[q], b0, 1);
          Jrow = b0 ? Jrow : Jheld2;
        }
        // the lane's j atom, and its force array; F_j = -sum
        if (v[0] != 0.f || v[1] != 0.f || v[2] != 0.f) {
          long long* f = a.force + (doSlow && b1 ? 3 * (size_t)a.stride : 0) + jstart + Jrow +
                         (lane & 4) + lj;
          atomicAddFixed(f, toFixedForce(-v[0]));
          atomicAddFixed(f + (size_t)a.stride, toFixedForce(-v[1]));
          atomicAddFixed(f + 2 * (size_t)a.stride, toFixedForce(-v[2]));
        }
      }
      if (doEnergy) s_evg[wib][lane] += (eV2.x + eV2.y) * (-1.0f / 6.0f);  // the terms are -6 E
      if (kLive) a.liveOut[(size_t)jt * kWarp + lane] = live;
      if (groupEnds(tl, jt, jtLast)) {
        // end of a tile group: its LJ energy and i forces into fixed point
        if (doEnergy) {
          s_ev[wib][lane] += toFixedEnergyF(s_evg[wib][lane]);
          s_evg[wib][lane] = 0.f;
        }
        // i sums over the four j lanes: bits 4 and 3 keep cluster I = lane >> 3,
        // so that every lane ends up with its own atom 8 I + li = lane
#pragma unroll
        for (int q = 0; q < kNC; ++q) {
          const float lo = keepHalf(fi[0][q], fi[2][q], b4, 16);
          const float hi = keepHalf(fi[1][q], fi[3][q], b4, 16);
          s_fi[wib][q][lane] += (long long)toFixedForce(keepHalf(lo, hi, b3, 8));
          fi[0][q] = fi[1][q] = fi[2][q] = fi[3][q] = 0.f;
        }
      }
      __syncwarp();
    }  // jt

    // i forces (fixed point)
    unsigned long long qx, qy, qz, sx = 0, sy = 0, sz = 0;
    qx = (unsigned long long)s_fi[wib][0][lane];
    qy = (unsigned long long)s_fi[wib][1][lane];
    qz = (unsigned long long)s_fi[wib][2][lane];
    s_fi[wib][0][lane] = s_fi[wib][1][lane] = s_fi[wib][2][lane] = 0;
    if (doSlow) {
      sx = (unsigned long long)s_fi[wib][3][lane];
      sy = (unsigned long long)s_fi[wib][4][lane];
      sz = (unsigned long long)s_fi[wib][5][lane];
      s_fi[wib][3][lane] = s_fi[wib][4][lane] = s_fi[wib][5][lane] = 0;
    }
    if (qx | qy | qz) {
      atomicAddFixed(&a.force[0 * (size_t)a.stride + iatom], qx);
      atomicAddFixed(&a.force[1 * (size_t)a.stride + iatom], qy);
      atomicAddFixed(&a.force[2 * (size_t)a.stride + iatom], qz);
    }
    if (doSlow && (sx | sy | sz)) {
      atomicAddFixed(&a.force[3 * (size_t)a.stride + iatom], sx);
      atomicAddFixed(&a.force[4 * (size_t)a.stride + iatom], sy);
      atomicAddFixed(&a.force[5 * (size_t)a.stride + iatom], sz);
    }
    if (doVirial && !zeroShift) {
      // the lattice-shift part of the fast virial, (sum_i F_i) (x) shift, is
      // formed per compute by the finalize kernel from these exact integer sums
      const long long Fx = warpSumLL((long long)qx), Fy = warpSumLL((long long)qy),
                      Fz = warpSumLL((long long)qz);
      long long* cf = a.compF + 6 * (size_t)tl.icompute;
      if (lane == 0) {
        if (Fx) atomicAddFixed(&cf[0], (unsigned long long)Fx);
        if (Fy) atomicAddFixed(&cf[1], (unsigned long long)Fy);
        if (Fz) atomicAddFixed(&cf[2], (unsigned long long)Fz);
      }
    }
    if (doEnergy) {
      const long long sV = warpSumLL(s_ev[wib][lane]);
      s_ev[wib][lane] = 0;
      if (lane == 0) s_evw[wib] += sV;
    }
  }  // lists

  // per-warp flush of the LJ energy (no block barrier, so a warp that runs
  // out of lists retires at once)
  if (lane == 0) accVdw = s_evw[wib];
  flushVdw<doEnergy>(a.acc + (size_t)curRep * kAccCount, lane, accVdw);
}

// The precise kernel: one warp per refined tile list (handed out by a global
// counter in the force kernel's order, longest first). Per list the i atoms,
// shifted in FP64 by the shift formed in FP64 from the FP32 offsets and
// lattice (the exact lattice translation, without the FP32 rounding of the
// force kernel's shift), go to the warp's FP64 rows; per tile with interacting
// pairs the j atoms and the precise pass; per group of kFoldTiles tiles
// (counted from the list start, as the force kernel's) the lanes' sums go into
// fixed point. Results do not depend on the order in which lists run.
constexpr int kPreciseWarps = 8;
constexpr int kPreciseThreads = kPreciseWarps * kWarp;
constexpr int kPreciseMinBlocks = 3;

template <bool doEnergy, bool doVirial, bool doSlow, bool doBatch, int kCopies>
__global__ void __launch_bounds__(kPreciseThreads, kPreciseMinBlocks)
    preciseKernel(const __grid_constant__ ForceArgs a) {
  __shared__ Atoms64 s_atoms[kPreciseWarps];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  Atoms64& A = s_atoms[wib];
  SlowTable T;
  T.last = (unsigned)(a.slowTableRows - 1);
  T.step = a.slowStep;
  T.invStep = a.slowInvStep;
  T.gl = a.slowTable;
  T.sMax = a.slowStep * (double)(a.slowTableRows - 1);
  if (doSlow && kCopies > 0) {
    constexpr int P = kSlowTableDeg1 / 2;
    for (int k = threadIdx.x; k < P * a.slowTableRows * kCopies; k += blockDim.x) {
      const int pair = k / (kCopies > 0 ? kCopies : 1);  // row * P + n
      s_slowTab[k] = a.slowTable[(size_t)(pair / P) * (kSlowTableRow / 2) + pair % P];
    }
    __syncthreads();
  }
  waitForPredecessor();
  const int numLists = a.numListsDev ? *a.numListsDev : a.numListsHost;
  long long accQ = 0;  // lane q < kNumQ: quantity q
  int npair = 0;       // interacting pairs counted by this lane (energy evaluations)
  LaneSums lsum{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int curRep = 0;
  const int split = 1 << a.splitLog2;
  for (;;) {
    const int W = drawItem(a.workCounter, lane);
    if (W >= numLists * split) break;
    const int part = W & (split - 1);
    const nbk_tile_list tl = a.lists[W >> a.splitLog2];
    int jtFirst, jtLast;
    listPart(a, tl, part, jtFirst, jtLast);
    if (jtLast < jtFirst) continue;  // this part has no tiles (warp-uniform)
    float3 la = a.lata, lb = a.latb, lc = a.latc;
    if (doBatch) {
      const int rep = __ldg(&a.compRep[tl.icompute]);
      if (rep != curRep) {
        flushPrecise<doEnergy>(a.acc + (size_t)curRep * kAccCount, lane, accQ, npair);
        curRep = rep;
      }
      la = a.repLat[3 * rep];
      lb = a.repLat[3 * rep + 1];
      lc = a.repLat[3 * rep + 2];
    }
    {
      const float3 off = make_float3(tl.offsetXYZ.x, tl.offsetXYZ.y, tl.offsetXYZ.z);
      const float4 xi = a.xyzq[tl.iatomStart + lane];
      A.ixy[lane] = make_double2(
          (double)xi.x + ((double)off.x * la.x + (double)off.y * lb.x + (double)off.z * lc.x),
          (double)xi.y + ((double)off.x * la.y + (double)off.y * lb.y + (double)off.z * lc.y));
      A.izq[lane] = make_double2(
          (double)xi.z + ((double)off.x * la.z + (double)off.y * lb.z + (double)off.z * lc.z),
          (double)xi.w);
    }
    // the next tile's live word and j atom are loaded while the current tile
    // is processed; the j-tile starts come 32 at a time (lane t holds tile
    // jt0 + t) and are handed out by a shuffle
    int jsBlock = 0;
    unsigned liveNext = 0;
    float4 xjNext = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int jt = jtFirst; jt <= jtLast; ++jt) {
      const int t = (jt - jtFirst) & 31;
      if (t == 0) {
        const int jtl = jt + lane;
        jsBlock = jtl <= jtLast ? a.tileJatomStart[jtl] : 0;
        liveNext = a.liveOut[(size_t)jt * kWarp + lane];
        xjNext = a.xyzq[__shfl_sync(0xffffffffu, jsBlock, 0) + lane];
      }
      const unsigned live = liveNext;
      const float4 xj = xjNext;
      if (jt < jtLast && t < 31) {
        liveNext = a.liveOut[(size_t)(jt + 1) * kWarp + lane];
        xjNext = a.xyzq[__shfl_sync(0xffffffffu, jsBlock, t + 1) + lane];
      }
      if (__any_sync(0xffffffffu, live != 0u)) {
        // the i rows and this j tile are visible after the pass's first __syncwarp
        A.j[8 * (lane & 3) + (lane >> 2)] = xj;
        precisePass<doEnergy, doVirial, doSlow, kCopies>(live, lane, A, T, a.c,
                                                         lsum, npair);
      }
      if (groupEnds(tl, jt, jtLast))
        reduceGroup(lane, lsum, accQ);
    }
  }
  flushPrecise<doEnergy>(a.acc + (size_t)curRep * kAccCount, lane, accQ, npair);
}

template <typename K>
static cudaError_t launchPersistent(K kernel, KernelLimits& limits, int threads, size_t shmem,
                                    int numSM, cudaStream_t st, const ForceArgs& a) {
  int blocks = 0;
  const cudaError_t e = limits.blocksPerSM(kernel, threads, shmem, &blocks);
  if (e != cudaSuccess) return e;
  return launchOverlapped(kernel, numSM * blocks, threads, shmem, st, a);
}

template <bool E, bool V, bool S, bool B, int MINB>
static cudaError_t launchT(const ForceArgs& a, int numSM, cudaStream_t st) {
  const size_t lj = B ? 0 : sizeof(float2) * (size_t)a.c.ljDim * a.c.ljDim;
  if constexpr (S) {
    if (a.pk.tabRows > 0 && !a.beyondTables) {  // the erfc form has no end
      // copies of the table, up to the 8 that keep quarter warps free of bank
      // conflicts, that cost no block: from 62 LJ types on the LJ table leaves no
      // room for 8 beside four blocks, and a block counts for more (94 rows, fast
      // and slow forces of 92,224 atoms: 70 types 287 -> 262 us, 80 types 371 ->
      // 306, 110 types 622 -> 377)
      static KernelLimits limits;
      ForceArgs t = a;
      const size_t one = sizeof(float4) * (size_t)a.pk.tabRows;
      const auto kernel = forceKernel<E, V, S, true, B, MINB>;
      int blocks = 0;
      const cudaError_t e = limits.tableCopies(kernel, kForceThreads, lj, one, kForceTableBytes,
                                               &t.tabCopies, &blocks);
      if (e != cudaSuccess) return e;
      return launchOverlapped(kernel, numSM * blocks, kForceThreads, one * t.tabCopies + lj, st, t);
    }
  }
  static KernelLimits limits;
  return launchPersistent(forceKernel<E, V, S, false, B, MINB>, limits, kForceThreads, lj, numSM,
                          st, a);
}

// A block less per SM costs more than the table gains over the erfc form: fast and
// slow forces of 92,224 atoms with a table of 739 rows, 294 against 267 us with 70
// LJ types (three blocks, four), 638 against 381 with 110 (one, two). One rule for
// every flag combination and launch shape, and for replicas (whose LJ tables stay
// in global memory), so that none of them changes a bit: by the shared memory of
// the instance without energies at the default four blocks.
cudaError_t forceTableFits(int ljDim, int rows, bool* fits) {
  int dev = 0, perSM = 0, reserved = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&perSM, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  cudaFuncAttributes at{};
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, forceKernel<false, false, true, true, false, 4>);
  if (e != cudaSuccess) return e;
  const size_t rest = at.sharedSizeBytes + (size_t)reserved + sizeof(float2) * (size_t)ljDim * ljDim;
  auto blocks = [&](size_t bytes) { return std::min<size_t>((size_t)perSM / bytes, 4); };
  *fits = blocks(rest + sizeof(float4) * (size_t)rows) == blocks(rest);
  return cudaSuccess;
}

template <bool E, bool V, bool S, bool B>
static cudaError_t launchShape(const ForceArgs& a, int minBlocks, int numSM, cudaStream_t st) {
  switch (minBlocks) {
    case 4: return launchT<E, V, S, B, 4>(a, numSM, st);
    case 5: return launchT<E, V, S, B, 5>(a, numSM, st);
    case 6: return launchT<E, V, S, B, 6>(a, numSM, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launchForce(const ForceArgs& a, unsigned flags, int minBlocks, int numSM,
                        cudaStream_t st) {
  const bool B = a.compRep != nullptr;
  const int idx = (B ? 8 : 0) | ((flags & NBK_ENERGY) ? 4 : 0) | ((flags & NBK_VIRIAL) ? 2 : 0) |
                  ((flags & NBK_SLOW) ? 1 : 0);
  switch (idx) {
#define NBK_CASE(i, e, v, s, b) \
  case i:                       \
    return launchShape<e, v, s, b>(a, minBlocks, numSM, st);
    NBK_CASE(0, false, false, false, false)
    NBK_CASE(1, false, false, true, false)
    NBK_CASE(2, false, true, false, false)
    NBK_CASE(3, false, true, true, false)
    NBK_CASE(4, true, false, false, false)
    NBK_CASE(5, true, false, true, false)
    NBK_CASE(6, true, true, false, false)
    NBK_CASE(7, true, true, true, false)
    NBK_CASE(8, false, false, false, true)
    NBK_CASE(9, false, false, true, true)
    NBK_CASE(10, false, true, false, true)
    NBK_CASE(11, false, true, true, true)
    NBK_CASE(12, true, false, false, true)
    NBK_CASE(13, true, false, true, true)
    NBK_CASE(14, true, true, false, true)
    NBK_CASE(15, true, true, true, true)
#undef NBK_CASE
  }
  return cudaErrorInvalidValue;
}

bool needsPrecise(unsigned flags) {
  return (flags & NBK_ENERGY) || ((flags & NBK_VIRIAL) && (flags & NBK_SLOW));
}

template <bool E, bool V, bool S, bool B, int C>
static cudaError_t launchPC(const ForceArgs& a, int numSM, cudaStream_t st) {
  static KernelLimits limits;
  const size_t shmem = (S && C > 0) ? sizeof(double) * kSlowTableDeg1 * (size_t)a.slowTableRows * C
                                    : 0;
  return launchPersistent(preciseKernel<E, V, S, B, C>, limits, kPreciseThreads, shmem, numSM, st,
                          a);
}

// The table in shared memory, in as many interleaved copies of 8, 4 or 1 as fit in
// 40 KB (106, 213, 853 rows), else in global memory; beyond its reach the
// instance that can go on from there. Global memory is the last choice because
// what is left of the L1 cache for it follows the force kernel's shared memory:
// while other kernels keep the SM busy the division stays. Energies, virials and
// slow forces of 92,224 atoms with 739 rows: 528 us with 34 LJ types and 603 with
// 61, which fill the SM's shared memory; with one copy here 519 and 525 (136
// rows, four copies: 356 and 365 -> 343 and 347).
template <bool E, bool V, bool S, bool B>
static cudaError_t launchP(const ForceArgs& a, int numSM, cudaStream_t st) {
  if constexpr (!S) {
    return launchPC<E, V, S, B, 0>(a, numSM, st);
  } else {
    if (a.beyondTables) return launchPC<E, V, S, B, kBeyond>(a, numSM, st);
    const size_t one = sizeof(double) * kSlowTableDeg1 * (size_t)a.slowTableRows, most = 40 * 1024;
    if (8 * one <= most) return launchPC<E, V, S, B, 8>(a, numSM, st);
    if (4 * one <= most) return launchPC<E, V, S, B, 4>(a, numSM, st);
    if (one <= most) return launchPC<E, V, S, B, 1>(a, numSM, st);
    return launchPC<E, V, S, B, 0>(a, numSM, st);
  }
}

cudaError_t launchPrecise(const ForceArgs& a, unsigned flags, int numSM, cudaStream_t st) {
  if (!needsPrecise(flags)) return cudaSuccess;
  const bool B = a.compRep != nullptr;
  const int idx = (B ? 8 : 0) | ((flags & NBK_ENERGY) ? 4 : 0) | ((flags & NBK_VIRIAL) ? 2 : 0) |
                  ((flags & NBK_SLOW) ? 1 : 0);
  switch (idx) {
#define NBK_CASE(i, e, v, s, b) \
  case i:                       \
    return launchP<e, v, s, b>(a, numSM, st);
    NBK_CASE(3, false, true, true, false)
    NBK_CASE(4, true, false, false, false)
    NBK_CASE(5, true, false, true, false)
    NBK_CASE(6, true, true, false, false)
    NBK_CASE(7, true, true, true, false)
    NBK_CASE(11, false, true, true, true)
    NBK_CASE(12, true, false, false, true)
    NBK_CASE(13, true, false, true, true)
    NBK_CASE(14, true, true, false, true)
    NBK_CASE(15, true, true, true, true)
#undef NBK_CASE
  }
  return cudaErrorInvalidValue;
}

}  // namespace nbk
