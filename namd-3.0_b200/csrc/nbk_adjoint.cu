// Adjoint of the nonbonded evaluation: for cotangents wF, wS on the fast and
// slow forces and cV, cE, cS on the three energies, the gradient of
//   L = sum_i wF_i . F_i + sum_i wS_i . Fslow_i + cV E_vdw + cE E_elec + cS E_slow
// with respect to the positions (a Hessian-vector product), the scaled charges
// and the scaled LJ table entries. Pair terms are recomputed from the refined
// tile lists; nothing from the forward pass is stored.
//
// Per pair, with s = r^2, d = x_j - x_i, uF = wF_i - wF_j, pF = uF . d (same
// for S), and g = (dE/dr)/r of each term (2 dE/ds = g):
//   dL/dd = g uF + gs uS + d [2 (pF g' + pS gs') + cV g_lj + cE qq g_f + cS qq g_s]
//   dL/dx_j = dL/dd, dL/dx_i = -dL/dd
//   dL/dqq = pF g_f + pS g_s + cE phi_f + cS phi_s
//   dL/dA = pF gA + cV EA, dL/dB = pF gB + cV EB   (LJ is linear in A and B)
// where ' = d/ds. The slow term comes from the FP64 table of phi_s (nbk_consts.cu)
// rounded to FP32: g_s = 2 phi_s' and g_s' = 2 phi_s'' are the derivatives of a
// row's polynomial, so nothing cancels at short range.
#include "nbk_internal.cuh"
#include "nbk_launch.h"

namespace nbk {

constexpr int kAdjWarps = 4;
constexpr int kAdjThreads = kAdjWarps * kWarp;
constexpr int kAdjRow = 8;  // floats per row of the FP32 slow table (degree 5, padded)
constexpr size_t kAdjTableBytes = 24 * 1024;  // most shared memory the table's copies take
static_assert(kSlowTableDeg == 5, "slow rows of six coefficients");

// phi_s, phi_s' and phi_s'' of one pair from its table row.
struct SlowRow {
  float phi, d1, d2;
};
__device__ __forceinline__ SlowRow slowRow(const float4 a, const float4 b, const float w) {
  SlowRow r;
  r.phi = fmaf(fmaf(fmaf(fmaf(fmaf(b.y, w, b.x), w, a.w), w, a.z), w, a.y), w, a.x);
  r.d1 = fmaf(fmaf(fmaf(fmaf(5.0f * b.y, w, 4.0f * b.x), w, 3.0f * a.w), w, 2.0f * a.z), w, a.y);
  r.d2 = fmaf(fmaf(fmaf(20.0f * b.y, w, 12.0f * b.x), w, 6.0f * a.w), w, 2.0f * a.z);
  return r;
}

// One warp per tile list, a tile as 16 blocks of 8 x 8 atoms as in the force
// kernel (two j atoms per lane through packed FP32, i and j sums in registers
// over a list part and over a row of blocks). By diagonals of the tile, one
// pair per lane and step with the j sums rotated between steps, it took 410 us
// at 24,000 atoms.
//
// The LJ gradients of a pair go to one of kAdjCopies FP64 tables in global
// memory with two reductions that nothing waits for. In shared memory an FP32
// add is a compare-and-swap loop, and the water model's few types make lanes
// meet in it: with one loop for both sums the kernel took 313 us.
// Reductions of many blocks into one word follow one another: with sixteen tables
// and all types wanted (the water model's pairs meet in a few words) 92,224 atoms
// took 1,445 us, with sixty-four 559; 24,000 atoms with the solute's types alone
// 151.5 and 148.8.
template <bool doSlow, bool kShared>
__global__ void __launch_bounds__(kAdjThreads, 4) adjointKernel(const __grid_constant__ AdjArgs a) {
  // the slow table's copies (kShared), the LJ table (A, -B)
  extern __shared__ __align__(16) float4 s_dyn[];
  // i atoms: (-x, -y, -z, q), (wF, type), (wS, -)
  __shared__ float4 s_i[kAdjWarps][3][kWarp];
  // j atoms by pairs (j, j + 4), two copies in turned order as in the force
  // kernel: (x, x', y, y'), (z, z', q, q'), -wF and -wS likewise; types
  __shared__ float4 s_j[kAdjWarps][2][5][16];
  __shared__ float2 s_jt[kAdjWarps][2][16];
  const NbkConst& c = a.c;
  const PackedConst& k = a.pk;
  const int dim = c.ljDim, d2 = dim * dim;
  const int tabEntries = kShared ? 2 * a.slowRows * a.tabCopies : 0;
  float2* s_lj = reinterpret_cast<float2*>(s_dyn + tabEntries);
  double* const gAB = a.gradCopies + (size_t)(blockIdx.x % kAdjCopies) * 2 * d2;
  for (int m = threadIdx.x; m < tabEntries; m += blockDim.x)
    s_dyn[m] = a.slowTable[(unsigned)m / (unsigned)a.tabCopies];
  for (int m = threadIdx.x; m < d2; m += blockDim.x)
    s_lj[m] = make_float2(a.ljTable[m].x, -a.ljTable[m].y);
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int li = lane & 7, lj = lane >> 3;
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
  const unsigned adrI = sharedAddr(&s_i[wib][0][li]), adrJ = sharedAddr(&s_j[wib][b2][0][lj]),
                 adrT = sharedAddr(&s_jt[wib][b2][lj]), adrLJ = sharedAddr(s_lj),
                 stride = 16u * a.tabCopies,
                 adrTab = sharedAddr(s_dyn + (lane & (a.tabCopies - 1))) - kRowMagicBits * 2u * stride;
  const float sMax = a.slowStep * (float)(a.slowRows - 1);
  const int numLists = *a.numListsDev;
  for (;;) {
    const int W = drawItem(a.workCounter, lane);
    if (W >= numLists << a.splitLog2) break;
    const nbk_tile_list tl = a.lists[W >> a.splitLog2];
    // the part's tiles (contiguous parts of equal length, the last ones shorter)
    const int split = 1 << a.splitLog2;
    const int chunk = (tl.jtileEnd - tl.jtileStart + split) >> a.splitLog2;
    const int jtFirst = tl.jtileStart + (W & (split - 1)) * chunk;
    const int jtLast = min(tl.jtileEnd, jtFirst + chunk - 1);
    if (jtLast < jtFirst) continue;  // warp-uniform
    const float3 sh = shiftOf(make_float3(tl.offsetXYZ.x, tl.offsetXYZ.y, tl.offsetXYZ.z), a.lata,
                              a.latb, a.latc);
    const int iatom = tl.iatomStart + lane;
    // byte offsets of types in the tables; bit 0 marks a type whose LJ gradients are wanted
    {
      const float4 xi = a.xyzq[iatom], wf = a.wF[iatom];
      const float4 ws = doSlow ? a.wS[iatom] : make_float4(0.f, 0.f, 0.f, 0.f);
      const int ty = a.vdwTypes[iatom];
      const float x = -__fadd_rn(xi.x, sh.x), y = -__fadd_rn(xi.y, sh.y), z = -__fadd_rn(xi.z, sh.z);
      const int off = ty * dim * 8 + (a.typeMask[ty] != 0 ? 1 : 0);
      s_i[wib][0][lane] = make_float4(x, y, z, xi.w);
      s_i[wib][1][lane] = make_float4(wf.x, wf.y, wf.z, __int_as_float(off));
      s_i[wib][2][lane] = ws;
    }
    float gi[4][4];  // sums of v (= -dL/dx_i) and of q_j dL/dqq for the atoms 8 I + li
#pragma unroll
    for (int I = 0; I < 4; ++I) gi[I][0] = gi[I][1] = gi[I][2] = gi[I][3] = 0.f;
    for (int jt = jtFirst; jt <= jtLast; ++jt) {
      const unsigned mask = a.tileExcls[jt].excl[lane];  // block order
      const int jstart = a.tileJatomStart[jt];
      {
        const float4 xj = a.xyzq[jstart + lane], wf = a.wF[jstart + lane];
        const float4 ws = doSlow ? a.wS[jstart + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int ty = a.vdwTypes[jstart + lane];
        const int off = ty * 8 + (a.typeMask[ty] != 0 ? 1 : 0);
        const int m = (lane >> 3) * 4 + (lane & 3), e = (lane >> 2) & 1;
#pragma unroll
        for (int copy = 0; copy < 2; ++copy) {
          const int ec = copy ? 1 - e : e;
          float* p = reinterpret_cast<float*>(&s_j[wib][copy][0][m]) + ec;
          p[0] = xj.x;
          p[2] = xj.y;
          p[64] = xj.z;
          p[66] = xj.w;
          p[128] = -wf.x;
          p[130] = -wf.y;
          p[192] = -wf.z;
          p[194] = -ws.z;
          p[256] = -ws.x;
          p[258] = -ws.y;
          reinterpret_cast<int*>(&s_jt[wib][copy][m])[ec] = off;
        }
      }
      unsigned todo = __reduce_or_sync(0xffffffffu, mask);
      __syncwarp();
#pragma unroll 1
      while (todo) {  // live rows of blocks (warp-uniform)
        const int J8 = (__ffs(todo) - 1) & 24;
        const unsigned rowAny = (todo >> J8) & 0xffu;
        todo &= ~(0xffu << J8);
        const unsigned mrow = mask >> J8;
        const unsigned aj = adrJ + J8 * 8;
        const float4 j0 = ldShared4(aj), j1 = ldShared4(aj + 256), j2 = ldShared4(aj + 512),
                     j3 = ldShared4(aj + 768);
        const float4 j4 = doSlow ? ldShared4(aj + 1024) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 tj = ldShared2(adrT + J8 * 4);
        const float2 QJ = make_float2(j1.z, j1.w);
        float2 gj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) gj[q] = f2(0.f);
#pragma unroll
        for (int I = 0; I < 4; ++I) {
          if (!(rowAny & (0x11u << I))) continue;  // warp-uniform
          const unsigned ai = adrI + 128 * I;
          const float4 xi = ldShared4(ai);
          const float2 DX = make_float2(j0.x + xi.x, j0.y + xi.x),
                       DY = make_float2(j0.z + xi.y, j0.w + xi.y),
                       DZ = make_float2(j1.x + xi.z, j1.y + xi.z);
          const float2 R2 = fma2(DZ, DZ, fma2(DX, DX, mul2(DY, DY)));  // dist2's order
          const bool aA = (mrow & (1u << I)) && (R2.x < c.cutoff2);
          const bool aB = (mrow & (0x10u << I)) && (R2.y < c.cutoff2);
          if (!__any_sync(0xffffffffu, aA || aB)) continue;
          const float4 wi = ldShared4(ai + 512);
          const float2 UX = make_float2(wi.x + j2.x, wi.x + j2.y),
                       UY = make_float2(wi.y + j2.z, wi.y + j2.w),
                       UZ = make_float2(wi.z + j3.x, wi.z + j3.y);
          const float2 pF = fma2(UZ, DZ, fma2(UY, DY, mul2(UX, DX)));
          const int ti = __float_as_int(wi.w);
          const int tA = ti + __float_as_int(tj.x), tB = ti + __float_as_int(tj.y);
          const float2 abA = ldShared2(adrLJ + (tA & ~7)), abB = ldShared2(adrLJ + (tB & ~7));
          const float2 A = make_float2(abA.x, abB.x), nB = make_float2(abA.y, abB.y);
          const float2 rinv = make_float2(rsqrtApprox(R2.x), rsqrtApprox(R2.y));
          const float2 si = mul2(rinv, rinv);  // 1/s
          const float2 rinv3 = mul2(rinv, si);
          const float2 s3 = mul2(mul2(si, si), si), s6 = mul2(s3, s3);
          // the switch S and its derivatives in s: with d and T as at
          // PackedConst, S = -(d (T - 6 c1 D d))/6, S' = T/2, S'' = 6 c1 (D - 2 d)
          // beyond rs, 0 below
          const float2 drs = make_float2(k.rc2 - R2.x, k.rc2 - R2.y);
          const float2 dd = make_float2(fminf(drs.x, k.dMax), fminf(drs.y, k.dMax));
          const float2 TT = mul2(dd, fma2(k.dB, dd, k.dA));
          const float2 S = mul2(mul2(dd, fma2(k.hA, dd, TT)), f2(-1.0f / 6.0f));
          const float2 S1 = mul2(TT, f2(0.5f));
          const float2 S2r = fma2(mul2(k.dB, f2(-1.0f)), dd, neg2(k.hA));
          const float2 S2 = make_float2(drs.x < k.dMax ? S2r.x : 0.f, drs.y < k.dMax ? S2r.y : 0.f);
          // LJ, E = A s^-6 S - B s^-3 S: gA, gB = 2 d/ds per unit A, -B, and g_lj'
          const float2 m = mul2(si, S);
          const float2 gA = mul2(s6, fma2(f2(-12.0f), m, TT));
          const float2 gnB = mul2(s3, fma2(f2(-6.0f), m, TT));
          const float2 glj = fma2(A, gA, mul2(nB, gnB));
          const float2 hA = mul2(s6, fma2(si, fma2(f2(42.0f), m, mul2(f2(-12.0f), S1)), S2));
          const float2 hB = mul2(s3, fma2(si, fma2(f2(12.0f), m, mul2(f2(-6.0f), S1)), S2));
          const float2 hlj = fma2(A, hA, mul2(nB, hB));  // g_lj' / 2
          const float2 qi = f2(xi.w), qq = mul2(qi, QJ);
          const float2 gf = add2(k.rc3inv, neg2(rinv3));
          const float2 hf = mul2(f2(0.75f), mul2(rinv3, si));  // g_f' / 2
          const float2 phif = add2(rinv, neg2(fma2(f2(c.hB), R2, f2(c.hA))));
          const float2 g = fma2(qq, gf, glj);
          // radial: 2 (pF g' + pS gs') + cV g_lj + cE qq g_f + cS qq g_s
          float2 rad = fma2(mul2(pF, f2(4.0f)), fma2(qq, hf, hlj), mul2(f2(a.cV), glj));
          float2 qr = mul2(f2(a.cE), gf);
          float2 dqq = fma2(pF, gf, mul2(f2(a.cE), phif));
          float2 VX = mul2(g, UX), VY = mul2(g, UY), VZ = mul2(g, UZ);
          if constexpr (doSlow) {
            const float4 vi = ldShared4(ai + 1024);
            const float2 WX = make_float2(vi.x + j4.x, vi.x + j4.y),
                         WY = make_float2(vi.y + j4.z, vi.y + j4.w),
                         WZ = make_float2(vi.z + j3.z, vi.z + j3.w);
            const float2 pS = fma2(WZ, DZ, fma2(WY, DY, mul2(WX, DX)));
            const float2 sc = make_float2(fminf(R2.x, sMax), fminf(R2.y, sMax));
            const float2 t = fma2(sc, f2(a.slowInvStep), f2(kRowMagic));
            const float2 w = fma2(add2(t, f2(-kRowMagic)), f2(-a.slowStep), sc);
            SlowRow ra, rb;
            if constexpr (kShared) {
              const unsigned pa = adrTab + __float_as_uint(t.x) * 2u * stride,
                             pb = adrTab + __float_as_uint(t.y) * 2u * stride;
              ra = slowRow(ldShared4(pa), ldShared4(pa + stride), w.x);
              rb = slowRow(ldShared4(pb), ldShared4(pb + stride), w.y);
            } else {
              const float4* pa = a.slowTable + 2 * (size_t)(__float_as_uint(t.x) - kRowMagicBits);
              const float4* pb = a.slowTable + 2 * (size_t)(__float_as_uint(t.y) - kRowMagicBits);
              ra = slowRow(__ldg(pa), __ldg(pa + 1), w.x);
              rb = slowRow(__ldg(pb), __ldg(pb + 1), w.y);
            }
            const float2 gs = make_float2(2.0f * ra.d1, 2.0f * rb.d1);
            const float2 d2s = make_float2(ra.d2, rb.d2);  // gs' / 2
            const float2 phis = make_float2(ra.phi, rb.phi);
            rad = fma2(mul2(pS, f2(4.0f)), mul2(qq, d2s), rad);
            qr = fma2(f2(a.cS), gs, qr);
            dqq = fma2(pS, gs, fma2(f2(a.cS), phis, dqq));
            const float2 gq = mul2(qq, gs);
            VX = fma2(gq, WX, VX);
            VY = fma2(gq, WY, VY);
            VZ = fma2(gq, WZ, VZ);
          }
          rad = fma2(qq, qr, rad);
          VX = fma2(rad, DX, VX);
          VY = fma2(rad, DY, VY);
          VZ = fma2(rad, DZ, VZ);
          // an element that is no interacting pair may hold anything (a padding
          // slot's cotangent may be NaN): exact zeros in place of what it adds
          VX = make_float2(aA ? VX.x : 0.f, aB ? VX.y : 0.f);
          VY = make_float2(aA ? VY.x : 0.f, aB ? VY.y : 0.f);
          VZ = make_float2(aA ? VZ.x : 0.f, aB ? VZ.y : 0.f);
          dqq = make_float2(aA ? dqq.x : 0.f, aB ? dqq.y : 0.f);
          gi[I][0] += VX.x + VX.y;
          gi[I][1] += VY.x + VY.y;
          gi[I][2] += VZ.x + VZ.y;
          gi[I][3] = fmaf(QJ.y, dqq.y, fmaf(QJ.x, dqq.x, gi[I][3]));
          gj[0] = add2(gj[0], VX);
          gj[1] = add2(gj[1], VY);
          gj[2] = add2(gj[2], VZ);
          gj[3] = fma2(qi, dqq, gj[3]);
          // dL/dA = pF gA + cV s^-6 S, dL/dB = -(pF gnB + cV s^-3 S)
          const float2 cS6 = mul2(f2(a.cV), S);
          const float2 LA = fma2(pF, gA, mul2(cS6, s6)), LB = neg2(fma2(pF, gnB, mul2(cS6, s3)));
          const bool wA = aA && ((ti | __float_as_int(tj.x)) & 1),
                     wB = aB && ((ti | __float_as_int(tj.y)) & 1);
          if (wA) {
            atomicAdd(gAB + (tA >> 3), (double)LA.x);
            atomicAdd(gAB + d2 + (tA >> 3), (double)LB.x);
          }
          if (wB) {
            atomicAdd(gAB + (tB >> 3), (double)LA.y);
            atomicAdd(gAB + d2 + (tB >> 3), (double)LB.y);
          }
        }
        // the row's sums over the eight i lanes; lane bits 1 and 0 keep one of
        // the components x, y, z, q of the lane's j atom
        float u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = gj[q].x + __shfl_xor_sync(0xffffffffu, gj[q].y, 4);
        const float lo = keepHalf(u[0], u[2], b1, 2), hi = keepHalf(u[1], u[3], b1, 2);
        const float v = keepHalf(lo, hi, b0, 1);
        if (v != 0.f)
          atomicAddFixed(&a.grad[(size_t)((b1 ? 2 : 0) + (b0 ? 1 : 0)) * a.stride + jstart + J8 +
                                 (lane & 4) + lj],
                         toFixedForce(v));
      }
      __syncwarp();
    }
    // i sums over the four j lanes: every lane ends up with its own atom
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float lo = keepHalf(gi[0][q], gi[2][q], b4, 16), hi = keepHalf(gi[1][q], gi[3][q], b4, 16);
      const float v = keepHalf(lo, hi, b3, 8);
      if (v != 0.f)
        atomicAddFixed(&a.grad[(size_t)q * a.stride + iatom], toFixedForce(q < 3 ? -v : v));
    }
    __syncwarp();
  }
}

// The LJ gradient tables' sum: a block sums 32 entries, each of its eight warps an
// eighth of the copies.
__global__ void __launch_bounds__(256) adjointTableKernel(int n, const double* __restrict__ copies,
                                                          double* __restrict__ out) {
  __shared__ double s_sum[8][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (i < n) {
#pragma unroll
    for (int k = 0; k < kAdjCopies / 8; ++k) s += copies[(size_t)(wib * (kAdjCopies / 8) + k) * n + i];
  }
  s_sum[wib][lane] = s;
  __syncthreads();
  if (wib || i >= n) return;
#pragma unroll
  for (int w = 1; w < 8; ++w) s += s_sum[w][lane];
  out[i] = s;
}

// Fixed-point gradients -> float4 (gx, gy, gz, gq) per slot.
__global__ void adjointOutKernel(int n, const long long* __restrict__ g, int stride,
                                 float4* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = make_float4((float)(g[i] * kForceScaleInv), (float)(g[stride + i] * kForceScaleInv),
                         (float)(g[2 * (size_t)stride + i] * kForceScaleInv),
                         (float)(g[3 * (size_t)stride + i] * kForceScaleInv));
}

template <bool S, bool SH>
static cudaError_t launchAdj(const AdjArgs& a, size_t shmem, int numSM, cudaStream_t st) {
  static KernelLimits limits;
  auto k = adjointKernel<S, SH>;
  int blocks = 0;
  const cudaError_t e = limits.blocksPerSM(k, kAdjThreads, shmem, &blocks);
  if (e != cudaSuccess) return e;
  k<<<numSM * blocks, kAdjThreads, shmem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launchAdjoint(const AdjArgs& args, bool doSlow, int numSM, int n, float4* out,
                          cudaStream_t st) {
  AdjArgs a = args;
  const int d2 = a.c.ljDim * a.c.ljDim;
  const size_t tables = sizeof(float2) * (size_t)d2;
  // eight interleaved copies of the slow table where they fit (the lanes of a
  // quarter warp then read from different bank groups whatever rows they want),
  // the table in global memory where not even one does
  const size_t one = sizeof(float) * kAdjRow * (size_t)a.slowRows;
  a.tabCopies = 8;
  while (a.tabCopies > 1 && one * a.tabCopies > kAdjTableBytes) a.tabCopies /= 2;
  cudaError_t e;
  if (!doSlow) {
    a.tabCopies = 1;
    e = launchAdj<false, false>(a, tables, numSM, st);
  } else if (one <= kAdjTableBytes) {
    e = launchAdj<true, true>(a, tables + one * a.tabCopies, numSM, st);
  } else {
    a.tabCopies = 1;
    e = launchAdj<true, false>(a, tables, numSM, st);
  }
  if (e != cudaSuccess) return e;
  adjointTableKernel<<<(2 * d2 + 31) / 32, 256, 0, st>>>(2 * d2, a.gradCopies, a.gradAB);
  e = cudaGetLastError();
  if (e != cudaSuccess || !out) return e;
  adjointOutKernel<<<min((n + 255) / 256, numSM * 4), 256, 0, st>>>(n, a.grad, a.stride, out);
  return cudaGetLastError();
}

}  // namespace nbk
