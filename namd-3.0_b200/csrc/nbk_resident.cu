// GPU-resident input marshaling: the patch sort, the patch-centred xyzq and
// the per-slot vdW types / exclusion indices built on the device from the
// integrator's per-atom arrays (declared in include/nbk.h).
//
// The reference does this work on the host for the non-resident path
// (src/SortAtoms.C:45-133, src/HomePatch.C:1054-1131,
// src/CudaComputeNonbonded.C:836-930) and with the GPU-resident integrator in
// setComputePositionsKernel (src/SequencerCUDAKernel.cu:1950-2041) and
// updateVdwTypesExclKernel (src/CudaComputeNonbondedKernel.cu:3648-3724).
// Here one block handles one patch for all three; the sort keeps the whole
// patch in shared memory and ranks atoms by counting, so it needs no global
// scratch and no host round trip.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "nbk.h"
#include "nbk_internal.cuh"
#include "nbk_launch.h"

namespace nbk {

namespace {

constexpr int kSortMaxThreads = 512;
// every part that is split straddles an 8-atom block boundary of its own, so a
// level splits at most N/8 parts into at most N/4
constexpr int kMaxRanges = NBK_MAX_PATCH_ATOMS / 4;

struct Lattice12 {
  double ax, ay, az, bx, by, bz, cx, cy, cz, ox, oy, oz;
};

// Split point of the part [begin, end) of a patch (positions within the
// patch): the first of 32, 16, 8 whose blocks the part straddles, at the
// block boundary nearest the middle; -1 when the part is not split further.
__device__ __forceinline__ int splitPoint(int begin, int end) {
  int W = 0;
  if (begin / 32 < (end - 1) / 32) W = 32;
  else if (begin / 16 < (end - 1) / 16) W = 16;
  else if (begin / 8 < (end - 1) / 8) W = 8;
  if (W == 0) return -1;
  int split = ((begin + end + W) / (2 * W)) * W;
  if (split <= begin) split += W;
  if (split >= end) split -= W;
  if (split <= begin || split >= end) return -1;
  return split;
}

// A coordinate as an integer of the same order, -0 as 0. NaN, which no comparison
// of doubles orders, lies beyond the infinities.
__device__ __forceinline__ long long orderKey(const double v) {
  const long long b = __double_as_longlong(v + 0.0);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// One block per patch, a thread per position (more positions than threads go
// round). Shared memory (dynamic) per atom for maxN atoms: x, y, z and the
// current split key (double), id, ord, tmp, the position's part and its rank (int).
//
// Every level orders all parts at once: a thread counts the keys of its
// position's part that are below its own, one FP64 compare a candidate read as
// a broadcast, and equal keys (and NaN) are found afterwards, as two atoms with
// one rank, and only then told apart by id. What bounds it is the sum of those counts,
// about 2 n^2 compares a patch over the levels, and the barriers between the
// steps. 92,224 atoms in 320 patches: 188 us when the parts of a level were
// taken one after the other by the whole block.
__global__ void __launch_bounds__(kSortMaxThreads)
    sortPatchAtomsKernel(int numPatches, const nbk_local_record* __restrict__ rec, int maxN,
                         const double* __restrict__ px, const double* __restrict__ py,
                         const double* __restrict__ pz, const int* __restrict__ gid,
                         int* __restrict__ sortOrder, int* __restrict__ status) {
  extern __shared__ double s_dyn[];
  double* s_x = s_dyn;
  double* s_y = s_x + maxN;
  double* s_z = s_y + maxN;
  double* s_key = s_z + maxN;  // by position: the coordinate the position's part is split on
  int* s_id = reinterpret_cast<int*>(s_key + maxN);
  int* s_ord = s_id + maxN;
  int* s_tmp = s_ord + maxN;
  int* s_part = s_tmp + maxN;  // by position: its part, -1 when it is split no further
  int* s_rank = s_part + maxN;
  __shared__ int s_rb[2][kMaxRanges], s_re[2][kMaxRanges], s_rs[kMaxRanges], s_ax[kMaxRanges];
  __shared__ int s_child[kMaxRanges];  // index of a split part among the split ones
  __shared__ int s_numNext, s_tie;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, warps = blockDim.x >> 5;
  admitSuccessor();
  for (int p = blockIdx.x; p < numPatches; p += gridDim.x) {
    const int n = rec[p].numAtoms, off = rec[p].bufferOffset;
    if (n <= 0) continue;  // block-uniform
    if (n > maxN) {
      for (int k = threadIdx.x; k < n; k += blockDim.x) sortOrder[off + k] = k;
      if (threadIdx.x == 0 && status) atomicAdd(status, 1);
      continue;
    }
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      s_x[k] = px[off + k];
      s_y[k] = py[off + k];
      s_z[k] = pz[off + k];
      s_id[k] = gid[off + k];
      s_ord[k] = k;
      s_part[k] = 0;
    }
    if (threadIdx.x == 0) {
      s_rb[0][0] = 0;
      s_re[0][0] = n;
      s_tie = 0;
    }
    __syncthreads();
    int cur = 0, nr = 1;
    while (nr) {  // one level of the bisection per pass (block-uniform)
      const int *rb = s_rb[cur], *re = s_re[cur];
      // split point and longest axis of every part (a warp per part)
      for (int r = wib; r < nr; r += warps) {
        const int b = rb[r], e = re[r];
        const int sp = splitPoint(b, e);
        // lows and negated highs: six minima over the warp. Lanes halve the
        // values they hold step by step (3, 2 of 4, 1), so that 8 instead of 30
        // values cross lanes; quantity 3 b16 + 2 b8 + b4 ends in the lanes of
        // those bits
        double v[6] = {1e300, 1e300, 1e300, 1e300, 1e300, 1e300};
        if (sp >= 0) {
          for (int k = b + lane; k < e; k += 32) {
            const int a = s_ord[k];
            v[0] = fmin(v[0], s_x[a]);
            v[1] = fmin(v[1], s_y[a]);
            v[2] = fmin(v[2], s_z[a]);
            v[3] = fmin(v[3], -s_x[a]);
            v[4] = fmin(v[4], -s_y[a]);
            v[5] = fmin(v[5], -s_z[a]);
          }
        }
        const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4;
        double u[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
          u[q] = fmin(b16 ? v[q + 3] : v[q], __shfl_xor_sync(0xffffffffu, b16 ? v[q] : v[q + 3], 16));
        double w0 = fmin(b8 ? u[2] : u[0], __shfl_xor_sync(0xffffffffu, b8 ? u[0] : u[2], 8));
        const double w1o = __shfl_xor_sync(0xffffffffu, u[1], 8);
        const double w1 = b8 ? w0 : fmin(u[1], w1o);
        double m = fmin(b4 ? w1 : w0, __shfl_xor_sync(0xffffffffu, b4 ? w0 : w1, 4));
        m = fmin(m, __shfl_xor_sync(0xffffffffu, m, 2));
        m = fmin(m, __shfl_xor_sync(0xffffffffu, m, 1));
        double lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int src = 8 * (d >> 1) + 4 * (d & 1);
          lo[d] = __shfl_sync(0xffffffffu, m, src);
          hi[d] = -__shfl_sync(0xffffffffu, m, 16 + src);
        }
        if (lane == 0) {
          int axis = 0;
          if (hi[1] - lo[1] > hi[0] - lo[0]) axis = 1;
          if (hi[2] - lo[2] > hi[axis] - lo[axis]) axis = 2;
          s_rs[r] = sp;
          s_ax[r] = axis;
        }
      }
      __syncthreads();
      // number the split parts in order, and write the next level's parts:
      // both halves of every split part
      if (wib == 0) {
        int m = 0;
        for (int r0 = 0; r0 < nr; r0 += 32) {
          const int r = r0 + lane;
          const bool split = r < nr && s_rs[r] >= 0;
          const unsigned ball = __ballot_sync(0xffffffffu, split);
          if (split) {
            const int c = m + __popc(ball & ((1u << lane) - 1u));
            s_child[r] = c;
            s_rb[cur ^ 1][2 * c] = rb[r];
            s_re[cur ^ 1][2 * c] = s_rs[r];
            s_rb[cur ^ 1][2 * c + 1] = s_rs[r];
            s_re[cur ^ 1][2 * c + 1] = re[r];
          }
          m += __popc(ball);
        }
        if (lane == 0) s_numNext = 2 * m;
      }
      // the split key of every position of a split part, by position, so that
      // the counting reads it without indirection
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int r = s_part[k];
        if (r >= 0 && s_rs[r] >= 0) {
          const double* key = s_ax[r] == 0 ? s_x : (s_ax[r] == 1 ? s_y : s_z);
          s_key[k] = key[s_ord[k]];
        }
      }
      __syncthreads();
      // rank every atom of a split part by its coordinate on the part's axis
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int r = s_part[k];
        if (r < 0 || s_rs[r] < 0) continue;
        const int b = rb[r], e = re[r];
        const double ka = s_key[k];
        int rank = 0;
#pragma unroll 4
        for (int m = b; m < e; ++m) rank += s_key[m] < ka ? 1 : 0;
        s_tmp[b + rank] = s_ord[k];
        s_rank[k] = b + rank;
      }
      __syncthreads();
      // an atom that does not find itself at its rank shares its coordinate
      // with another (or one of them is NaN): ranks are taken again below, with
      // the id as tie break. Otherwise the ranks fill every part; where they did
      // not, the order would hold what the shared memory did before.
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int r = s_part[k];
        if (r < 0 || s_rs[r] < 0) continue;
        if (s_tmp[s_rank[k]] != s_ord[k]) s_tie = 1;
      }
      __syncthreads();
      if (s_tie) {  // block-uniform
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
          const int r = s_part[k];
          if (r < 0 || s_rs[r] < 0) continue;
          const int b = rb[r], e = re[r];
          const double ka = s_key[k];
          const int ia = s_id[s_ord[k]];
          int rank = 0;
          for (int m = b; m < e; ++m) {
            const double kc = s_key[m];
            rank += (kc < ka || (kc == ka && s_id[s_ord[m]] < ia)) ? 1 : 0;
          }
          s_tmp[b + rank] = s_ord[k];
          s_rank[k] = b + rank;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
          const int r = s_part[k];
          if (r < 0 || s_rs[r] < 0) continue;
          if (s_tmp[s_rank[k]] != s_ord[k]) s_tie = 2;
        }
        __syncthreads();
        if (s_tie == 2) {  // block-uniform: NaN, or two atoms with one id
          // a strict order of any input: by coordinate, id and position
          for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const int r = s_part[k];
            if (r < 0 || s_rs[r] < 0) continue;
            const int b = rb[r], e = re[r];
            const long long ka = orderKey(s_key[k]);
            const int ia = s_id[s_ord[k]];
            int rank = 0;
            for (int m = b; m < e; ++m) {
              const long long kc = orderKey(s_key[m]);
              const int ic = s_id[s_ord[m]];
              rank += (kc < ka || (kc == ka && (ic < ia || (ic == ia && m < k)))) ? 1 : 0;
            }
            s_tmp[b + rank] = s_ord[k];
          }
          __syncthreads();
        }
      }
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int r = s_part[k];
        if (r < 0) continue;
        if (s_rs[r] < 0) {
          s_part[k] = -1;
          continue;
        }
        s_ord[k] = s_tmp[k];
        s_part[k] = 2 * s_child[r] + (k >= s_rs[r] ? 1 : 0);
      }
      nr = s_numNext;
      cur ^= 1;
      __syncthreads();
      if (threadIdx.x == 0) s_tie = 0;
    }
    for (int k = threadIdx.x; k < n; k += blockDim.x) sortOrder[off + k] = s_ord[k];
    __syncthreads();
  }
}

__global__ void computePositionsKernel(int numPatches, const nbk_local_record* __restrict__ rec,
                                       const double3* __restrict__ centre, const Lattice12 L,
                                       const int* __restrict__ sortOrder, double qscale,
                                       const double* __restrict__ px, const double* __restrict__ py,
                                       const double* __restrict__ pz,
                                       const float* __restrict__ charge, float4* __restrict__ xyzq) {
  waitForPredecessor();
  for (int p = blockIdx.x; p < numPatches; p += gridDim.x) {
    const int n = rec[p].numAtoms, off = rec[p].bufferOffset, offNB = rec[p].bufferOffsetNBPad;
    const int npad = rec[p].numAtomsNBPad;
    if (n <= 0) continue;
    const double3 s = centre[p];
    // Lattice::unscale: o + a sx + b sy + c sz
    const double ux = L.ox + L.ax * s.x + L.bx * s.y + L.cx * s.z;
    const double uy = L.oy + L.ay * s.x + L.by * s.y + L.cy * s.z;
    const double uz = L.oz + L.az * s.x + L.bz * s.y + L.cz * s.z;
    for (int i = threadIdx.x; i < npad; i += blockDim.x) {
      const int a = off + min(max(sortOrder[off + min(i, n - 1)], 0), n - 1);
      float4 q;
      q.x = (float)(px[a] - ux);
      q.y = (float)(py[a] - uy);
      q.z = (float)(pz[a] - uz);
      q.w = (float)((double)charge[a] * qscale);
      xyzq[offNB + i] = q;
    }
  }
}

__global__ void updateVdwTypesExclDeviceKernel(int numPatches, const nbk_local_record* __restrict__ rec,
                                               const int* __restrict__ vdw, const int* __restrict__ gid,
                                               const int* __restrict__ sortOrder,
                                               const int2* __restrict__ exclByAtom, int numExclAtoms,
                                               int ljDim, int storage, int* __restrict__ vdwTypes,
                                               int* __restrict__ atomIndex, int2* __restrict__ excl,
                                               int* __restrict__ status) {
  waitForPredecessor();
  admitSuccessor();
  for (int p = blockIdx.x; p < numPatches; p += gridDim.x) {
    const int n = rec[p].numAtoms, off = rec[p].bufferOffset, offNB = rec[p].bufferOffsetNBPad;
    const int npad = rec[p].numAtomsNBPad;
    if (n <= 0) continue;
    for (int i = threadIdx.x; i < npad; i += blockDim.x) {
      if (offNB + i >= storage) break;
      const int a = off + min(max(sortOrder[off + min(i, n - 1)], 0), n - 1);
      int t = vdw[a];
      const int id = gid[a];
      int2 e = make_int2(0, 0);
      bool bad = false;
      if (t < 0 || t >= ljDim) {
        t = 0;
        bad = true;
      }
      if (id >= 0 && id < numExclAtoms) {
        const int2 m = exclByAtom[id];  // (maxdiff, base)
        e = make_int2(m.y, m.x);
      } else {
        bad = true;
      }
      vdwTypes[offNB + i] = t;
      atomIndex[offNB + i] = id;
      excl[offNB + i] = e;
      if (bad && status && i < n) atomicAdd(status, 1);
    }
  }
}

__global__ void accumulateForcesKernel(const __grid_constant__ AccumulateArgs a) {
  waitForPredecessor();
  for (int p = blockIdx.x; p < a.numPatches; p += gridDim.x) {
    const int n = a.rec[p].numAtoms, off = a.rec[p].bufferOffset, offNB = a.rec[p].bufferOffsetNBPad;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      const int b = off + min(max(a.sortOrder[off + k], 0), n - 1);  // buffer index of slot k
      const size_t slot = (size_t)offNB + k;
      double fn[3], fb[3], fs[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        fn[c] = a.fBond ? a.fBond[b + (size_t)c * a.forceStride] : 0.0;
        fb[c] = (double)a.fixed[slot + (size_t)c * a.stride] * kForceScaleInv;
        if (a.fBondNbond) fb[c] += a.fBondNbond[b + (size_t)c * a.forceStride];
        fs[c] = a.fPme ? (double)(&a.fPme[b].x)[c] : 0.0;
        fs[c] += (double)a.fixed[slot + (size_t)(3 + c) * a.stride] * kForceScaleInv;
        if (a.fBondSlow) fs[c] += a.fBondSlow[b + (size_t)c * a.forceStride];
      }
      a.fNormal[0][b] = fn[0];
      a.fNormal[1][b] = fn[1];
      a.fNormal[2][b] = fn[2];
      if (a.maxForceNumber >= 1) {
        a.fNbond[0][b] = fb[0];
        a.fNbond[1][b] = fb[1];
        a.fNbond[2][b] = fb[2];
      }
      if (a.maxForceNumber >= 2) {
        a.fSlow[0][b] = fs[0];
        a.fSlow[1][b] = fs[1];
        a.fSlow[2][b] = fs[2];
      }
    }
  }
}

}  // namespace

cudaError_t launchAccumulateForces(const AccumulateArgs& a, cudaStream_t st) {
  if (a.numPatches <= 0) return cudaSuccess;
  return launchOverlapped(accumulateForcesKernel, min(a.numPatches, 65535), 256, 0, st, a);
}

cudaError_t launchUpdateVdwTypesExclDevice(int numPatches, const nbk_local_record* rec,
                                           const int* vdw, const int* gid, const int* sortOrder,
                                           const int2* exclByAtom, int numExclAtoms, int ljDim,
                                           int storage, int* vdwTypes, int* atomIndex, int2* excl,
                                           int* status, cudaStream_t st) {
  if (numPatches <= 0) return cudaSuccess;
  return launchOverlapped(updateVdwTypesExclDeviceKernel, min(numPatches, 65535), 256, 0, st, numPatches,
                          rec, vdw, gid, sortOrder, exclByAtom, numExclAtoms, ljDim, storage, vdwTypes,
                          atomIndex, excl, status);
}

}  // namespace nbk

using namespace nbk;

extern "C" NBK_API int nbk_sort_patch_atoms(int numPatches, const nbk_local_record* d_rec,
                                            int maxPatchAtoms, const double* d_x, const double* d_y,
                                            const double* d_z, const int* d_id, int* d_sortOrder,
                                            int* d_status, void* stream) {
  if (numPatches < 0 || (numPatches && (!d_rec || !d_x || !d_y || !d_z || !d_id || !d_sortOrder)))
    return setLastError(NBK_ERR_ARG, "nbk_sort_patch_atoms: NULL argument");
  if (maxPatchAtoms < 1 || maxPatchAtoms > NBK_MAX_PATCH_ATOMS)
    return setLastError(NBK_ERR_ARG, "nbk_sort_patch_atoms: maxPatchAtoms must be in 1.." +
                                         std::to_string(NBK_MAX_PATCH_ATOMS));
  if (numPatches == 0) return NBK_OK;
  const size_t smem = (size_t)maxPatchAtoms * (4 * sizeof(double) + 5 * sizeof(int));
  static KernelLimits limits;
  cudaError_t e = limits.allow(sortPatchAtomsKernel, smem);
  if (e == cudaSuccess) {
    // a thread per atom of the largest patch where a block can have as many
    const int threads = std::min(kSortMaxThreads, std::max(64, (maxPatchAtoms + 31) / 32 * 32));
    sortPatchAtomsKernel<<<min(numPatches, 65535), threads, smem, (cudaStream_t)stream>>>(
        numPatches, d_rec, maxPatchAtoms, d_x, d_y, d_z, d_id, d_sortOrder, d_status);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess)
    return setLastError(NBK_ERR_CUDA, std::string("nbk_sort_patch_atoms: ") + cudaGetErrorString(e));
  return NBK_OK;
}

extern "C" NBK_API int nbk_set_compute_positions(int numPatches, const nbk_local_record* d_rec,
                                                 const nbk_double3* d_centre, const double* lattice,
                                                 const int* d_sortOrder, double chargeScaling,
                                                 const double* d_x, const double* d_y,
                                                 const double* d_z, const float* d_charge,
                                                 nbk_float4* d_xyzq, void* stream) {
  if (numPatches < 0 || !lattice ||
      (numPatches && (!d_rec || !d_centre || !d_sortOrder || !d_x || !d_y || !d_z || !d_charge ||
                      !d_xyzq)))
    return setLastError(NBK_ERR_ARG, "nbk_set_compute_positions: NULL argument");
  if (numPatches == 0) return NBK_OK;
  Lattice12 L;
  double* l = &L.ax;
  for (int k = 0; k < 12; ++k) l[k] = lattice[k];
  const cudaError_t e = launchOverlapped(
      computePositionsKernel, min(numPatches, 65535), 128, 0, (cudaStream_t)stream, numPatches, d_rec,
      reinterpret_cast<const double3*>(d_centre), L, d_sortOrder, chargeScaling, d_x, d_y, d_z,
      d_charge, reinterpret_cast<float4*>(d_xyzq));
  if (e != cudaSuccess)
    return setLastError(NBK_ERR_CUDA,
                        std::string("nbk_set_compute_positions: ") + cudaGetErrorString(e));
  return NBK_OK;
}
