// Host-side launchers of the B200 nonbonded kernels (internal to libnbk).
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "nbk_internal.cuh"

namespace nbk {

// Dynamic shared memory and occupancy of one kernel instance, per device. Handles
// on several host threads launch one instance with different sizes at once, so
// the limit is only ever raised: a launch that follows outside the lock finds at
// least what it asked for. Occupancy is looked up once for each of the sizes
// last in use.
class KernelLimits {
 public:
  template <typename K>
  cudaError_t allow(K kernel, size_t shmem) {
    int dev = 0;
    const cudaError_t e = device(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    return raise(kernel, dev, shmem);
  }
  template <typename K>
  cudaError_t blocksPerSM(K kernel, int threads, size_t shmem, int* blocks) {
    int dev = 0;
    cudaError_t e = device(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    PerDevice& d = devices[dev];
    for (int k = 0; k < kSizes; ++k)
      if (d.blocks[k] > 0 && d.shmem[k] == shmem) {
        *blocks = d.blocks[k];
        return cudaSuccess;
      }
    e = raise(kernel, dev, shmem);
    int nb = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, shmem);
    if (e != cudaSuccess) return e;
    d.shmem[d.next] = shmem;
    *blocks = d.blocks[d.next] = nb > 0 ? nb : 1;
    d.next = (d.next + 1) % kSizes;
    return cudaSuccess;
  }
  // Interleaved copies of a table of `one` bytes beside `rest` bytes of other dynamic
  // shared memory: as many of 8, 4, 2, 1 as `most` bytes hold and as leave the
  // blocks per SM that one copy leaves.
  template <typename K>
  cudaError_t tableCopies(K kernel, int threads, size_t rest, size_t one, size_t most, int* copies,
                          int* blocks) {
    cudaError_t e = blocksPerSM(kernel, threads, rest + one, blocks);
    for (*copies = 8; e == cudaSuccess && *copies > 1; *copies /= 2) {
      int nb = 0;
      if (one * *copies > most) continue;
      e = blocksPerSM(kernel, threads, rest + one * *copies, &nb);
      if (nb == *blocks) break;
    }
    return e;
  }

 private:
  static constexpr int kDevices = 64, kSizes = 16;
  struct PerDevice {
    size_t allowed = 0;
    size_t shmem[kSizes] = {};
    int blocks[kSizes] = {};  // 0: free
    int next = 0;
  };
  static cudaError_t device(int* dev) {
    const cudaError_t e = cudaGetDevice(dev);
    return e != cudaSuccess ? e : (*dev < 0 || *dev >= kDevices) ? cudaErrorInvalidDevice : cudaSuccess;
  }
  template <typename K>
  cudaError_t raise(K kernel, int dev, size_t shmem) {
    if (shmem <= devices[dev].allowed) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shmem);
    if (e == cudaSuccess) devices[dev].allowed = shmem;
    return e;
  }
  std::mutex mu;
  PerDevice devices[kDevices];
};

// Launches a kernel that may be scheduled while the kernel before it in the
// stream still runs; it calls waitForPredecessor before it uses anything that
// one writes. Saves the gap between two small kernels.
template <typename... P, typename... A>
cudaError_t launchOverlapped(void (*kernel)(P...), int blocks, int threads, size_t shmem,
                             cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = shmem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Copies host data up and returns once it has landed: a copy from pageable
// memory may return before that, and the caller's next stream need not wait for
// the default one.
inline cudaError_t uploadNow(void* dst, const void* src, size_t bytes) {
  const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

// Zeroes the 64-bit words a[0, na), b[0, nb) and the 32-bit words c[0, nc),
// d[0, nd) in one launch (memsets cost a gap each).
cudaError_t launchClear(long long* a, size_t na, long long* b, size_t nb, int* c, int nc, int* d,
                        int nd, int numSM, cudaStream_t st);

// Pair-math constants from the caller's parameters (nbk_consts.cu); shared by
// the handle and by the allocation-free entry point.
void makeConstants(const nbk_params& p, int ljDim, NbkConst& c, NbkConst64& k);
void makePacked(const NbkConst64& k, PackedConst& c);
int buildForceTable(double beta, double cutoff, double pairlistdist, std::vector<float4>& out,
                    double* step);
// The FP64 slow-term table of the force kernel's precise pass; returns rows.
int buildSlowTable(double beta, double cutoff, double pairlistdist, std::vector<double>& out,
                   double* step);

// minBlocks: 4, 5 or 6 CTAs per SM (the register cap); a.splitLog2 set by the caller.
cudaError_t launchForce(const ForceArgs& a, unsigned flags, int minBlocks, int numSM,
                        cudaStream_t st);
// Whether the force kernel's slow table leaves it the blocks per SM that it has
// without one.
cudaError_t forceTableFits(int ljDim, int rows, bool* fits);
// The precise energy / virial kernel after the force kernel (same lists, the
// force kernel's live words, its own work counter a.workCounter); no-op when
// flags need neither energies nor the slow virial.
bool needsPrecise(unsigned flags);
cudaError_t launchPrecise(const ForceArgs& a, unsigned flags, int numSM, cudaStream_t st);
// Pairlist refinement of the culled lists a.lists[0, a.numListsHost): writes
// a.tileExcls, a.tileJatomOut, a.listActive, a.lenHist (unless NULL),
// a.counts[1] (tiles kept) and the excluded-pair counts.
cudaError_t launchRefine(const ForceArgs& a, int numSM, cudaStream_t st);

// The lists of src that kept tiles (listActive), as dst in order of decreasing
// j-tile count; hist: their counts by length 1..maxLen (clamped), used up as
// cursors; counts[0] receives their number.
cudaError_t launchSortLists(int numLists, const nbk_tile_list* src, const int* listActive,
                            int maxLen, int* hist, int* counts, nbk_tile_list* dst, int numSM,
                            cudaStream_t st);

cudaError_t launchBBoxes(int numTiles, const float4* xyzq, BBox* bb, cudaStream_t st);

cudaError_t launchBuildLists(int numLists, const ListSeed* seeds,
                             const nbk_compute_record* computes, const nbk_patch_record* patches,
                             const BBox* bb, float3 lata, float3 latb, float3 latc,
                             const int* compRep, const float3* repLat, float plcutoff2Culling,
                             nbk_tile_list* lists, PatchPair* pp, int* tileJatomStart,
                             cudaStream_t st);

// The same lists in their own order (counters[0] zeroed before).
cudaError_t launchCompact(int numLists, const nbk_tile_list* src, const int* listActive,
                          nbk_tile_list* dst, int* counters, int numSM, cudaStream_t st);

// Tiles of the refined lists into packed arrays (list k's at dst[k]) in the
// interface's bit order.
cudaError_t launchExportTiles(int numLists, const nbk_tile_list* lists, const int* dst,
                              const int* jatom, const nbk_tile_excl* excl, int* jatomOut,
                              nbk_tile_excl* exclOut, cudaStream_t st);

struct CorrArgs {
  const nbk_exclusion* modified;
  int numModified;
  const nbk_exclusion* excluded;
  int numExcluded;
  const float4* xyzq;
  const float2* ljExclTable;  // (A14 - A, B14 - B) * scaling
  float3 lata, latb, latc;
  NbkConst c;
  long long* force;
  int stride;
  long long* acc;
  NbkConst64 c64;
  // replicas (batched evaluation; NULL for a single system)
  const int* slotRep;          // [atomStorageSize] replica of each atom slot
  const float3* repLat;        // [3*numReplicas]
  const float2* repLJExcl;     // [numReplicas][ljDim*ljDim] (A14 - A, B14 - B) * scaling
};
// besideForce: the kernel before it in the stream is the force kernel, whose end
// it does not need (its own end waits for it).
cudaError_t launchCorrections(const CorrArgs& a, unsigned flags, bool besideForce, cudaStream_t st);

// The lattice-shift part of the virial, (sum_i F_i) (x) shift per compute,
// from the exact integer i-force sums the force kernel leaves per compute.
struct ShiftVirialArgs {
  int numComputes;
  const long long* compF;                // [numComputes][6] (0..2: fast i-force sums)
  const nbk_compute_record* computes;
  float3 lata, latb, latc;
  const int* compRep;                    // batched replicas, else NULL
  const float3* repLat;
};

// With NBK_VIRIAL: the per-atom part of the fast virial, and with shift also
// its lattice-shift part, into the accumulators.
cudaError_t launchFinalizeForces(int n, const long long* force, int stride, const float4* xyzq,
                                 float4* outF, float4* outS, unsigned flags, long long* acc,
                                 int numSM, cudaStream_t st, const int* slotRep = nullptr,
                                 const ShiftVirialArgs* shift = nullptr,
                                 float4* outFHost = nullptr, float4* outSHost = nullptr);

// Device-visible address of host memory page-locked in the current device's
// context (the same pointer under unified addressing), or nullptr for any
// other pointer.
void* mappedHostPointer(void* p);

// Converts numReplicas accumulator blocks into numReplicas nbk_virial_energy records.
cudaError_t launchEnergyVirial(const long long* acc, nbk_virial_energy* out, cudaStream_t st,
                               int numReplicas = 1);

constexpr int kAdjCopies = 64;  // a multiple of 8
struct AdjArgs {
  const nbk_tile_list* lists;
  const int* numListsDev;
  const int* tileJatomStart;
  const nbk_tile_excl* tileExcls;
  const float4* xyzq;
  const int* vdwTypes;
  const float2* ljTable;
  const int* typeMask;   // [ljDim] 1: accumulate LJ gradients of pairs touching this type
  const float4* wF;      // fast-force cotangent per slot (w ignored)
  const float4* wS;      // slow-force cotangent per slot (NULL: zero)
  float cV, cE, cS;
  float3 lata, latb, latc;
  NbkConst c;
  PackedConst pk;
  const float4* slowTable;  // phi_s rows rounded to FP32: (c0..c3), (c4, c5, -, -)
  int slowRows, tabCopies;  // tabCopies: set by the launch
  float slowStep, slowInvStep;
  long long* grad;       // SoA [4][stride]: gx, gy, gz, gq (fixed point, force scale)
  int stride;
  double* gradAB;        // [2][ljDim*ljDim]
  double* gradCopies;    // [kAdjCopies][2][ljDim*ljDim], zeroed (FP64 atomics)
  int splitLog2;         // 2^splitLog2 work items per list
  int* workCounter;
};
cudaError_t launchAdjoint(const AdjArgs& a, bool doSlow, int numSM, int n, float4* out,
                          cudaStream_t st);

// Integrator force arrays from the fixed-point sums (nbk_accumulate_forces_to_soa).
struct AccumulateArgs {
  int numPatches, maxForceNumber, stride, forceStride;
  const nbk_local_record* rec;
  const int* sortOrder;
  const long long* fixed;     // [6][stride]: fast x y z, slow x y z
  const double* fBond;        // [3][forceStride] or NULL
  const double* fBondNbond;
  const double* fBondSlow;
  const float3* fPme;         // per buffer atom or NULL
  double* fNormal[3];
  double* fNbond[3];
  double* fSlow[3];
};
cudaError_t launchAccumulateForces(const AccumulateArgs& a, cudaStream_t st);

// Sets the message nbk_last_error returns on this thread; returns code.
int setLastError(int code, const std::string& msg);

// Per-slot vdW types, atom indices and exclusion indices from per-atom arrays
// in buffer order (GPU-resident marshaling, nbk_resident.cu).
cudaError_t launchUpdateVdwTypesExclDevice(int numPatches, const nbk_local_record* rec,
                                           const int* vdw, const int* gid, const int* sortOrder,
                                           const int2* exclByAtom, int numExclAtoms, int ljDim,
                                           int storage, int* vdwTypes, int* atomIndex, int2* excl,
                                           int* status, cudaStream_t st);

}  // namespace nbk
