// Host-callable launchers of the hydro kernels (defined in hydro.cu) and the
// gravity kernels (gravity.cu).
#pragma once
#include "fields.cuh"
#include "sort.cuh"

namespace sph {

struct TableDev {
  const double* w;      // 3*(N1+1) quadratic coefficients of W
  const double* g;      // 3*(N1+1) quadratic coefficients of dW/deta
  const double* herm;   // 2*hermN Hermite knots of the nperh lookup (values, slopes)
  const float4* p32a;   // per interval (w0, w1, w2, g0) in FP32
  const float2* p32b;   // per interval (g1, g2) in FP32
};

struct NeighborLists {
  const uint32_t* nbr;      // entries (index | cell-offset code << 26), warp-interleaved with capacity cap
  const int* count;         // neighbours per node
  int cap;                  // slots per node
  const uint32_t* cell;     // home cell of every node (packed, 10 bits per axis)
};

constexpr int kEntrySums = 32;
constexpr int kDtReasons = 6;
// Values the kernels of a step leave for the host, one per handle.  Reset by
// the first kernel of a neighbour build.
struct StepScratch {
  long long bounds[10];        // end of step: order keys of min h^-1, min xyz, max xyz, tensor half-widths
  int bad;                     // non-finite or non-positive state
  int sortTimeout;             // a bounded wait of the sort ran out
  int maxCount;                // largest neighbour count of the search
  int items;                   // work chunks of the search
  unsigned long long entries[kEntrySums];   // neighbour entries (partial sums)
  unsigned long long voteKey;  // time-step vote of FP32 limits: the smallest dtKey
  unsigned long long votes[kDtReasons];   // of FP64 limits: the smallest of each reason, as bits
  unsigned voteEst, pad;       // their running FP32 estimate
};

// Reductions ------------------------------------------------------------------
// sc->bounds: order keys of min hinv; min x,y,z; max x,y,z; (tensor H) max over
// nodes of (H^-2)_aa per axis, else 0.  NaN is passed over.
constexpr int kBoundsVals = 10;
void launchBounds(const Fields& F, long n, bool tensor, StepScratch* sc, cudaStream_t s, LaunchCounter* lc);

// Neighbour build -------------------------------------------------------------
// The first kernel of the build forms the keys, counts their digits for the
// sort and zeroes the sort's other counters and the cell ranges.
void launchCellKeys(const Fields& F, long n, Grid g, uint32_t* keys, int* vals, uint32_t* cellc, StepScratch* sc,
                    const SortPrep& prep, unsigned* ranges, long long nranges, cudaStream_t s, LaunchCounter* lc);   // resets *sc
// carriedOnly: move only the state and the derivatives the next step reads
// before recomputing them (the step rewrites every other field before it
// returns); otherwise every permuted field.  The same pass writes the cells'
// node ranges (cellStart, cellEnd; cleared before) and the FP32 mirrors
// (mirrors false: only what the search reads).
void launchPermute(const Fields& Fin, Fields Fout, const int* perm, const int* origIn, int* origOut,
                   const int* listIn, int* listOut, const uint32_t* cellIn, uint32_t* cellOut, long n,
                   bool carriedOnly, bool tensor, bool crk, bool limitedQ, Fields32 P, const Grid& g,
                   bool mirrors, const uint32_t* sortedKeys, uint32_t space, int* cellStart, int* cellEnd, const SortPrep& prep,
                   cudaStream_t s, LaunchCounter* lc);   // zeroes prep.hist for the next build
// FP32 mirror of the limited Q's DvDx (3 float4 per node).
void launchQGradient32(Fields F, float4* dvq, long n, cudaStream_t s, LaunchCounter* lc);
// Work items of the group-cooperative search: the chunks of up to `width` (8,
// 16 or 32) consecutive nodes of a cell, their first nodes, each cell's first
// chunk and the chunks' bounding boxes; the count goes to sc->items.  After a
// sort that gave up waiting (sc->sortTimeout): no items, and counts[0, n) zero.
void launchItems(const uint32_t* sortedKeys, long n, int shift, uint32_t space, const int* cellEnd, int width,
                 int nItemsBound, Grid g, bool tensor, Fields32 P, int* items, int* chunkOf, int* counts, float4* box,
                 StepScratch* sc, cudaStream_t s, LaunchCounter* lc);
// nItems: an upper bound on the item count (sizes the grid); sc->items holds
// the count itself.  The largest count and the sum of all go to *sc.
void launchNeighborsWarp(const Fields& F, Fields32 P, long n, const int* items, int nItems, StepScratch* sc,
                         int width, Grid g, const int* cellStart, const int* cellEnd, int* counts, uint32_t* nbr, int cap, double ext2, bool tensor, const float4* box, const int* chunkOf,
                         cudaStream_t s, LaunchCounter* lc);

// Sweeps ---------------------------------------------------------------------
void launchSumDensity(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                      cudaStream_t s, LaunchCounter* lc);
void launchGradh(Fields F, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp, cudaStream_t s,
                 LaunchCounter* lc);
void launchPairFP64(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                    double* pacc, cudaStream_t s, LaunchCounter* lc);   // tensor H, as launchSumDensity, launchGradh
// FP64 sweeps with isotropic H (hydro64.cu).  rec: n node records of
// nodeRecordBytes64() bytes; launchDensityDt64 takes the density sum, the dt
// vote (dOut as launchDt; dScratch 2 doubles per block) or both in one pass;
// launchEnergy64 serves every FP64 mode (vel: 4 doubles per node).
size_t nodeRecordBytes64();
void launchDensityDt64(Fields F, void* rec, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                       HydroParams hp, bool density, bool dt, double maxNperh, double* dScratch, double* dOut,
                       cudaStream_t s, LaunchCounter* lc);
void launchGradh64(Fields F, void* rec, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp, cudaStream_t s,
                   LaunchCounter* lc);
void launchPair64(Fields F, void* rec, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                  double* pacc, cudaStream_t s, LaunchCounter* lc);
void launchEnergy64(Fields F, void* vel, long n, Grid g, NeighborLists nl, const double* pacc, double dt,
                    cudaStream_t s, LaunchCounter* lc);
constexpr int kPairVariants = 2;   // autotuned variants of launchPairFP32 (isotropic H)
constexpr int kPairVariantsMax = 4;   // values sphgpu_set_pair_variant takes (any path)
constexpr int kRetuneAfter = 2;    // uses between an autotuner's first timing and its one retiming
constexpr int kPairVariantsTensor = 4;   // of its tensor-H (ASPH) path
constexpr int kPairVariantsCRK = 2;      // of the mixed CRKSPH pair kernel
// Do the variants differ at this size (else there is nothing to time)?
bool pairVariantsDiffer32(long n, const HydroParams& hp);
// Form of the isotropic pair sweep's per-node inputs (Fields32::pk, dvq).
struct PairForm {
  int on = 0;        // written by the update (and kept current by the grad-h sweep)
  float Cl = 0.f;
  int spline = 0;    // times the cubic B-spline's normalisation
  int limited = 0;   // limited Q: its DvDx too
  int full = 0;      // all nine components of it
};
PairForm pairForm32(long n, const HydroParams& hp);
// The energy sweep's half-step velocities v0 + DvDt hdt, written by the pair
// sweep (v null: not wanted): (hi, DepsDt), (lo, -) per node.
struct HalfStep {
  float4* v = nullptr;
  double hdt = 0.0;
};
// inputs: pk and dvq are already those of the state being evaluated.
void launchPairFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                    HydroParams hp, float* pacc, int variant, bool inputs, const HalfStep& half, cudaStream_t s,
                    LaunchCounter* lc);
void launchPrepareFP32(Fields F, Fields32 F32, long n, Grid g, cudaStream_t s, LaunchCounter* lc);
void launchSumDensityFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                          HydroParams hp, cudaStream_t s, LaunchCounter* lc);
void launchGradhFP32(Fields F, Fields32 F32, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                     const PairForm& pf, cudaStream_t s, LaunchCounter* lc);
void launchDtReset(StepScratch* sc, cudaStream_t s, LaunchCounter* lc);
void launchDtFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, HydroParams hp,
                  double maxNperh, StepScratch* sc, cudaStream_t s, LaunchCounter* lc);
// Mixed mode: density sum and dt vote fused in one sweep; the vote goes to
// sc->voteKey (reset: clear it first; the neighbour build has done so).
void launchDensityDtFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                         HydroParams hp, double maxNperh, StepScratch* sc, bool reset, cudaStream_t s,
                         LaunchCounter* lc);
// dt: writes per-block (value, reason) pairs then a final min into dOut[0], dOut[1] (reason as double)
void launchDt(Fields F, const int* list, long n, Grid g, NeighborLists nl, HydroParams hp,
              double maxNperh, double* dScratch, int nScratch, double* dOut,
              cudaStream_t s, LaunchCounter* lc);
// variant: slots per batch of the sweep, 0 -> 4, 1 -> 8, 2 -> 2 (the same
// result for every variant; picked by the autotuner).
constexpr int kEnergyVariants = 3;
// half: launch the half-step velocities too (else the pair sweep wrote them).
void launchCompatibleEnergyFP32(Fields F, long n, Grid g, NeighborLists nl, const float* pacc, float4* v12,
                                double dt, int variant, bool half, cudaStream_t s, LaunchCounter* lc);
// CRKSPH (crk.cu): the RK volumes (RKCorrections::preStepInitialize), the CRK
// mass density sum (CRKSPHBase::preStepInitialize), the LinearOrder
// corrections (RKCorrections::initialize) and the CRKSPH pair loop with the
// SPHSmoothingScale moments and node finalize (FP64).
void launchRKVolumes(Fields F, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp, cudaStream_t s,
                     LaunchCounter* lc);
void launchCRKDensity(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                      cudaStream_t s, LaunchCounter* lc);
void launchRKCorrections(Fields F, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp, cudaStream_t s,
                         LaunchCounter* lc);
void launchPairCRK(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                   double* pacc, cudaStream_t s, LaunchCounter* lc);
// Mixed-precision CRKSPH (crk32.cu): FP32 sweeps on the FP32 mirror, FP64
// per-node completions; the volume and correction mirrors are written too.
void launchRKVolumesFP32(Fields F, Fields32 P, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                         cudaStream_t s, LaunchCounter* lc);
// vote: take the time-step vote along (its slots reset; null: density only).
void launchCRKDensityFP32(Fields F, Fields32 P, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                          HydroParams hp, double maxNperh, StepScratch* vote, cudaStream_t s, LaunchCounter* lc);
void launchRKCorrectionsFP32(Fields F, Fields32 P, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                             cudaStream_t s, LaunchCounter* lc);
// variant: 0 one neighbour slot per loop iteration, 1 two (autotuned,
// kPairVariantsCRK; the same bits either way)
void launchPairCRKFP32(Fields F, Fields32 P, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                       HydroParams hp, float* pacc, int variant, cudaStream_t s, LaunchCounter* lc);
// ASPH: F_HINV / F_HLMAX <- smallest / largest eigenvalue of the tensor H
void launchTensorExtent(Fields F, long n, cudaStream_t s, LaunchCounter* lc);
// ASPH radialOnly: F_RAD0 <- |x|
void launchRadius0(Fields F, long n, cudaStream_t s, LaunchCounter* lc);
// mid == true: save the beginning-of-step copies (state0), then the
// timeAdvanceOnly increment with multiplier; else full update (eps
// already advanced by the compatible-energy sweep when compatible).  mirror:
// also refresh the FP32 mirrors of the new state (mixed mode), cells of grid g.
// What the update takes along where the step wants it.
struct UpdateExtras {
  PairForm pair;        // half step: the inputs of the mixed pair sweep (pair.on)
  int copyQ = 0;        // the limited Q's DvDx <- the hydro DvDx
  StepScratch* end = nullptr;   // full step: walls, state check and bounds (launchEndStep)
};
void launchUpdate(Fields F, const int* list, long n, HydroParams hp, double mult, bool mid, bool gravity,
                  const Fields32* mirror, const Grid& g, const UpdateExtras& ex, cudaStream_t s, LaunchCounter* lc);
// ASPHSmoothingScale end of step: zeroth moment, IdealH and limits of H
// (P.posh non-null: the mixed mode's FP32 extents and mirrors are refreshed).
void launchASPHEnd(Fields F, Fields32 P, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                   HydroParams hp, cudaStream_t s, LaunchCounter* lc);
// lists: device table of NodeListParams (HydroParams::lists).
void launchEOS(Fields F, const int* list, long n, const NodeListParams* lists, cudaStream_t s, LaunchCounter* lc);
// Walls, end-of-step check and the next build's bounds (sc->bad, sc->bounds).
void launchEndStep(Fields F, long n, Grid g, bool tensor, StepScratch* sc, cudaStream_t s, LaunchCounter* lc);
// out[0..7] conservation totals
void launchConservation(Fields F, long n, bool gravity, double* dScratch, int nScratch, double* dOut, cudaStream_t s,
                        LaunchCounter* lc);
// Domain-decomposition exchange rows: w field ids; mirror 1 refreshes the FP32
// density mirror, 2 the FP32 grad-h mirror of the halo nodes after a put.
struct ExchangeFields {
  int w, mirror;
  int ids[8];
};
void launchExchangeGet(Fields F, const int* inv, const int* idx, long count, ExchangeFields ef, double* out,
                       cudaStream_t s, LaunchCounter* lc);
void launchExchangePut(Fields F, Fields32 P, const int* inv, long nOwn, long count, ExchangeFields ef,
                       const double* in, cudaStream_t s, LaunchCounter* lc);
// caller-order transfers through a device staging buffer (stride doubles per node)
void launchGatherOut(Fields F, const int* orig, double* stage, int first, int ncomp, int stride, long n,
                     cudaStream_t s, LaunchCounter* lc);
void launchScatterIn(Fields F, const int* orig, const double* stage, int first, int ncomp, int stride, long n,
                     cudaStream_t s, LaunchCounter* lc);
void launchGatherOutH(Fields F, const int* orig, double* stage, int field, long n, cudaStream_t s, LaunchCounter* lc);
// caller-order transfers on pinned host arrays addressed in place (inv: the
// internal index of each caller index)
void launchInverseOrder(const int* orig, int* inv, long n, cudaStream_t s, LaunchCounter* lc);
// The state fields of one hand-over between the device and mapped host arrays
// in caller order, in one launch.
struct HostBatch {
  int count = 0, maxStride = 0;
  struct Item {
    double* host;
    int first, ncomp, stride, isoH;
  } it[6];
  void add(const void* host, int first, int ncomp, int stride, bool isoH) {
    it[count++] = Item{static_cast<double*>(const_cast<void*>(host)), first, ncomp, stride, isoH ? 1 : 0};
    if (stride > maxStride) maxStride = stride;
  }
};
void launchScatterInHost(Fields F, const int* inv, const HostBatch& batch, long n, cudaStream_t s, LaunchCounter* lc);
void launchGatherOutHost(Fields F, const int* inv, const HostBatch& batch, long n, cudaStream_t s, LaunchCounter* lc);
void launchCountsOut(const int* counts, const int* orig, double* stage, long n, cudaStream_t s, LaunchCounter* lc);

// Gravity (gravity.cu) ---------------------------------------------------------
struct GravityWork;
GravityWork* gravityCreate();
void gravityDestroy(GravityWork* w);
// Build the octree of the current positions and walk it; writes F_GRAV_*,
// F_POT (already multiplied by G) and returns dtMinAcc via dOut[0], extra
// energy via dOut[1].
// mixed: FP32 interaction terms on double-float coordinates with compensated
// accumulation (decisions as in FP64); otherwise FP64 throughout.
int gravityEvaluate(GravityWork* w, Fields F, long n, double G, double softening, double opening, bool mixed,
                    double* dOut,
                    cudaStream_t s, LaunchCounter* lc, char* err, int errlen);

}  // namespace sph
