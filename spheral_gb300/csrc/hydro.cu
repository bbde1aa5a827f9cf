// SPH hydro kernels of libsphgpu (sm_103a): cell-list neighbour build,
// density sum, grad-h correction, the FP64 pair loop with its per-node
// finalisation and smoothing-scale update, the time-step vote, the
// compatible-energy sweep and the CheapSynchronousRK2 state updates.
//
// Formulation.  The reference walks an unordered pair list and scatters into
// both nodes through thread-private copies of 13 FieldLists
// (src/SPH/SPH.cc:271-475).  Here every kernel is a gather: one thread owns
// node i and walks i's neighbour list, so each unordered pair is evaluated
// twice (once per side) with no atomics and a fixed summation order.  Ghost
// nodes of periodic and reflecting boundaries are implicit: a neighbour
// entry carries a 6-bit image code and the neighbour's coordinates are mapped
// with the reference's own plane formula (imageCoord).
#include "device.cuh"
#include "packed32.cuh"
#include <algorithm>
#include <climits>

namespace sph {
namespace {
using namespace dev;

//------------------------------------------------------------------------------
// Bounds: min hinv, bounding box (for open axes) and, for tensor H, the
// largest half-width per axis of the unit ellipsoids {r : |H r| <= 1}, i.e.
// sqrt((H^-2)_aa) = |row a of H^-1| (the cell edge per axis).
//------------------------------------------------------------------------------
// A signed integer with the order of the double x (for non-NaN x; -0 sorts
// just below +0, which only sends a node at a wall to the exact test).
__device__ __forceinline__ long long orderKey(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
// Bit tests of the end-of-step check (integer pipe).
__device__ __forceinline__ bool finiteBits(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}
__device__ __forceinline__ bool positiveBits(double x) {   // x > 0 and finite
  const long long b = __double_as_longlong(x);
  return b > 0 && b < 0x7ff0000000000000LL;
}

// Running bounds of a thread's nodes on order keys (the FP64 pipe, which
// FP64 comparisons take, is narrow); NaN is passed over.
struct NodeBounds {
  long long mn[4] = {LLONG_MAX, LLONG_MAX, LLONG_MAX, LLONG_MAX};
  long long mx[6] = {LLONG_MIN, LLONG_MIN, LLONG_MIN, 0, 0, 0};
  static __device__ bool isNaN(double x) {
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ULL;
  }
  __device__ void add(double a, const double* p) {
    if (!isNaN(a)) mn[0] = min(mn[0], orderKey(a));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (isNaN(p[k])) continue;
      const long long o = orderKey(p[k]);
      mn[1 + k] = min(mn[1 + k], o);
      mx[k] = max(mx[k], o);
    }
  }
  __device__ void addTensor(const Sym& H) {   // squares: the host takes the roots of the largest
    const Sym w = symInverse(H);
    const double e[3] = {w.xx * w.xx + w.xy * w.xy + w.xz * w.xz, w.xy * w.xy + w.yy * w.yy + w.yz * w.yz,
                         w.xz * w.xz + w.yz * w.yz + w.zz * w.zz};
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (!isNaN(e[k])) mx[3 + k] = max(mx[3 + k], orderKey(e[k]));
  }
};
// Block minima and maxima into sc->bounds.  Every thread of a 256-thread block
// calls it; a bound is only written where it moves.
__device__ __forceinline__ void mergeBounds(const NodeBounds& b, bool tensor, StepScratch* __restrict__ sc) {
  __shared__ long long sm[8][10];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 10; ++k) {
    if (k >= 7 && !tensor) break;
    long long v = k < 4 ? b.mn[k] : b.mx[k - 4];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long w = __shfl_xor_sync(0xffffffffu, v, o);
      v = k < 4 ? min(v, w) : max(v, w);
    }
    if (lane == 0) sm[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < (tensor ? 10 : 7)) {
    const int k = threadIdx.x;
    long long v = sm[0][k];
    for (int w = 1; w < 8; ++w) v = k < 4 ? min(v, sm[w][k]) : max(v, sm[w][k]);
    const long long seen = *(volatile long long*)&sc->bounds[k];
    if (k < 4) { if (v < seen) atomicMin(&sc->bounds[k], v); }
    else { if (v > seen) atomicMax(&sc->bounds[k], v); }
  }
}
__global__ void resetScratchKernel(StepScratch* __restrict__ sc) { resetScratch(sc); }
__global__ void __launch_bounds__(256) boundsKernel(Fields F, long n, int tensor, StepScratch* __restrict__ sc) {
  NodeBounds b;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double p[3] = {F.f[F_X][i], F.f[F_Y][i], F.f[F_Z][i]};
    b.add(F.f[F_HINV][i], p);
    if (tensor) b.addTensor(loadSym(F, F_HT_XX, i));
  }
  mergeBounds(b, tensor != 0, sc);
}

//------------------------------------------------------------------------------
// Neighbour build.
//------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) cellKeyKernel(Fields F, long n, Grid g, uint32_t* __restrict__ keys,
                                                     int* __restrict__ vals, uint32_t* __restrict__ cellc,
                                                     StepScratch* __restrict__ sc, SortPrep prep,
                                                     unsigned* __restrict__ ranges, long long nranges) {
  __shared__ unsigned h[4][256];
  for (int d = 0; d < prep.digits; ++d) h[d][threadIdx.x] = 0u;
  __syncthreads();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
  if (t == 0) resetScratch(sc);
  for (long long w = t; w < prep.nclear; w += nt) prep.clear[w] = 0u;
  for (long long w = t; w < nranges; w += nt) ranges[w] = 0u;
  const int lane = threadIdx.x & 31;
  for (long b = t - lane; b < n; b += nt) {   // whole warps
  const long i = b + lane < n ? b + lane : n - 1;
  const bool live = b + lane < n;
  const double p[3] = {F.f[F_X][i], F.f[F_Y][i], F.f[F_Z][i]};
  uint32_t c[3], f[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // position in half-cells, rounded down by the conversion itself: three
    // FP64-pipe instructions per axis (no division; the FP64 pipe is the
    // narrow one).  A node within rounding of a cell face may land in either
    // cell: the cells exceed the kernel support by a relative 1e-9, far
    // above that rounding.  NaN converts to the most negative value and is
    // clamped into cell 0.
    const long long hc = __double2ll_rd(__dmul_rn(__dsub_rn(p[a], g.lo[a]), g.inv2[a]));
    long long ci = hc >> 1;
    const bool clamped = ci < 0 || ci >= g.nc[a];
    ci = ci < 0 ? 0 : (ci >= g.nc[a] ? g.nc[a] - 1 : ci);
    c[a] = (uint32_t)ci;
    // the half of the cell the node is in (order within the cell only)
    f[a] = 2u * c[a] + ((!clamped && (hc & 1)) ? 1u : 0u);
  }
  // With a sub-cell level the key is the Morton key of the half-cells, whose
  // top bits are the cell's Morton key: nodes stay grouped by cell and within
  // a cell they are ordered by octant, so consecutive nodes of a cell (a work
  // chunk or a candidate batch of the neighbour search) sit close together.
  const uint32_t key = g.subShift ? cellKey(g, f[0], f[1], f[2], 1) : cellKey(g, c[0], c[1], c[2], 0);
  if (live) {
    keys[i] = key;
    vals[i] = (int)i;
    cellc[i] = c[0] | (c[1] << 10) | (c[2] << 20);
  }
  for (int d = 0; d < prep.digits; ++d) {
    const unsigned digit = live ? (key >> (8 * d)) & 0xffu : 256u;
    int all;   // the high digits of a warp are mostly equal
    __match_all_sync(0xffffffffu, digit, &all);
    if (all) {
      if (lane == 0) atomicAdd(&h[d][digit], 32u);
    } else if (live) {
      atomicAdd(&h[d][digit], 1u);
    }
  }
  }
  __syncthreads();
  for (int d = 0; d < prep.digits; ++d)
    if (const unsigned c = h[d][threadIdx.x]) atomicAdd(&prep.hist[d * 256 + threadIdx.x], c);
}

// Gather of the carried fields into the new order, with what the same pass can
// take along: the cells' node ranges (from the sorted keys) and the FP32
// mirrors of the new order.  Indices and keys of a sort that gave up waiting
// stay in range here, and itemsKernel passes no lists on; the host then fails
// the call on the sort's flag.
__global__ void permuteKernel(Fields Fin, Fields Fout, const int* __restrict__ perm, const int* __restrict__ origIn,
                              int* __restrict__ origOut, const int* __restrict__ listIn, int* __restrict__ listOut,
                              const uint32_t* __restrict__ cellIn, uint32_t* __restrict__ cellOut, long n,
                              FieldRanges sel, Fields32 P, Grid g, int mirrors, const uint32_t* __restrict__ keys,
                              uint32_t space, int* __restrict__ cellStart, int* __restrict__ cellEnd, SortPrep prep) {
  if (blockIdx.x == 0 && blockIdx.y == 0)   // the sort is done with them
    for (int w = threadIdx.x; w < 256 * prep.digits; w += blockDim.x) prep.hist[w] = 0u;
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int p = (int)min((unsigned)perm[k], (unsigned)(n - 1));
  // gridDim.y > 1: the last row of blocks takes the rest, the others a share of
  // the fields each
  const int rows = gridDim.y > 1 ? gridDim.y - 1 : 1, row = blockIdx.y;
  if (row < rows)
    for (int r = 0; r < sel.n; ++r) {
      const int len = sel.last[r] - sel.first[r];
      const int f1 = sel.first[r] + len * (row + 1) / rows;
#pragma unroll 8
      for (int f = sel.first[r] + len * row / rows; f < f1; ++f) Fout.f[f][k] = Fin.f[f][p];
    }
  if (row != (int)gridDim.y - 1) return;
  origOut[k] = origIn[p];
  listOut[k] = listIn[p];
  const uint32_t cell = cellIn[p];
  cellOut[k] = cell;
  const uint32_t key = keys[k] >> g.subShift;
  if (key < space) {
    if (k == 0 || (keys[k - 1] >> g.subShift) != key) cellStart[key] = (int)k;
    if (k == n - 1 || (keys[k + 1] >> g.subShift) != key) cellEnd[key] = (int)(k + 1);
  }
  writeMirrors(Fin, p, P, k, cell, g, mirrors != 0);
}

// Pair criterion of ConnectivityMap::computeConnectivity
// (src/Neighbor/ConnectivityMap.cc:917-929): (Hi rij)^2 <= ext^2 or
// (Hj rij)^2 <= ext^2, self excluded.  An FP32 test on cell-relative
// positions settles every candidate outside a narrow band around the
// threshold; candidates inside the band get the exact FP64 test with the
// reference's operation order, so the neighbour sets are exact.
//
// Candidate cells are visited in a fixed order (dz, dy, dx from -1 to 1) and
// nodes within a cell in sorted order, so every list has a reproducible order.
// WRITE false: count only; true: count and write the warp-interleaved lists
// (slots beyond cap are counted, not written).

// Relative half-width of the FP32 band around |H r|^2 = ext^2 for a node with
// eigenvalues in [lmin, lmax].  Each FP32 separation component carries at
// most ~10 u C of rounding (C the largest cell edge, u = 2^-24), and the
// products and sums of H r add ~4 u |H| |r| per component; near the threshold
// (|H r| ~ ext, |r| <= ext / lmin) |H r| is then off by at most
// 30 u C lmax + 12 u ext lmax / lmin and its square by
// ext^2 u (60 C lmax / ext + 24 lmax / lmin + 3).  The band is four times that.
__device__ __forceinline__ float tensorBand(float lmax, float lmin, const Grid& g) {
  const float u = 5.9604645e-8f;
  const float C = fmaxf(g.cellf[0], fmaxf(g.cellf[1], g.cellf[2]));
  return 4.0f * u * (60.0f * C * lmax / sqrtf(g.ext2f) + 24.0f * lmax / lmin + 3.0f);
}

// The exact FP64 tensor criterion |H_i r|^2 <= ext^2 or |H_j r|^2 <= ext^2
// (H_j through the image).  Out of line: it runs for few candidates, and
// inlined its FP64 tensors would set the register count of the whole search.
__device__ __noinline__ bool exactTensorCriterion(const Fields& F, const Grid& g, long i, int j, int code, double qx,
                                                  double qy, double qz, double ext2) {
  Sym Hj = loadSym(F, F_HT_XX, j);
  imageSym(g, code, Hj);
  return eta2ExactSym(loadSym(F, F_HT_XX, i), qx, qy, qz) <= ext2 || eta2ExactSym(Hj, qx, qy, qz) <= ext2;
}

//------------------------------------------------------------------------------
// The search.  A warp (CW = 1) or the block's four warps (CW = 4) own one work
// item: up to 32 consecutive nodes of a cell, one per lane, so the 27 candidate
// cells, their offset codes and mirror flags are uniform across it.
//
//  1. The chunks of the 27 candidate cells (in cell order, up to kTile at a
//     time) are listed and culled lane-parallel: a chunk whose bounding box is
//     farther from the item's box than the item's largest FP32 band edge
//     allows holds no neighbour of any lane.
//  2. The candidates of the surviving chunks, one per lane, are culled against
//     the item's box in the same way, and the rest are staged densely in the
//     item's frame (a candidate at q in its cell sits at q - o there).
//  3. Every 32 staged candidates (a batch) are tested two per packed FP32
//     operation; the lane's hits up to the top of its guard band form a 32-bit
//     mask.  A lane whose largest hit lies inside the band forms the mask of
//     that batch again with the exact FP64 criterion.
//  4. The masks are written out as list entries, the q-th hit of every lane in
//     the same iteration, so a row of the warp-interleaved list is one 128-byte
//     store.
// CW = 4: the warps take a quarter of a tile's chunks each, in order.
//
// Every list is in candidate order, whatever the item width and CW.
//
// TENSOR (ASPH): h^-1 of the FP32 mirror is the smallest eigenvalue of H, which
// bounds |H r| from below for the culling, as does a diagonal bound of H^2
// (tensorDiagonal); the test takes |H_i r|^2 and |H_j r|^2 from the tensor
// mirror, each with its node's band (tensorBand), and a batch that may hold a
// candidate inside a band repeats its mask with the exact FP64 tensor criterion
// for those.
//
// What bounds it: instruction issue.  Testing and storing candidate by
// candidate took ~36 warp instructions per candidate of a group; the masks take
// ~9 (TENSOR ~20, the FMA pipe, which a packed operation fills for two) for the
// test and ~3 for the writing, and the culling of single candidates ~1.  With
// the last, 2.1 M nodes of a Kelvin-Helmholtz slab (cells sized by the light
// layer's h): 1704 -> 1345 us; 303,912 ASPH nodes: 820 -> 600 us.
//------------------------------------------------------------------------------
constexpr int kTile = 32;   // batches listed at a time
// min(a, |b|, |c|) for a >= 0
__device__ __forceinline__ float minAbs3(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The 27 candidate cells of home cell hc, one per lane (lanes 0..26): node
// range, first work chunk, offset code and offset.
struct CandidateCell {
  int start, end, chunk, dcode;
  float ox, oy, oz;
};
__device__ __forceinline__ CandidateCell candidateCell(int t, const int* hc, const Grid& g,
                                                       const int* __restrict__ cellStart,
                                                       const int* __restrict__ cellEnd,
                                                       const int* __restrict__ chunkOf) {
  CandidateCell r{0, 0, 0, 0, 0.f, 0.f, 0.f};
  const int d[3] = {t % 3, (t / 3) % 3, t / 9};   // 0, 1, 2 for -1, 0, +1
  int cell[3];
  bool ok = t < 27;
  float o[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int nn = hc[a] + d[a] - 1;
    if (nn < 0) {
      if (g.kindLo[a] == AXIS_PERIODIC) nn = g.nc[a] - 1;
      else if (g.kindLo[a] == AXIS_REFLECT) nn = 0;
      else ok = false;
    } else if (nn >= g.nc[a]) {
      if (g.kindHi[a] == AXIS_PERIODIC) nn = 0;
      else if (g.kindHi[a] == AXIS_REFLECT) nn = g.nc[a] - 1;
      else ok = false;
    }
    cell[a] = nn;
    r.dcode |= (d[a] == 0 ? 1 : (d[a] == 2 ? 2 : 0)) << (2 * a);
    o[a] = d[a] == 0 ? g.cellf[a] : (d[a] == 2 ? -g.cellf[a] : 0.0f);
  }
  r.ox = o[0]; r.oy = o[1]; r.oz = o[2];
  if (ok) {
    const uint32_t key = cellKey(g, (uint32_t)cell[0], (uint32_t)cell[1], (uint32_t)cell[2], 0);
    r.start = cellStart[key];
    r.end = cellEnd[key];
    if (r.start < r.end) r.chunk = chunkOf[r.start];
  }
  return r;
}

template <bool WRITE, int CW, bool TENSOR>
__global__ void __launch_bounds__(128, TENSOR ? 4 : 6) neighborMaskKernel(Fields F, Fields32 P, const int* __restrict__ items,
                                                          int nItems, int width, Grid g,
                                                          const int* __restrict__ cellStart,
                                                          const int* __restrict__ cellEnd, int* __restrict__ counts,
                                                          uint32_t* __restrict__ nbr, double ext2, float bandA,
                                                          float bandB, int cap, StepScratch* __restrict__ sc,
                                                          const float4* __restrict__ box,
                                                          const float4* __restrict__ tbox,
                                                          const int* __restrict__ chunkOf) {
  constexpr int G = 4 / CW;                  // items per block
  constexpr int UNROLL = TENSOR ? 1 : 8;     // 35 loads per iteration with TENSOR
  constexpr int NB = CW == 4 ? 8 : 16;       // ring of batches whose masks wait for the writing
  static_assert(CW == 1 || CW == 4, "one warp or the block's four per item");
  static_assert(kTile <= 32, "a tile's chunks are listed one per lane");
  // CW = 4 writes after every tile: a warp stages the candidates of at most
  // ceil(kTile / 4) chunks of up to 32.  CW = 1 writes when NB - 1 batches wait,
  // with one more being staged.  `nonempty` has a bit per waiting batch.
  static_assert(CW == 1 || (kTile + 3) / 4 <= NB, "the ring holds a warp's share of a tile");
  static_assert(NB >= 3 && NB <= 32, "the ring holds the waiting batches and the two being staged");
  // per warp, 64 slots: the staged candidates' -x, -y, -z and (h^-1)^2; TENSOR:
  // H (xx xy xz yy yz zz) as seen through the mirrors, minus the band's top and
  // its bottom
  __shared__ __align__(16) float stage[4][TENSOR ? 11 : 4][64];
  __shared__ uint32_t masks[4][NB][32], ids[4][NB][32];   // hits of each lane; list entries of the slots
  __shared__ int2 desc[G][kTile];            // kept chunks: entry of the first node, size
  __shared__ float4 offs[G][kTile];          // and the cell offset
  __shared__ float4 diag[TENSOR ? G : 1][TENSOR ? kTile : 1];   // and the diagonal bound with the item's
  __shared__ int part[CW == 4 ? 4 : 1][32];  // CW = 4: hits per lane of each warp's chunks
  __shared__ int keptCount[G];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = CW == 4 ? 0 : warp, sub = CW == 4 ? warp : 0;
  const int item = blockIdx.x * G + grp;
  if (item >= min(nItems, sc->items)) return;   // uniform over the item's warps
  auto groupSync = [] {
    if (CW == 4) __syncthreads();
    else __syncwarp();
  };
  const int k0 = items[item];
  int hc[3];
  unpackCell(P.cell[k0], hc);
  const CandidateCell cc = candidateCell(lane, hc, g, cellStart, cellEnd, chunkOf);
  const int k1 = min(k0 + width, __shfl_sync(0xffffffffu, cc.end, 13));   // cell 13 is the home cell
  const long i = k0 + lane;
  const bool active = i < k1;
  const float4 pi = active ? P.posh[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float ai2 = pi.w * pi.w;
  const float e2t = g.ext2f;
  // a band's bottom and top; a candidate whose e2 is farther than the returned
  // gap from the top is outside the band on one side or the other (with room
  // for the rounding of the difference)
  auto bandOf = [&](float d, float& lo, float& hi) {
    lo = d < 0.5f ? e2t * (1.0f - d) : -1.0f;
    hi = d < 0.5f ? e2t * (1.0f + d) : FLT_MAX;
    return d < 0.5f ? 1.01f * (hi - lo) + 4.0e-7f * hi : FLT_MAX;
  };
  float bandLo = 0.f, bandHi = 0.f, bandGap = 0.f;
  f32x2 hxx = 0, hxy = 0, hxz = 0, hyy = 0, hyz = 0, hzz = 0;
  if (!TENSOR) {
    bandGap = bandOf(__fmaf_rn(bandA, pi.w, bandB), bandLo, bandHi);
  } else if (active) {
    const float4 h0 = P.hten[i], h1 = P.hten[P.stride + i];
    bandGap = bandOf(tensorBand(h1.w, pi.w, g), bandLo, bandHi);
    hxx = pack2(h0.x, h0.x); hxy = pack2(h0.y, h0.y); hxz = pack2(h0.z, h0.z);
    hyy = pack2(h0.w, h0.w); hyz = pack2(h1.x, h1.x); hzz = pack2(h1.y, h1.y);
  }
  const f32x2 nhi2 = pack2(-bandHi, -bandHi);
  const f32x2 px2 = pack2(pi.x, pi.x), py2 = pack2(pi.y, pi.y), pz2 = pack2(pi.z, pi.z);
  const uint32_t mm = mirrorMask(g, hc);
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 gLo = box[2 * item], gHi = box[2 * item + 1];
  const float delMax = __fmaf_rn(bandA, gHi.w, bandB);
  const bool cull = delMax < 0.5f;
  const float cullThr = e2t * (1.0f + delMax) * 1.0001f;
  const float4 gT = TENSOR ? tbox[item] : make_float4(0.f, 0.f, 0.f, 0.f);
  // chunks of each candidate cell, and how many come before them
  const int nb = (cc.end - cc.start + width - 1) / width;
  int before = nb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += y;
  }
  const int chunks = __shfl_sync(0xffffffffu, before, 31);
  before -= nb;

  int staged = 0, tested = 0;   // candidates staged, batches tested by this warp
  int window = 0;               // first batch whose masks are not written yet
  int selfPos = -1;             // where node i itself was staged
  uint32_t nonempty = 0u;       // batches from `window` that hold hits of this lane
  int hits = 0;                 // and their number
  int cnt = 0;                  // this lane's hits so far

  // Tests the next batch, of nval candidates.
  auto test = [&](int nval) {
    __syncwarp();
    const int half = (tested & 1) * 32, ring = tested % NB;
    float gap = bandGap;   // the widest band of the batch and this lane
    if (TENSOR) {
      const float jHi = -stage[warp][9][half + lane], jLo = stage[warp][10][half + lane];
      const float jGap = jHi < FLT_MAX ? 1.01f * (jHi - jLo) + 4.0e-7f * jHi : FLT_MAX;
      // positive floats order as integers
      gap = fmaxf(gap, __uint_as_float(__reduce_max_sync(0xffffffffu, lane < nval ? __float_as_uint(jGap) : 0u)));
    }
    // e2 - top of the band: its sign bits, shifted in one by one, are the mask
    // (bit order reversed), and its smallest magnitude tells whether a candidate
    // may lie inside the band
    uint32_t mask = 0u;
    float near = FLT_MAX;
#pragma unroll UNROLL
    for (int u = 0; u < 32; u += 4) {
      if (u >= nval) { mask <<= 32 - u; break; }   // uniform
      auto at = [&](int c) { return *reinterpret_cast<const ulonglong2*>(&stage[warp][c][half + u]); };
      const ulonglong2 X = at(0), Y = at(1), Z = at(2);
      const f32x2 rx0 = add2(px2, X.x), ry0 = add2(py2, Y.x), rz0 = add2(pz2, Z.x);
      const f32x2 rx1 = add2(px2, X.y), ry1 = add2(py2, Y.y), rz1 = add2(pz2, Z.y);
      float e[4];
      if (TENSOR) {
        const ulonglong2 XX = at(3), XY = at(4), XZ = at(5), YY = at(6), YZ = at(7), ZZ = at(8), NH = at(9);
        auto top = [](f32x2 xx, f32x2 xy, f32x2 xz, f32x2 yy, f32x2 yz, f32x2 zz, f32x2 x, f32x2 y, f32x2 z,
                      f32x2 nh) {   // |H r|^2 - top
          const f32x2 ex = fma2(xz, z, fma2(xy, y, mul2(xx, x)));
          const f32x2 ey = fma2(yz, z, fma2(yy, y, mul2(xy, x)));
          const f32x2 ez = fma2(zz, z, fma2(yz, y, mul2(xz, x)));
          return fma2(ez, ez, fma2(ey, ey, fma2(ex, ex, nh)));
        };
        float d[4];
        unpack2(top(hxx, hxy, hxz, hyy, hyz, hzz, rx0, ry0, rz0, nhi2), e[0], e[1]);
        unpack2(top(XX.x, XY.x, XZ.x, YY.x, YZ.x, ZZ.x, rx0, ry0, rz0, NH.x), d[0], d[1]);
        unpack2(top(hxx, hxy, hxz, hyy, hyz, hzz, rx1, ry1, rz1, nhi2), e[2], e[3]);
        unpack2(top(XX.y, XY.y, XZ.y, YY.y, YZ.y, ZZ.y, rx1, ry1, rz1, NH.y), d[2], d[3]);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          mask = __funnelshift_l(__float_as_uint(e[v]) | __float_as_uint(d[v]), mask, 1);
          near = minAbs3(near, e[v], d[v]);
        }
      } else {
        const float4 A = *reinterpret_cast<const float4*>(&stage[warp][3][half + u]);
        const f32x2 s0 = fma2(fma2(rz0, rz0, fma2(ry0, ry0, mul2(rx0, rx0))), pack2(fminf(ai2, A.x), fminf(ai2, A.y)), nhi2);
        const f32x2 s1 = fma2(fma2(rz1, rz1, fma2(ry1, ry1, mul2(rx1, rx1))), pack2(fminf(ai2, A.z), fminf(ai2, A.w)), nhi2);
        unpack2(s0, e[0], e[1]);
        unpack2(s1, e[2], e[3]);
#pragma unroll
        for (int v = 0; v < 4; ++v) mask = __funnelshift_l(__float_as_uint(e[v]), mask, 1);
        near = minAbs3(minAbs3(near, e[0], e[1]), e[2], e[3]);
      }
    }
    mask = __brev(mask);
    if (nval < 32) mask &= (1u << nval) - 1u;
    if (active && near <= gap) {   // guard band: this lane's mask again, band candidates by the exact FP64 criterion
      mask = 0u;
      for (int u = 0; u < nval; ++u) {
        const float* st = &stage[warp][0][half + u];
        const float rx = __fadd_rn(pi.x, st[0]), ry = __fadd_rn(pi.y, st[64]), rz = __fadd_rn(pi.z, st[128]);
        bool in;
        if (TENSOR) {
          auto lo = [](f32x2 v) { return __uint_as_float((unsigned)v); };
          const float e2i = eta2Sym32(make_float4(lo(hxx), lo(hxy), lo(hxz), lo(hyy)),
                                      make_float4(lo(hyz), lo(hzz), 0.f, 0.f), rx, ry, rz);
          const float e2j = eta2Sym32(make_float4(st[192], st[256], st[320], st[384]),
                                      make_float4(st[448], st[512], 0.f, 0.f), rx, ry, rz);
          in = (e2i <= bandLo) | (e2j <= st[640]);
          if (!in && (e2i >= bandHi) & (e2j >= -st[576])) continue;
        } else {
          const float e2 = fminf(ai2, st[192]) * (rx * rx + ry * ry + rz * rz);
          if (e2 > bandHi) continue;
          in = e2 < bandLo;
        }
        if (!in) {
          const uint32_t ent = ids[warp][ring][u];
          const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
          double xjd = F.f[F_X][j], yjd = F.f[F_Y][j], zjd = F.f[F_Z][j];
          imagePos(g, code, xjd, yjd, zjd);
          const double qx = __dsub_rn(F.f[F_X][i], xjd), qy = __dsub_rn(F.f[F_Y][i], yjd),
                       qz = __dsub_rn(F.f[F_Z][i], zjd);
          in = TENSOR ? exactTensorCriterion(F, g, i, j, code, qx, qy, qz, ext2)
                      : eta2Exact(F.f[F_HINV][i], qx, qy, qz) <= ext2 || eta2Exact(F.f[F_HINV][j], qx, qy, qz) <= ext2;
        }
        if (in) mask |= 1u << u;
      }
    }
    const int own = selfPos - 32 * tested;
    if (own >= 0 && own < 32) mask &= ~(1u << own);
    if (!active) mask = 0u;
    masks[warp][ring][lane] = mask;
    if (mask) nonempty |= 1u << (tested - window);
    hits += __popc(mask);
    ++tested;
    __syncwarp();
  };
  // Writes the hits of the window's batches from slot `at` of the lane's list.
  auto writeOut = [&](int at) {
    if (WRITE) {
      uint32_t* out = nbr + nbSlot(active ? i : k0, 0, cap) + (size_t)at * 32;
      const int stored = min(hits, cap - at);
      const int most = __reduce_max_sync(0xffffffffu, stored);
      uint32_t m = 0u;
      int ring = 0;
      for (int h = 0; h < most; ++h, out += 32)
        if (h < stored) {
          if (m == 0u) {
            const int b = __ffs(nonempty) - 1;
            nonempty &= nonempty - 1u;
            ring = (window + b) % NB;
            m = masks[warp][ring][lane];
          }
          *out = ids[warp][ring][__ffs(m) - 1];
          m &= m - 1u;
        }
      __syncwarp();
    }
    window = tested;
    nonempty = 0u;
    hits = 0;
  };

  for (int tile = 0; tile < chunks; tile += kTile) {
    const int inTile = min(kTile, chunks - tile);
    if (sub == 0) {
      // list and cull the tile's chunks, one per lane
      const int b = tile + lane;
      // the cell of chunk b: the last one that starts at or before it
      int t = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1) {
        const int c = __shfl_sync(0xffffffffu, before, min(t + st, 26));
        if (t + st <= 26 && c <= b) t += st;
      }
      const int cs = __shfl_sync(0xffffffffu, cc.start, t), ce = __shfl_sync(0xffffffffu, cc.end, t);
      const int cb = b - __shfl_sync(0xffffffffu, before, t);
      const int chunk = __shfl_sync(0xffffffffu, cc.chunk, t) + cb;
      const int dcode = __shfl_sync(0xffffffffu, cc.dcode, t);
      const float ox = __shfl_sync(0xffffffffu, cc.ox, t), oy = __shfl_sync(0xffffffffu, cc.oy, t);
      const float oz = __shfl_sync(0xffffffffu, cc.oz, t);
      bool keep = lane < inTile;
      float4 bT = make_float4(0.f, 0.f, 0.f, 0.f);
      if (TENSOR && keep) {
        // x, y, z: the bound for both; w: the squared extent it is held against
        bT = tbox[chunk];
        const float band = fmaxf(gT.w, bT.w);
        bT = make_float4(fminf(gT.x, bT.x), fminf(gT.y, bT.y), fminf(gT.z, bT.z),
                         band < 0.5f ? e2t * (1.0f + band) * 1.0001f : FLT_MAX);
      }
      if (keep && cull) {
        // the chunk's box in the item's frame
        const float4 bLo = box[2 * chunk], bHi = box[2 * chunk + 1];
        const uint32_t mir = (uint32_t)dcode & mm;
        float lx = bLo.x, hx = bHi.x, ly = bLo.y, hy = bHi.y, lz = bLo.z, hz = bHi.z;
        if (mir & 3u) { lx = cx - bHi.x; hx = cx - bLo.x; }
        if (mir & 12u) { ly = cy - bHi.y; hy = cy - bLo.y; }
        if (mir & 48u) { lz = cz - bHi.z; hz = cz - bLo.z; }
        const float gx = fmaxf(0.0f, fmaxf((lx - ox) - gHi.x, gLo.x - (hx - ox)));
        const float gy = fmaxf(0.0f, fmaxf((ly - oy) - gHi.y, gLo.y - (hy - oy)));
        const float gz = fmaxf(0.0f, fmaxf((lz - oz) - gHi.z, gLo.z - (hz - oz)));
        const float am = fminf(gLo.w, bLo.w);
        keep = !((am * am) * (gx * gx + gy * gy + gz * gz) > cullThr) &&
               !(TENSOR && bT.x * (gx * gx) + bT.y * (gy * gy) + bT.z * (gz * gz) > bT.w);
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int first = cs + cb * width;
        const int at = __popc(m & ((1u << lane) - 1u));
        desc[grp][at] = make_int2(first | (int)((uint32_t)dcode << kIndexBits), min(width, ce - first));
        offs[grp][at] = make_float4(ox, oy, oz, 0.0f);
        if (TENSOR) diag[grp][at] = bT;
      }
      if (lane == 0) keptCount[grp] = __popc(m);
    }
    groupSync();
    const int kept = keptCount[grp];
    const int b0 = CW == 4 ? sub * kept / 4 : 0, b1 = CW == 4 ? (sub + 1) * kept / 4 : kept;
    float4 qn = make_float4(0.f, 0.f, 0.f, 0.f), hn0 = qn, hn1 = qn;
    auto ahead = [&](int b) {   // candidate `lane` of chunk b
      const int2 d = desc[grp][b];
      if (lane >= d.y) return;
      const int j = (d.x & kIndexMask) + lane;
      qn = P.posh[j];
      if (TENSOR) { hn0 = P.hten[j]; hn1 = P.hten[P.stride + j]; }
    };
    if (b0 < b1) ahead(b0);
    for (int b = b0; b < b1; ++b) {
      const int2 ds = desc[grp][b];
      const int first = ds.x & kIndexMask, nval = ds.y, dcode = (int)((uint32_t)ds.x >> kIndexBits);
      float4 q = qn;
      const float4 qh0 = hn0, qh1 = hn1;
      if (b + 1 < b1) ahead(b + 1);
      const uint32_t mir = (uint32_t)dcode & mm;
      if (mir) {
        if (mir & 3u) q.x = cx - q.x;
        if (mir & 12u) q.y = cy - q.y;
        if (mir & 48u) q.z = cz - q.z;
      }
      const float4 o = offs[grp][b];
      const float nx = __fsub_rn(o.x, q.x), ny = __fsub_rn(o.y, q.y), nz = __fsub_rn(o.z, q.z);
      bool keep = lane < nval;
      if (keep && cull) {
        const float gx = fmaxf(0.0f, fmaxf(-nx - gHi.x, gLo.x + nx));
        const float gy = fmaxf(0.0f, fmaxf(-ny - gHi.y, gLo.y + ny));
        const float gz = fmaxf(0.0f, fmaxf(-nz - gHi.z, gLo.z + nz));
        const float am = fminf(gLo.w, q.w);
        keep = !((am * am) * (gx * gx + gy * gy + gz * gz) > cullThr);
        if (TENSOR) {
          const float4 bT = diag[grp][b];
          keep &= !(bT.x * (gx * gx) + bT.y * (gy * gy) + bT.z * (gz * gz) > bT.w);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (dcode == 0 && first == k0) selfPos = staged + lane;   // the item's own chunk, none of it culled
      if (keep) {
        const int pos = staged + __popc(m & ((1u << lane) - 1u));
        float* st = &stage[warp][0][pos & 63];
        st[0] = nx;
        st[64] = ny;
        st[128] = nz;
        if (TENSOR) {
          float jLo, jHi;
          bandOf(tensorBand(qh1.w, q.w, g), jLo, jHi);
          const float sx = (mir & 3u) ? -1.f : 1.f, sy = (mir & 12u) ? -1.f : 1.f, sz = (mir & 48u) ? -1.f : 1.f;
          st[192] = qh0.x; st[256] = qh0.y * (sx * sy); st[320] = qh0.z * (sx * sz);
          st[384] = qh0.w; st[448] = qh1.x * (sy * sz); st[512] = qh1.y;
          st[576] = -jHi; st[640] = jLo;
        } else {
          st[192] = q.w * q.w;
        }
        ids[warp][(pos >> 5) % NB][pos & 31] = (uint32_t)(ds.x + lane);
      }
      staged += __popc(m);
      if (staged - 32 * tested >= 32) {
        test(32);
        if (CW == 1 && tested - window == NB - 1) {
          const int h = hits;
          writeOut(cnt);
          cnt += h;
        }
      }
    }
    if (CW == 4) {
      if (staged > 32 * tested) test(staged - 32 * tested);
      staged = 32 * tested;
      part[sub][lane] = hits;
      __syncthreads();
      int at = cnt;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (w < sub) at += part[w][lane];
        cnt += part[w][lane];
      }
      writeOut(at);
    }
    groupSync();   // the next tile overwrites desc, offs and part
  }
  if (CW == 1) {
    if (staged > 32 * tested) test(staged - 32 * tested);
    const int h = hits;
    writeOut(cnt);
    cnt += h;
  }
  if (sub != 0) return;
  // The stored count never exceeds the capacity: sweeps that run before an
  // overflow is noticed read only written slots.  The true maximum goes to
  // maxCount (the overflow signal).
  if (active) counts[i] = WRITE ? min(cnt, cap) : cnt;
  const int gmax = __reduce_max_sync(0xffffffffu, active ? cnt : 0);
  const int gsum = __reduce_add_sync(0xffffffffu, active ? cnt : 0);
  if (lane == 0) {
    if (gmax > *(volatile int*)&sc->maxCount) atomicMax(&sc->maxCount, gmax);
    atomicAdd(&sc->entries[blockIdx.x & (kEntrySums - 1)], (unsigned long long)gsum);
  }
}

// Work items of the search: every chunk of up to `width` consecutive nodes of
// a cell, in items[], the chunks of one cell consecutive (their order among
// cells is free); chunkOf[first node of the cell] = its first chunk.
// The keys of a sort that gave up waiting are in no order: a cell may come up in
// several runs, and its chunks would not fit items[].  Then there are no items
// (the search finds nothing to do) and every list is empty, until the host reads
// the flag.
__global__ void itemsKernel(const uint32_t* __restrict__ keys, long n, int shift, uint32_t space,
                            const int* __restrict__ cellEnd, int width, int* __restrict__ items,
                            int* __restrict__ chunkOf, int* __restrict__ counts, StepScratch* __restrict__ sc) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (sc->sortTimeout) {   // uniform
    if (k < n) counts[k] = 0;
    return;
  }
  const int lane = threadIdx.x & 31;
  int chunks = 0, first = 0;
  if (k < n) {
    const uint32_t key = keys[k] >> shift;
    if (key < space && (k == 0 || (keys[k - 1] >> shift) != key)) {
      chunks = (cellEnd[key] - (int)k + width - 1) / width;
      first = (int)k;
    }
  }
  // block prefix, one atomic per block (one per warp, all on one address: items
  // of 2.1 M nodes 62 us, now 45)
  __shared__ int warpSum[8], blockBase;
  const int warp = threadIdx.x >> 5;
  int incl = chunks;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warpSum[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < 8; ++w) { const int c = warpSum[w]; warpSum[w] = sum; sum += c; }
    blockBase = sum > 0 ? atomicAdd(&sc->items, sum) : 0;
  }
  __syncthreads();
  const int base = blockBase + warpSum[warp] + incl - chunks;
  if (chunks > 0) chunkOf[first] = base;
  for (int c = 0; c < chunks; ++c) items[base + c] = first + c * width;
}
// Bounding box of every work chunk in its cell's FP32 coordinates, with the
// smallest and largest h^-1, W lanes per chunk: box[2k] = (min x, min y,
// min z, min a), box[2k+1] = (max x, max y, max z, max a).
// TENSOR adds what bounds |H r|^2 of all its nodes from below and the widest
// tensor band: tbox[k] = (d_x, d_y, d_z, band) with H^2 - diag(d) positive
// semidefinite for every node.  Per node (tensorDiagonal) one of two such d, and
// a chunk takes the smallest of each component, which keeps the property:
//  * d_a = (H^2)_aa - sum_b |(H^2)_ab| (Gershgorin) where all three are
//    positive.  With one of them negative it bounds nothing, not even with
//    that one raised to zero;
//  * else 1 / (H^-2)_aa on the axis where that is largest and zero on the other
//    two: r_a is row a of H^-1 times H r, so r_a^2 <= (H^-2)_aa |H r|^2 for any
//    H.  Axis ratios above 1 + sqrt(2) reach it when the axes are tilted.
// Both are lowered by more than the FP32 error of their terms (in units of the
// largest eigenvalue the components are at most 1, their products in the rows
// and the determinant then carry a few 2^-24 each).
__device__ __forceinline__ void tensorDiagonal(const float4& a, const float4& b, float& dx, float& dy, float& dz) {
  const float xy = fabsf(a.x * a.y + a.y * a.w + a.z * b.x), xz = fabsf(a.x * a.z + a.y * b.x + a.z * b.y);
  const float yz = fabsf(a.y * a.z + a.w * b.x + b.x * b.y);
  const float l2 = b.w * b.w, m = 1.0e-5f * l2;
  dx = a.x * a.x + a.y * a.y + a.z * a.z - xy - xz - m;
  dy = a.y * a.y + a.w * a.w + b.x * b.x - xy - yz - m;
  dz = a.z * a.z + b.x * b.x + b.y * b.y - xz - yz - m;
  if (dx >= 0.0f && dy >= 0.0f && dz >= 0.0f) return;
  // rows of det(H) H^-1 in units of the largest eigenvalue
  const float i = 1.0f / b.w, u = 5.9604645e-8f;
  const float xx = a.x * i, hxy = a.y * i, hxz = a.z * i, yy = a.w * i, hyz = b.x * i, zz = b.y * i;
  const float cxx = yy * zz - hyz * hyz, cxy = hxz * hyz - hxy * zz, cxz = hxy * hyz - hxz * yy;
  const float cyy = xx * zz - hxz * hxz, cyz = hxy * hxz - xx * hyz, czz = xx * yy - hxy * hxy;
  const float rx = cxx * cxx + cxy * cxy + cxz * cxz, ry = cxy * cxy + cyy * cyy + cyz * cyz;
  const float rz = cxz * cxz + cyz * cyz + czz * czz;
  const float r = fminf(rx, fminf(ry, rz));
  const float q = fmaxf(0.0f, xx * cxx + hxy * cxy + hxz * cxz - 32.0f * u) / (sqrtf(r) + 32.0f * u);
  const float d = (q * q) * l2 * (1.0f - 32.0f * u);
  dx = r == rx ? d : 0.0f;
  dy = r != rx && r == ry ? d : 0.0f;
  dz = r != rx && r != ry ? d : 0.0f;
}
template <int W, bool TENSOR>
__global__ void __launch_bounds__(128) itemBoxKernel(const int* __restrict__ items, const StepScratch* __restrict__ sc,
                                                     long n, Grid g, Fields32 P, float4* __restrict__ box,
                                                     float4* __restrict__ tbox) {
  const int k = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) / W);
  const int lane = threadIdx.x % W;
  const bool live = k < sc->items;
  const int s = live ? items[k] : 0;
  const long j = (long)s + lane;
  const bool in = live && j < n && P.cell[j] == P.cell[s];
  const float4 q = P.posh[in ? j : s];
  constexpr int NC = TENSOR ? 8 : 4;
  float lo[NC] = {q.x, q.y, q.z, q.w}, hi[4] = {q.x, q.y, q.z, q.w};
  if (TENSOR) {
    const float4 a = P.hten[in ? j : s], b = P.hten[P.stride + (in ? j : s)];
    tensorDiagonal(a, b, lo[4 % NC], lo[5 % NC], lo[6 % NC]);
    lo[7 % NC] = -tensorBand(b.w, q.w, g);
  }
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
#pragma unroll
    for (int c = 0; c < 4; ++c) hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
  }
  if (live && lane == 0) {
    box[2 * k] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    box[2 * k + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
    if (TENSOR) tbox[k] = make_float4(lo[4 % NC], lo[5 % NC], lo[6 % NC], -lo[7 % NC]);
  }
}

//------------------------------------------------------------------------------
// computeSPHSumMassDensity (src/SPH/computeSPHSumMassDensity.cc:15-87),
// gathered: rho_i = m_i W(0) Hdet_i + sum_j m W(|Hj ri - Hj rj|, Hdet_j) with
// m = m_j for the same NodeList and m_i otherwise.  Tensor H_j (ASPH), seen
// through the image of the entry.
//------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) sumDensityKernel(Fields F, const int* __restrict__ list, long n, Grid g,
                                                        NeighborLists nl, TableDev t, HydroParams hp) {
  extern __shared__ double smem[];
  const int ntab = 3 * (hp.tableN1 + 1);
  for (int k = threadIdx.x; k < ntab; k += blockDim.x) smem[k] = t.w[k];
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const double* __restrict__ X = F.f[F_X];
  const double* __restrict__ Y = F.f[F_Y];
  const double* __restrict__ Z = F.f[F_Z];
  const double* __restrict__ Ms = F.f[F_MASS];
  const double xi = X[i], yi = Y[i], zi = Z[i], mi = Ms[i];
  const int li = list[i];
  const double Hdeti = symDet(loadSym(F, F_HT_XX, i));
  const double self = mi * (Hdeti * smem[0]);
  double sum = 0.0;
  const int cnt = nl.count[i];
  for (int q = 0; q < cnt; ++q) {
    const long long k = nbSlot(i, q, nl.cap);
    const uint32_t ent = nl.nbr[k];
    const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
    double xj = X[j], yj = Y[j], zj = Z[j];
    imagePos(g, code, xj, yj, zj);
    double dx, dy, dz, Hdetj;
    {   // |Hj ri - Hj rj|
      Sym Hj = loadSym(F, F_HT_XX, j);
      imageSym(g, code, Hj);
      double ax, ay, az, bx, by, bz;
      symDot(Hj, xi, yi, zi, ax, ay, az);
      symDot(Hj, xj, yj, zj, bx, by, bz);
      dx = ax - bx; dy = ay - by; dz = az - bz;
      Hdetj = symDet(Hj);
    }
    const double eta = sqrt(dx * dx + dy * dy + dz * dz);
    if (eta < hp.extent) {
      const int i0 = tableIndex(eta, hp.tableN1, hp.tableXstep);
      const double Wj = Hdetj * tableEval(smem, i0, eta);
      sum += (list[j] == li ? Ms[j] : mi) * Wj;
    }
  }
  F.f[F_RHO][i] = self + sum;
}

//------------------------------------------------------------------------------
// computeSPHOmegaGradhCorrection (src/SPH/computeSPHOmegaGradhCorrection.cc:15-116).
//------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) gradhKernel(Fields F, long n, Grid g, NeighborLists nl, TableDev t,
                                                   HydroParams hp) {
  extern __shared__ double smem[];
  const int ntab = 3 * (hp.tableN1 + 1);
  for (int k = threadIdx.x; k < ntab; k += blockDim.x) { smem[k] = t.w[k]; smem[ntab + k] = t.g[k]; }
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const double* __restrict__ X = F.f[F_X];
  const double* __restrict__ Y = F.f[F_Y];
  const double* __restrict__ Z = F.f[F_Z];
  const double xi = X[i], yi = Y[i], zi = Z[i];
  const Sym Hi = loadSym(F, F_HT_XX, i);
  const double Hdeti = symDet(Hi);
  double wsum = 0.0, gsum = 0.0;
  const int cnt = nl.count[i];
  for (int q = 0; q < cnt; ++q) {
    const long long k = nbSlot(i, q, nl.cap);
    const uint32_t ent = nl.nbr[k];
    const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
    double xj = X[j], yj = Y[j], zj = Z[j];
    imagePos(g, code, xj, yj, zj);
    const double rx = xi - xj, ry = yi - yj, rz = zi - zj;
    double ex, ey, ez;
    symDot(Hi, rx, ry, rz, ex, ey, ez);
    const double eta = sqrt(ex * ex + ey * ey + ez * ez);
    if (eta < hp.extent) {
      const int i0 = tableIndex(eta, hp.tableN1, hp.tableXstep);
      wsum += Hdeti * tableEval(smem, i0, eta);
      gsum += eta * (Hdeti * tableEval(smem + ntab, i0, eta));
    }
  }
  double omega;
  if (cnt == 0) omega = 1.0;
  else omega = fmax(1.0e-30, -gsum / (3.0 * (wsum + Hdeti * hp.W0)));
  F.f[F_OMEGA][i] = omega;
}

//------------------------------------------------------------------------------
// SPH::evaluateDerivativesImpl (src/SPH/SPH.cc:294-552) with
// MonaghanGingoldViscosity::QPiij (MonaghanGingoldViscosity.cc:41-101) and the
// SPHSmoothingScale moments + IdealH (SPHSmoothingScale.cc:154-272), FP64.
//------------------------------------------------------------------------------
// ASPH: symmetric-tensor H_i, H_j (eta = H r, grad W = gW H eta^), the
// ASPHClassicSmoothingScale second moment and its finalize.
template <bool XSPH, bool COMPAT>
__global__ void __launch_bounds__(128) pairKernelFP64(Fields F, const int* __restrict__ list, long n, Grid g,
                                                      NeighborLists nl, TableDev t, HydroParams hp,
                                                      double* __restrict__ pacc) {
  extern __shared__ double smem[];
  const int ntab = 3 * (hp.tableN1 + 1);
  for (int k = threadIdx.x; k < ntab; k += blockDim.x) { smem[k] = t.w[k]; smem[ntab + k] = t.g[k]; }
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const double* __restrict__ X = F.f[F_X];
  const double* __restrict__ Y = F.f[F_Y];
  const double* __restrict__ Z = F.f[F_Z];
  const double* __restrict__ VX = F.f[F_VX];
  const double* __restrict__ VY = F.f[F_VY];
  const double* __restrict__ VZ = F.f[F_VZ];
  const double* __restrict__ Ms = F.f[F_MASS];
  const double* __restrict__ RHO = F.f[F_RHO];
  const double* __restrict__ PP = F.f[F_P];
  const double* __restrict__ CS = F.f[F_CS];
  const double* __restrict__ OM = F.f[F_OMEGA];
  const double* __restrict__ tw = smem;
  const double* __restrict__ tg = smem + ntab;

  const double xi = X[i], yi = Y[i], zi = Z[i], vxi = VX[i], vyi = VY[i], vzi = VZ[i];
  const double mi = Ms[i], rhoi = RHO[i], Pi = PP[i], ci = CS[i], omi = OM[i];
  const int li = list[i];
  const Sym Hi = loadSym(F, F_HT_XX, i);
  const double Hdeti = symDet(Hi);
  const double safeOmegai = omi / (omi * omi + kTiny30);
  const double tiny = kTiny30;
  const double Clij = 0.5 * (1.0 + 1.0) * 1.0 * hp.Cl;
  const double Cqij = 0.5 * (1.0 + 1.0) * 1.0 * hp.Cq;
  double DQi[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) DQi[k] = hp.limitedQ ? F.f[F_DVDXQ_XX + k][i] : 0.0;

  NodeAcc a;
  a.rhoSum = a.norm = a.dvx = a.dvy = a.dvz = a.deps = a.gx = a.gy = a.gz = 0.0;
  a.maxQ = 0.0; a.effQ = a.xw = a.xdx = a.xdy = a.xdz = a.m0 = a.m1x = a.m1y = a.m1z = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) { a.D[k] = 0.0; a.M[k] = 0.0; }
#pragma unroll
  for (int k = 0; k < 6; ++k) a.m2[k] = 0.0;

  const int cnt = nl.count[i];
  for (int q = 0; q < cnt; ++q) {
    const long long k = nbSlot(i, q, nl.cap);
    const uint32_t ent = nl.nbr[k];
    const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
    double xj = X[j], yj = Y[j], zj = Z[j], vxj = VX[j], vyj = VY[j], vzj = VZ[j];
    imagePos(g, code, xj, yj, zj);
    imageVec(g, code, vxj, vyj, vzj);
    const double mj = Ms[j], rhoj = RHO[j], Pj = PP[j], cj = CS[j], omj = OM[j];
    const int lj = list[j];
    Sym Hj = loadSym(F, F_HT_XX, j);
    imageSym(g, code, Hj);
    const double Hdetj = symDet(Hj);
    const double safeOmegaj = omj / (omj * omj + kTiny30);

    const double rx = xi - xj, ry = yi - yj, rz = zi - zj;
    double eix, eiy, eiz, ejx, ejy, ejz;
    symDot(Hi, rx, ry, rz, eix, eiy, eiz);
    symDot(Hj, rx, ry, rz, ejx, ejy, ejz);
    const double etaMag2i = eix * eix + eiy * eiy + eiz * eiz;
    const double etaMag2j = ejx * ejx + ejy * ejy + ejz * ejz;
    const double etaMagi = sqrt(etaMag2i), etaMagj = sqrt(etaMag2j);
    const double sIi = 1.0 / fmax(tiny, etaMagi), sIj = 1.0 / fmax(tiny, etaMagj);
    const double uix = eix * sIi, uiy = eiy * sIi, uiz = eiz * sIi;
    const double ujx = ejx * sIj, ujy = ejy * sIj, ujz = ejz * sIj;
    double Wi = 0.0, gi = 0.0, Wj = 0.0, gj = 0.0;
    if (etaMagi < hp.extent) {
      const int i0 = tableIndex(etaMagi, hp.tableN1, hp.tableXstep);
      Wi = tableEval(tw, i0, etaMagi);
      gi = tableEval(tg, i0, etaMagi);
    }
    if (etaMagj < hp.extent) {
      const int i0 = tableIndex(etaMagj, hp.tableN1, hp.tableXstep);
      Wj = tableEval(tw, i0, etaMagj);
      gj = tableEval(tg, i0, etaMagj);
    }
    const double WSPHi = fabs(gi);
    Wi *= Hdeti; Wj *= Hdetj;
    const double gWi = Hdeti * gi, gWj = Hdetj * gj;
    double gwix, gwiy, gwiz, gwjx, gwjy, gwjz;
    {   // gW H eta^
      double hx, hy, hz;
      symDot(Hi, uix, uiy, uiz, hx, hy, hz);
      gwix = gWi * hx; gwiy = gWi * hy; gwiz = gWi * hz;
      symDot(Hj, ujx, ujy, ujz, hx, hy, hz);
      gwjx = gWj * hx; gwjy = gWj * hy; gwjz = gWj * hz;
    }

    if (lj == li) {
      a.rhoSum += mj * Wi;
      a.norm += mi / rhoi * Wi;
    }
    const double vijx = vxi - vxj, vijy = vyi - vyj, vijz = vzi - vzj;
    // Monaghan-Gingold Q; the limited form first corrects the two velocities
    // along the pair with the Q's DvDx (LimitedMonaghanGingoldViscosity.cc:171-200)
    double vqx = vijx, vqy = vijy, vqz = vijz;
    if (hp.limitedQ) {
      double Dj[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) Dj[k] = F.f[F_DVDXQ_XX + k][j];
      imageTensor(g, code, Dj);
      const double hx = 0.5 * rx, hy = 0.5 * ry, hz = 0.5 * rz;
      const double aix = DQi[0] * hx + DQi[1] * hy + DQi[2] * hz;
      const double aiy = DQi[3] * hx + DQi[4] * hy + DQi[5] * hz;
      const double aiz = DQi[6] * hx + DQi[7] * hy + DQi[8] * hz;
      const double ajx = Dj[0] * hx + Dj[1] * hy + Dj[2] * hz;
      const double ajy = Dj[3] * hx + Dj[4] * hy + Dj[5] * hz;
      const double ajz = Dj[6] * hx + Dj[7] * hy + Dj[8] * hz;
      const double gri = aix * hx + aiy * hy + aiz * hz;
      const double grj = ajx * hx + ajy * hy + ajz * hz;
      const double rri = gri / ((grj < 0.0 ? -1.0 : 1.0) * fmax(1.0e-30, fabs(grj)));
      const double rrj = grj / ((gri < 0.0 ? -1.0 : 1.0) * fmax(1.0e-30, fabs(gri)));
      const double xl = fmin(rri, rrj);
      double phi = xl > 0.0 ? 2.0 / (1.0 + xl) * 2.0 * xl / (1.0 + xl) : 0.0;   // van Leer
      const double etaij = fmin(etaMagi, etaMagj);
      if (etaij < hp.etaCrit) {
        const double z = (etaij - hp.etaCrit) / hp.etaFold;
        phi *= exp(-(z * z));
      }
      vqx = (vxi - phi * aix) - (vxj + phi * ajx);
      vqy = (vyi - phi * aiy) - (vyj + phi * ajy);
      vqz = (vzi - phi * aiz) - (vzj + phi * ajz);
    }
    const double mui = (vqx * eix + vqy * eiy + vqz * eiz) / (etaMag2i + hp.eps2);
    const double muj = (vqx * ejx + vqy * ejy + vqz * ejz) / (etaMag2j + hp.eps2);
    const double lmi = hp.linearInExpansion ? mui : fmin(0.0, mui);
    const double lmj = hp.linearInExpansion ? muj : fmin(0.0, muj);
    const double qmi = hp.quadraticInExpansion ? -(mui < 0.0 ? -1.0 : 1.0) * mui * mui : fmin(0.0, mui) * fmin(0.0, mui);
    const double qmj = hp.quadraticInExpansion ? -(muj < 0.0 ? -1.0 : 1.0) * muj * muj : fmin(0.0, muj) * fmin(0.0, muj);
    const double ei = -Clij * ci * lmi + Cqij * qmi;
    const double ej = -Clij * cj * lmj + Cqij * qmj;
    const double QPiij = ei / rhoi, QPiji = ej / rhoj;
    const double Qi = rhoi * ei;
    const double qai = 0.5 * QPiij, qaj = 0.5 * QPiji;
    const double Qaix = qai * gwix, Qaiy = qai * gwiy, Qaiz = qai * gwiz;
    const double Qajx = qaj * gwjx, Qajy = qaj * gwjy, Qajz = qaj * gwjz;
    const double workQi = vijx * Qaix + vijy * Qaiy + vijz * Qaiz;
    a.maxQ = fmax(a.maxQ, Qi);
    a.effQ += mj * Qi * Wi / rhoj;
    double Peffi = Pi, Peffj = Pj;
    if (hp.epsTensile != 0.0) {
      const double ri = Wi / (Hdeti * hp.WnPerh), rj = Wj / (Hdetj * hp.WnPerh);
      Peffi += hp.epsTensile * (ri * ri * ri * ri) * (Pi < 0.0 ? -Pi : 0.0);
      Peffj += hp.epsTensile * (rj * rj * rj * rj) * (Pj < 0.0 ? -Pj : 0.0);
    }
    const double Prhoi = safeOmegai * Peffi / (rhoi * rhoi);
    const double Prhoj = safeOmegaj * Peffj / (rhoj * rhoj);
    const double ddx = Prhoi * gwix + Prhoj * gwjx + Qaix + Qajx;
    const double ddy = Prhoi * gwiy + Prhoj * gwjy + Qaiy + Qajy;
    const double ddz = Prhoi * gwiz + Prhoj * gwjz + Qaiz + Qajz;
    a.dvx -= mj * ddx;
    a.dvy -= mj * ddy;
    a.dvz -= mj * ddz;
    if (COMPAT) {
      double* out = pacc + paccSlot(k);
      out[0] = -mj * ddx;
      out[32] = -mj * ddy;
      out[64] = -mj * ddz;
    }
    a.deps += mj * (Prhoi * (vijx * gwix + vijy * gwiy + vijz * gwiz) + workQi);
    const double mvx = mj * vijx, mvy = mj * vijy, mvz = mj * vijz;
    a.D[0] -= mvx * gwix; a.D[1] -= mvx * gwiy; a.D[2] -= mvx * gwiz;
    a.D[3] -= mvy * gwix; a.D[4] -= mvy * gwiy; a.D[5] -= mvy * gwiz;
    a.D[6] -= mvz * gwix; a.D[7] -= mvz * gwiy; a.D[8] -= mvz * gwiz;
    if (XSPH) {
      const double wx = 0.5 * (mi / rhoi * Wi + mj / rhoj * Wj);
      a.xw += wx;
      a.xdx -= wx * vijx; a.xdy -= wx * vijy; a.xdz -= wx * vijz;
    }
    const double gr = mj * (rhoj - rhoi);
    a.gx += gr * gwix; a.gy += gr * gwiy; a.gz += gr * gwiz;
    const double mrx = mj * rx, mry = mj * ry, mrz = mj * rz;
    a.M[0] -= mrx * gwix; a.M[1] -= mrx * gwiy; a.M[2] -= mrx * gwiz;
    a.M[3] -= mry * gwix; a.M[4] -= mry * gwiy; a.M[5] -= mry * gwiz;
    a.M[6] -= mrz * gwix; a.M[7] -= mrz * gwiy; a.M[8] -= mrz * gwiz;
    // SPHSmoothingScale zeroth / first moments
    const double fw = (lj != li) ? mj * rhoi / (mi * rhoj) : 1.0;
    a.m0 += fw * WSPHi;
    const double fwW = fw * WSPHi;
    a.m1x -= fwW * eix; a.m1y -= fwW * eiy; a.m1z -= fwW * eiz;
    {   // ASPHClassicSmoothingScale second moment: WSPH^2 r r / |r|^5
      const double rm = sqrt(rx * rx + ry * ry + rz * rz);
      const double f5 = 1.0 / fmax(kTiny30, rm * rm * rm * rm * rm);
      const double w2 = fwW * WSPHi;
      a.m2[0] += w2 * (rx * rx * f5); a.m2[1] += w2 * (rx * ry * f5); a.m2[2] += w2 * (rx * rz * f5);
      a.m2[3] += w2 * (ry * ry * f5); a.m2[4] += w2 * (ry * rz * f5); a.m2[5] += w2 * (rz * rz * f5);
    }
  }
  finalizeNodeASPH(F, i, li, a, Hi, mi, rhoi, vxi, vyi, vzi, cnt, hp, t.herm);
}

//------------------------------------------------------------------------------
// GenericHydro::dt (src/Physics/GenericHydro.cc:113-381): node limits and the
// pairwise velocity-difference limit, min-reduced.  The reason code travels
// with the value (value, reason) through both reduction stages.
//------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) dtKernel(Fields F, const int* __restrict__ list, long n, Grid g,
                                                NeighborLists nl, HydroParams hp, double maxNperh,
                                                double* __restrict__ part) {
  __shared__ double sv[128];
  __shared__ int sr[128];
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const double tiny = DBL_EPSILON;
  double best = DBL_MAX;
  int reason = -1;
  if (i < n && !isGhost(hp, i)) {
    int hc[3];
    unpackCell(nl.cell[i], hc);
    const NodeListParams L = hp.lists[list[i]];
    // max eigenvalue of H: h^-1 when isotropic, the stored extent for tensor H
    const double* __restrict__ HX = F.f[hp.asph ? F_HLMAX : F_HINV];
    const double ai = HX[i];
    const double nodeScalei = 1.0 / ai / L.nPerh;
    const double vxi = F.f[F_VX][i], vyi = F.f[F_VY][i], vzi = F.f[F_VZ][i];
    const double rhoi = F.f[F_RHO][i];
    const double csDt = nodeScalei / (F.f[F_CS][i] + tiny);
    if (csDt < best) { best = csDt; reason = 0; }
    const double csq = sqrt(F.f[F_MAXQ][i] / rhoi);
    const double csqDt = nodeScalei / (csq + tiny);
    if (csqDt < best) { best = csqDt; reason = 1; }
    const double divv = F.f[F_DVDX_XX][i] + F.f[F_DVDX_YY][i] + F.f[F_DVDX_ZZ][i];
    const double divvDt = 1.0 / (fabs(divv) + tiny);
    if (divvDt < best) { best = divvDt; reason = 2; }
    const double vmag = sqrt(vxi * vxi + vyi * vyi + vzi * vzi);
    const double ax = F.f[F_DVDT_X][i], ay = F.f[F_DVDT_Y][i], az = F.f[F_DVDT_Z][i];
    const double amag = sqrt(ax * ax + ay * ay + az * az);
    const double dtAcc = 0.1 * fmax(nodeScalei / (vmag + tiny), vmag / (amag + tiny));
    if (dtAcc < best) { best = dtAcc; reason = 3; }
    if (hp.useVelMagDt) {
      const double velDt = nodeScalei / (vmag + 1.0e-10);
      if (velDt < best) { best = velDt; reason = 4; }
    }
    const double nsi = 1.0 / ai / maxNperh;
    const int cnt = nl.count[i];
    for (int q = 0; q < cnt; ++q) {
      const long long k = nbSlot(i, q, nl.cap);
      const uint32_t ent = nl.nbr[k];
      const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
      double vxj = F.f[F_VX][j], vyj = F.f[F_VY][j], vzj = F.f[F_VZ][j];
      imageVec(g, code, vxj, vyj, vzj);
      const double nsj = 1.0 / HX[j] / maxNperh;
      const double dvx = vxi - vxj, dvy = vyi - vyj, dvz = vzi - vzj;
      const double vm = sqrt(dvx * dvx + dvy * dvy + dvz * dvz);
      const double dtv = fmin(nsi, nsj) * (1.0 / fmax(tiny, vm));
      if (dtv < best) { best = dtv; reason = 5; }
    }
  }
  sv[threadIdx.x] = best;
  sr[threadIdx.x] = reason;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o && sv[threadIdx.x + o] < sv[threadIdx.x]) {
      sv[threadIdx.x] = sv[threadIdx.x + o];
      sr[threadIdx.x] = sr[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = sv[0]; part[2 * blockIdx.x + 1] = (double)sr[0]; }
}
__global__ void dtFinalKernel(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double sv[256];
  __shared__ double sr[256];
  double best = DBL_MAX, reason = -1.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    if (part[2 * b] < best) { best = part[2 * b]; reason = part[2 * b + 1]; }
  sv[threadIdx.x] = best;
  sr[threadIdx.x] = reason;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o && sv[threadIdx.x + o] < sv[threadIdx.x]) {
      sv[threadIdx.x] = sv[threadIdx.x + o];
      sr[threadIdx.x] = sr[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { out[0] = sv[0]; out[1] = sr[0]; }
}

//------------------------------------------------------------------------------
// State updates (State::update with IncrementState / IncrementBoundedState /
// ReplaceBoundedState, PressurePolicy, SoundSpeedPolicy) and GammaLawGas.
//------------------------------------------------------------------------------
__device__ __forceinline__ void eosNode(Fields& F, long i, const NodeListParams& L) {
  const double rho = F.f[F_RHO][i], eps = F.f[F_EPS][i];
  double p = (L.gamma - 1.0) * rho * eps;
  p = p < L.minP ? L.minP : (p > L.maxP ? L.maxP : p);
  F.f[F_P][i] = p;
  F.f[F_CS][i] = sqrt(fmax(0.0, L.gamma * (L.gamma - 1.0) * eps));
}

// Extent of tensor H (ASPH): smallest eigenvalue -> F_HINV (cell size,
// neighbour pre-filter), largest -> F_HLMAX (dt node scale).
__device__ __forceinline__ void storeExtent(Fields& F, long i, const Sym& h) {
  double lmin, lmax;
  symExtent(h, lmin, lmax);
  F.f[F_HINV][i] = lmin;
  F.f[F_HLMAX][i] = lmax;
}
// Mixed mode: the same extents from an FP32 Jacobi decomposition (GB300's
// FP64 transcendental sequences would dominate the update).  The smallest
// eigenvalue only has to bound |H r| / |r| from below (neighbour pre-filter),
// so it is lowered by a margin far above the FP32 eigenvalue error; the
// largest feeds the FP32 dt vote.
__device__ __forceinline__ void storeExtent32(Fields& F, long i, const Sym& h) {
  const SymT<float> hf{(float)h.xx, (float)h.xy, (float)h.xz, (float)h.yy, (float)h.yz, (float)h.zz};
  float val[3], V[3][3];
  symEigen(hf, val, V);
  F.f[F_HINV][i] = (double)fminf(val[0], fminf(val[1], val[2])) * (1.0 - 1.0e-5);
  F.f[F_HLMAX][i] = (double)fmaxf(val[0], fmaxf(val[1], val[2]));
}
// ASPH radialOnly: the radius of every node at the start of the step
// (SmoothingScaleBase::preStepInitialize).
__global__ void radius0Kernel(Fields F, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = F.f[F_X][i], y = F.f[F_Y][i], z = F.f[F_Z][i];
  F.f[F_RAD0][i] = sqrt(x * x + y * y + z * z);
}
// ASPHSmoothingScale::finalize (src/SmoothingScale/ASPHSmoothingScale.cc:157-380)
// in its fixShape and radialOnly forms, gathered: the zeroth moment of the
// end-of-step state over the step's neighbour lists (fweight_ij WSPH(|H_i r_ij|)),
// the IdealH size ratio, H scaled (fixShape) or reshaped radially about the
// origin (radialOnly), then the eigenvalue limits; with IntegrateH or FixedH
// only the limits.  FP64 in both precision modes; in the mixed mode the FP32
// extents and mirrors of the new H are written as the update writes them.
__global__ void __launch_bounds__(128) asphEndKernel(Fields F, Fields32 P, const int* __restrict__ list, long n,
                                                    Grid g, NeighborLists nl, TableDev t, HydroParams hp) {
  extern __shared__ double smem[];   // dW/deta coefficients
  const int ntab = 3 * (hp.tableN1 + 1);
  for (int k = threadIdx.x; k < ntab; k += blockDim.x) smem[k] = t.g[k];
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int li = list[i];
  const NodeListParams L = hp.lists[li];
  const Sym Hi = loadSym(F, F_HT_XX, i);
  Sym Hn;
  if (hp.hUpdate != 0) {
    Hn = limitASPH(Hi, L.hminInv, L.hmaxInv, L.hminratio);
  } else {
    int hc[3];
    unpackCell(nl.cell[i], hc);
    const double* __restrict__ X = F.f[F_X];
    const double* __restrict__ Y = F.f[F_Y];
    const double* __restrict__ Z = F.f[F_Z];
    const double xi = X[i], yi = Y[i], zi = Z[i];
    const double mi = F.f[F_MASS][i], rhoi = F.f[F_RHO][i];
    const bool multi = hp.numLists > 1;
    double m0 = 0.0;
    const int cnt = nl.count[i];
    for (int q = 0; q < cnt; ++q) {
      const uint32_t ent = nl.nbr[nbSlot(i, q, nl.cap)];
      const int j = (int)(ent & kIndexMask), code = imageCode(g, hc, (int)(ent >> kIndexBits));
      double xj = X[j], yj = Y[j], zj = Z[j];
      imagePos(g, code, xj, yj, zj);
      double ex, ey, ez;
      symDot(Hi, xi - xj, yi - yj, zi - zj, ex, ey, ez);
      const double eta = sqrt(ex * ex + ey * ey + ez * ez);
      if (eta < hp.extent) {
        const double wsph = fabs(tableEval(smem, tableIndex(eta, hp.tableN1, hp.tableXstep), eta));
        const double fw = (multi && list[j] != li) ? F.f[F_MASS][j] * rhoi / (mi * F.f[F_RHO][j]) : 1.0;
        m0 += fw * wsph;
      }
    }
    const double mz = rootnu3T(fmax(0.0, m0));
    F.f[F_M0][i] = mz;
    const bool isolated = fabs(mz) <= 1.0e-15 * fmax(1.0, fabs(mz));
    const double cur = isolated ? 0.5 * L.nPerh : fmax(0.0, hermiteLookup(t.herm, hp, mz));
    const double s = fmin(4.0, fmax(0.25, L.nPerh / (cur + 1.0e-30)));
    const double aa = s < 1.0 ? 0.4 * (1.0 + s * s) : 0.4 * (1.0 + 1.0 / (s * s * s));
    const double f = 1.0 - aa + aa * s;
    const Sym Hid = hp.fixShape ? symDiv(Hi, f) : radialEvolution(Hi, xi, yi, zi, f, F.f[F_RAD0][i]);
    Hn = limitASPH(Hid, L.hminInv, L.hmaxInv, L.hminratio);
    storeSym(F, F_HIDEALT_XX, i, Hn);
  }
  storeSym(F, F_HT_XX, i, Hn);
  if (P.posh) {
    storeExtent32(F, i, Hn);
    P.posh[i].w = (float)F.f[F_HINV][i];
    writeTensorMirror(F, i, P, i);
  } else {
    storeExtent(F, i, Hn);
  }
}

__global__ void tensorExtentKernel(Fields F, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  storeExtent(F, i, loadSym(F, F_HT_XX, i));
}

__global__ void eosKernel(Fields F, const int* __restrict__ list, long n, const NodeListParams* __restrict__ lists) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  eosNode(F, i, lists[list[i]]);
}

// Boundary::setAllViolationNodes + enforceBoundary (PlanarBoundary.cc:153-190,
// ReflectingBoundary.cc:465-473): nodes strictly outside a plane are mapped
// back; reflecting walls also mirror the velocity.
__device__ __forceinline__ bool fuzzyZero(double x) { return fabs(x) <= 1.0e-15 * fmax(1.0, fabs(x)); }
// tensor: the H of a node mapped back through a reflecting wall is reflected
// too (PlanarBoundary::updateViolationNodes -> enforceBoundary(Hfield),
// (R H R).Symmetric()).
// p: the node's position, in and out.
__device__ __forceinline__ void enforceNode(Fields& F, long i, double* p_, const Grid& g, int tensor) {
  auto reflectH = [&](int a) {
    if (!tensor) return;
    if (a == 0) { F.f[F_HT_XY][i] = -F.f[F_HT_XY][i]; F.f[F_HT_XZ][i] = -F.f[F_HT_XZ][i]; }
    else if (a == 1) { F.f[F_HT_XY][i] = -F.f[F_HT_XY][i]; F.f[F_HT_YZ][i] = -F.f[F_HT_YZ][i]; }
    else { F.f[F_HT_XZ][i] = -F.f[F_HT_XZ][i]; F.f[F_HT_YZ][i] = -F.f[F_HT_YZ][i]; }
  };
  double* P[3] = {F.f[F_X], F.f[F_Y], F.f[F_Z]};
  double* V[3] = {F.f[F_VX], F.f[F_VY], F.f[F_VZ]};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double lo = g.wallLo[a], hi = g.wallHi[a];
    double p = p_[a];
    // Integer pre-test on order-preserving keys of the bit patterns: a node
    // strictly inside (lo, hi) needs nothing, and the FP64 tests below (the
    // FP64 pipe is narrow) run only for the few on or beyond a wall.
    if (orderKey(p) > orderKey(lo) && orderKey(p) < orderKey(hi)) continue;
    const double sdLo = p - lo, sdHi = hi - p;
    if (g.kindLo[a] == AXIS_PERIODIC) {
      if (sdLo < 0.0 && !fuzzyZero(sdLo)) p = imageCoord(p, 2, AXIS_PERIODIC, AXIS_PERIODIC, lo, hi);
      else if (sdHi < 0.0 && !fuzzyZero(sdHi)) p = imageCoord(p, 1, AXIS_PERIODIC, AXIS_PERIODIC, lo, hi);
      P[a][i] = p_[a] = p;
    } else {
      if (g.kindLo[a] == AXIS_REFLECT && sdLo < 0.0 && !fuzzyZero(sdLo)) {
        p = imageCoord(p, 1, AXIS_REFLECT, g.kindHi[a], lo, hi);
        P[a][i] = p_[a] = p;
        V[a][i] = -V[a][i];
        reflectH(a);
      }
      const double sdHi2 = hi - p;
      if (g.kindHi[a] == AXIS_REFLECT && sdHi2 < 0.0 && !fuzzyZero(sdHi2)) {
        p = imageCoord(p, 2, g.kindLo[a], AXIS_REFLECT, lo, hi);
        P[a][i] = p_[a] = p;
        V[a][i] = -V[a][i];
        reflectH(a);
      }
    }
  }
}

// End of a node's step: a node outside a wall is mapped back, the state is
// checked (finite, positive) and the bounds the next neighbour build needs are
// taken.  Returns whether the state is bad.
__device__ __forceinline__ bool endNode(Fields& F, long i, double* p, double vx, double vy, double vz, double m,
                                        double rho, double a, double eps, const Sym& H, bool tensor, const Grid& g,
                                        NodeBounds& b) {
  enforceNode(F, i, p, g, tensor);
  b.add(a, p);
  if (tensor) b.addTensor(H);   // the mirror of H through a wall has the same squares
  return !positiveBits(m) | !positiveBits(rho) | !positiveBits(a) | !finiteBits(eps) | !finiteBits(p[0]) |
         !finiteBits(p[1]) | !finiteBits(p[2]) | !finiteBits(vx) | !finiteBits(vy) | !finiteBits(vz);
}
// The same pass by itself, where something has to run between it and the update.
__global__ void __launch_bounds__(256) endStepKernel(Fields F, long n, Grid g, int tensor, StepScratch* __restrict__ sc) {
  NodeBounds b;
  bool bad = false;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double p[3] = {F.f[F_X][i], F.f[F_Y][i], F.f[F_Z][i]};
    Sym H{};
    if (tensor) H = loadSym(F, F_HT_XX, i);
    bad |= endNode(F, i, p, F.f[F_VX][i], F.f[F_VY][i], F.f[F_VZ][i], F.f[F_MASS][i], F.f[F_RHO][i], F.f[F_HINV][i],
                   F.f[F_EPS][i], H, tensor != 0, g, b);
  }
  if (bad) atomicExch(&sc->bad, 1);
  mergeBounds(b, tensor != 0, sc);
}

// The half-step update (mid) advances the current state and keeps its
// beginning-of-step copy (state0); the full update advances state0 itself
// (State::update after the reference's state.assign(state0)), eps already
// advanced by the compatible-energy sweep when compatible.
// P != nullptr (mixed mode): the FP32 mirrors of the new state are written
// here as well (the prepare pass folded into the update).
// tensor (ASPH): H is the symmetric tensor, bounded on its eigenvalues
// (IncrementBoundedState / ReplaceBoundedState with SymTensor min/max).
// hUpdate: HEvolutionType -- 0 IdealH (the full update replaces H by Hideal),
// 1 IntegrateH (both updates increment H by DHDt), 2 FixedH (H never changes).
// asphEnd (ASPHSmoothingScale): both updates integrate H with
// IncrementASPHHtensor (fixShape / radialOnly forms) unless FixedH.
// ex: what the step wants done in the same pass (UpdateExtras); END: its end.
template <bool TENSOR, bool END>
__global__ void __launch_bounds__(256, TENSOR ? 4 : 5) updateKernel(Fields F, const int* __restrict__ list, long n, const NodeListParams* __restrict__ lists,
                             double mult, int mid, int gravity, int epsIncrement, int hUpdate, int totalEnergy,
                             int crk, Fields32 P, Grid g, int asphEnd, int fixShape, int radialOnly,
                                                    UpdateExtras ex) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  NodeBounds bounds;
  if (i < n) {
  const NodeListParams L = lists[list[i]];
  // state the update starts from
  const int bx = mid ? F_X : F_X0, bvx = mid ? F_VX : F_VX0;
  // the position before this update (the radial direction of radialOnly:
  // State::update applies the "H" policy before the "position" one)
  const double xOld = F.f[bx][i], yOld = F.f[bx + 1][i], zOld = F.f[bx + 2][i];
  const double vxOld = F.f[bvx][i], vyOld = F.f[bvx + 1][i], vzOld = F.f[bvx + 2][i];
  const double rhoOld = F.f[mid ? F_RHO : F_RHO0][i], hOld = F.f[mid ? F_HINV : F_HINV0][i];
  const double volOld = crk ? F.f[mid ? F_VOL : F_VOL0][i] : 0.0;
  Sym HOld{}, HNew{};
  if (TENSOR) HOld = loadSym(F, mid ? F_HT_XX : F_HT0_XX, i);
  double eps = F.f[mid || !epsIncrement ? F_EPS : F_EPS0][i];
  if (mid) {   // state0
    F.f[F_X0][i] = xOld; F.f[F_Y0][i] = yOld; F.f[F_Z0][i] = zOld;
    F.f[F_VX0][i] = vxOld; F.f[F_VY0][i] = vyOld; F.f[F_VZ0][i] = vzOld;
    F.f[F_RHO0][i] = rhoOld; F.f[F_EPS0][i] = eps; F.f[F_HINV0][i] = hOld;
    if (TENSOR) storeSym(F, F_HT0_XX, i, HOld);
    if (crk) F.f[F_VOL0][i] = volOld;
  }
  const double ax = F.f[F_DVDT_X][i], ay = F.f[F_DVDT_Y][i], az = F.f[F_DVDT_Z][i];
  if (epsIncrement) {
    if (totalEnergy) {
      // SpecificFromTotalThermalEnergyPolicy::update: eps from the total
      // energy m (v^2/2 + eps) advanced by DEDt, with the hydro acceleration
      // for the new kinetic part (it fires before the velocity update)
      const double mi = F.f[F_MASS][i];
      const double v1x = vxOld + mult * ax, v1y = vyOld + mult * ay, v1z = vzOld + mult * az;
      const double E0 = mi * (0.5 * (vxOld * vxOld + vyOld * vyOld + vzOld * vzOld) + eps);
      const double E1 = E0 + mult * F.f[F_DEPSDT][i];
      eps = E1 / mi - 0.5 * (v1x * v1x + v1y * v1y + v1z * v1z);
    } else {
      eps += mult * F.f[F_DEPSDT][i];
    }
    F.f[F_EPS][i] = eps;
  }
  const double x = xOld + mult * F.f[F_DXDT_X][i];
  const double y = yOld + mult * F.f[F_DXDT_Y][i];
  const double z = zOld + mult * F.f[F_DXDT_Z][i];
  F.f[F_X][i] = x;
  F.f[F_Y][i] = y;
  F.f[F_Z][i] = z;
  // velocity: "delta velocity hydro" sorts before "delta velocity" (gravity)
  double vx = vxOld + mult * ax;
  double vy = vyOld + mult * ay;
  double vz = vzOld + mult * az;
  if (gravity) {
    vx += mult * F.f[F_GRAV_X][i];
    vy += mult * F.f[F_GRAV_Y][i];
    vz += mult * F.f[F_GRAV_Z][i];
  }
  F.f[F_VX][i] = vx;
  F.f[F_VY][i] = vy;
  F.f[F_VZ][i] = vz;
  const double rho = fmin(L.rhoMax, fmax(L.rhoMin, rhoOld + mult * F.f[F_DRHODT][i]));
  F.f[F_RHO][i] = rho;
  const double hminInv = L.hminInv, hmaxInv = L.hmaxInv;
  double h;
  const bool increment = mid || hUpdate == 1;
  if (hUpdate == 2) {   // FixedH: both copies hold the same H
    h = hOld;
    HNew = HOld;
  } else if (TENSOR && asphEnd) {
    const Sym t = incrementASPHHtensor(HOld, loadSym(F, F_DHDTT_XX, i), mult, xOld, yOld, zOld, fixShape != 0,
                                       radialOnly != 0, hminInv, hmaxInv, L.hminratio);
    storeSym(F, F_HT_XX, i, t);
    HNew = t;
    if (P.posh) storeExtent32(F, i, t);
    else storeExtent(F, i, t);
    h = F.f[F_HINV][i];
  } else if (TENSOR) {
    Sym t;
    if (increment) {
      const Sym d = loadSym(F, F_DHDTT_XX, i);
      t = Sym{HOld.xx + mult * d.xx, HOld.xy + mult * d.xy, HOld.xz + mult * d.xz, HOld.yy + mult * d.yy,
              HOld.yz + mult * d.yz, HOld.zz + mult * d.zz};
    } else {
      t = loadSym(F, F_HIDEALT_XX, i);
    }
    t = symBound(t, hmaxInv, hminInv);
    storeSym(F, F_HT_XX, i, t);
    HNew = t;
    if (P.posh) storeExtent32(F, i, t);
    else storeExtent(F, i, t);
    h = F.f[F_HINV][i];
  } else {
    h = increment ? hOld + mult * F.f[F_DHDT][i] : F.f[F_HIDEAL][i];
    if (h < hmaxInv) h = hmaxInv;
    if (h > hminInv) h = hminInv;
    F.f[F_HINV][i] = h;
  }
  if (crk) {
    // ContinuityVolumePolicy::update (src/RK/ContinuityVolumePolicy.cc:40-75):
    // it depends on the mass density, so it sees the updated rho and H
    const double mi = F.f[F_MASS][i];
    const double volMin = 0.5 * mi * safeInvVarD(rho);
    const double volMax = 4.0 * 3.141592653589793 / (3.0 * ((h * h) * h));
    const double dVdt = -mi * safeInvVarD(rho * rho) * F.f[F_DRHODT][i];
    F.f[F_VOL][i] = fmax(volMin, fmin(volMax, volOld + mult * dVdt));
  }
  if (P.posh) {
    // Mixed mode.  The sound speed feeds only FP32 sweeps (Q, dt vote), so it
    // is evaluated in FP32; the conversions between double and float take
    // the integer pipe (convert.cuh) and the cell origins an integer-built
    // index: GB300's FP64 pipe, which runs FP64 arithmetic and the
    // conversion instructions at ~1/64 of the FP32 rate, bounds this kernel.
    double p = L.gm1 * rho * eps;
    p = p < L.minP ? L.minP : (p > L.maxP ? L.maxP : p);
    F.f[F_P][i] = p;
    const float cs = sqrtf(fmaxf(0.0f, toFloatRN(L.ggm1 * eps)));
    F.f[F_CS][i] = toDouble(cs);
    int c[3];
    unpackCell(P.cell[i], c);
    const double ox = g.lo[0] + smallIntToDouble(c[0]) * g.cell[0];
    const double oy = g.lo[1] + smallIntToDouble(c[1]) * g.cell[1];
    const double oz = g.lo[2] + smallIntToDouble(c[2]) * g.cell[2];
    P.posh[i] = make_float4(toFloatRN(x - ox), toFloatRN(y - oy), toFloatRN(z - oz), toFloatRN(h));
    P.velm[i] = make_float4(toFloatRN(vx), toFloatRN(vy), toFloatRN(vz), toFloatRN(F.f[F_MASS][i]));
    const float om = toFloatRN(F.f[F_OMEGA][i]);
    const float4 th = make_float4(toFloatRN(rho), toFloatRN(p), cs, om / (om * om + 1.0e-30f));
    P.thermo[i] = th;
    if (ex.pair.on) P.pk[i] = pairRecord(th, ex.pair);
    if (TENSOR) writeTensorMirror(F, i, P, i);
    if (crk && P.vol) P.vol[i] = toFloatRN(F.f[F_VOL][i]);
  } else {
    eosNode(F, i, L);
  }
  if (ex.copyQ) {   // ArtificialViscosityHandle::postStateUpdate
    float v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double d = F.f[F_DVDX_XX + k][i];
      F.f[F_DVDXQ_XX + k][i] = d;
      v[k] = toFloatRN(d);
    }
    if (!TENSOR && ex.pair.on && ex.pair.limited) writeQGradient(P, i, v, ex.pair);
  }
  if (END) {
    double p[3] = {x, y, z};
    if (endNode(F, i, p, vx, vy, vz, F.f[F_MASS][i], rho, h, eps, HNew, TENSOR, g, bounds)) atomicExch(&ex.end->bad, 1);
  }
  }
  if (END) mergeBounds(bounds, TENSOR, ex.end);
}


// SpheralConservation totals (SpheralConservation.py:54-150) in FP64:
// mass, momentum, kinetic, thermal, gravitational (1/2 m phi).
__global__ void conservationKernel(Fields F, long n, int gravity, double* __restrict__ part) {
  __shared__ double sm[32];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double m = F.f[F_MASS][i], vx = F.f[F_VX][i], vy = F.f[F_VY][i], vz = F.f[F_VZ][i];
    acc[0] += m;
    acc[1] += m * vx; acc[2] += m * vy; acc[3] += m * vz;
    acc[4] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
    acc[5] += m * F.f[F_EPS][i];
    if (gravity) acc[6] += 0.5 * m * F.f[F_POT][i];
  }
  for (int k = 0; k < 7; ++k) {
    const double r = blockSum(acc[k], sm);
    if (threadIdx.x == 0) part[blockIdx.x * 7 + k] = r;
  }
}
__global__ void conservationFinalKernel(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double sm[32];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    for (int k = 0; k < 7; ++k) acc[k] += part[b * 7 + k];
  for (int k = 0; k < 7; ++k) {
    const double r = blockSum(acc[k], sm);
    if (threadIdx.x == 0) out[k] = r;
  }
  if (threadIdx.x == 0) out[7] = out[4] + out[5] + out[6];
}

// Caller-order transfers: stage[orig[k] * stride + c] <-> F[first + c][k].
__global__ void gatherOutKernel(Fields F, const int* __restrict__ orig, double* __restrict__ stage, int first,
                                int ncomp, int stride, long n) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const long o = (long)orig[k] * stride;
  for (int c = 0; c < ncomp; ++c) stage[o + c] = F.f[first + c][k];
}
// Domain-decomposition exchange: rows of `w` values of the fields ids[0..w)
// for caller indices idx (get), or for the halo nodes, caller indices
// nOwn..nOwn+count-1 in order (put).  inv: internal index of each caller index.
__global__ void exchangeGetKernel(Fields F, const int* __restrict__ inv, const int* __restrict__ idx, long count,
                                  ExchangeFields ef, double* __restrict__ out) {
  const long r = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (r >= count) return;
  const long k = inv[idx[r]];
  for (int c = 0; c < ef.w; ++c) out[r * ef.w + c] = F.f[ef.ids[c]][k];
}
__global__ void exchangePutKernel(Fields F, Fields32 P, const int* __restrict__ inv, long nOwn, long count,
                                  ExchangeFields ef, const double* __restrict__ in) {
  const long r = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (r >= count) return;
  const long k = inv[nOwn + r];
  for (int c = 0; c < ef.w; ++c) F.f[ef.ids[c]][k] = in[r * ef.w + c];
  // the FP32 mirror entries the sweeps read next, written as their own
  // kernels write them for owned nodes
  if (P.thermo) {
    if (ef.mirror == 1) P.thermo[k].x = (float)F.f[F_RHO][k];
    if (ef.mirror == 2) {
      const float om = (float)F.f[F_OMEGA][k];
      P.thermo[k].w = om / (om * om + 1.0e-30f);
    }
  }
}

__global__ void scatterInKernel(Fields F, const int* __restrict__ orig, const double* __restrict__ stage, int first,
                                int ncomp, int stride, long n) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const long o = (long)orig[k] * stride;
  for (int c = 0; c < ncomp; ++c) F.f[first + c][k] = stage[o + c];
}
// Caller-order transfers that address a pinned host array in place: the
// threads walk the flat host array (n records of `stride` doubles), so the
// host link sees contiguous reads (writes), and the permutation to the
// internal order (inv: caller index -> internal index) lands on the device
// side.  Components past ncomp are skipped on the way in; on the way out an
// isotropic H (isoH) is written as the SymTensor (a, 0, 0, a, 0, a).
__global__ void inverseOrderKernel(const int* __restrict__ orig, int* __restrict__ inv, long n) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < n) inv[orig[k]] = (int)k;
}
__global__ void scatterInHostKernel(Fields F, const int* __restrict__ inv, HostBatch batch, long n) {
  const HostBatch::Item it = batch.it[blockIdx.y];
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= n * it.stride) return;
  const long m = e / it.stride;
  const int c = (int)(e - m * it.stride);
  if (c < it.ncomp) F.f[it.first + c][inv[m]] = it.host[e];
}
__global__ void gatherOutHostKernel(Fields F, const int* __restrict__ inv, HostBatch batch, long n) {
  const HostBatch::Item it = batch.it[blockIdx.y];
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= n * it.stride) return;
  const long m = e / it.stride;
  const int c = (int)(e - m * it.stride);
  double v;
  if (it.isoH) v = (c == 0 || c == 3 || c == 5) ? F.f[it.first][inv[m]] : 0.0;
  else v = c < it.ncomp ? F.f[it.first + c][inv[m]] : 0.0;
  it.host[e] = v;
}
// H as SymTensor (xx, xy, xz, yy, yz, zz) <-> isotropic hinv.
__global__ void gatherOutHKernel(Fields F, const int* __restrict__ orig, double* __restrict__ stage, int field,
                                 long n) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  double* o = stage + (long)orig[k] * 6;
  const double a = F.f[field][k];
  o[0] = a; o[1] = 0.0; o[2] = 0.0; o[3] = a; o[4] = 0.0; o[5] = a;
}
__global__ void countsOutKernel(const int* __restrict__ counts, const int* __restrict__ orig,
                                double* __restrict__ stage, long n) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  stage[orig[k]] = (double)counts[k];
}

inline unsigned gridFor(long n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

//==============================================================================
// Launchers
//==============================================================================
void launchBounds(const Fields& F, long n, bool tensor, StepScratch* sc, cudaStream_t s, LaunchCounter* lc) {
  resetScratchKernel<<<1, 1, 0, s>>>(sc);
  boundsKernel<<<std::min(gridFor(n, 256), 1216u), 256, 0, s>>>(F, n, tensor ? 1 : 0, sc);
  lc->add(2);
}
void launchCellKeys(const Fields& F, long n, Grid g, uint32_t* keys, int* vals, uint32_t* cellc, StepScratch* sc,
                    const SortPrep& prep, unsigned* ranges, long long nranges, cudaStream_t s, LaunchCounter* lc) {
  // at most 8 blocks per SM: each adds its digit counts to the global ones
  cellKeyKernel<<<std::min(gridFor(n, 256), 1216u), 256, 0, s>>>(F, n, g, keys, vals, cellc, sc, prep, ranges, nranges);
  lc->add(1);
}
// FP32 mirror of the Q's DvDx for the mixed pair sweep.
__global__ void qGradient32Kernel(Fields F, float4* __restrict__ dvq, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) v[k] = (float)F.f[F_DVDXQ_XX + k][i];
  dvq[i] = make_float4(v[0], v[1], v[2], v[3]);
  dvq[n + i] = make_float4(v[4], v[5], v[6], v[7]);
  dvq[2 * n + i] = make_float4(v[8], 0.0f, 0.0f, 0.0f);
}
void launchQGradient32(Fields F, float4* dvq, long n, cudaStream_t s, LaunchCounter* lc) {
  qGradient32Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, dvq, n);
  lc->add(1);
}
// 3375 nodes 17.9 us in one row of blocks, 10.6 in nine; 2.1 M nodes 292 in one,
// 303 in four.
constexpr long kSplitPermute = 200000;
void launchPermute(const Fields& Fin, Fields Fout, const int* perm, const int* origIn, int* origOut,
                   const int* listIn, int* listOut, const uint32_t* cellIn, uint32_t* cellOut, long n,
                   bool carriedOnly, bool tensor, bool crk, bool limitedQ, Fields32 P, const Grid& g,
                   bool mirrors, const uint32_t* sortedKeys, uint32_t space, int* cellStart, int* cellEnd, const SortPrep& prep,
                   cudaStream_t s, LaunchCounter* lc) {
  // the tensor-H fields (the end of the carried block and of the permuted
  // block) move only in ASPH mode, the RK volume and corrections (the end of
  // the permuted block) only in CRKSPH mode
  FieldRanges sel{};
  auto add = [&](int a, int b) { sel.first[sel.n] = a; sel.last[sel.n] = b; ++sel.n; };
  if (carriedOnly) {
    // of DvDx the vote reads the trace, the limited Q all of it
    if (limitedQ) {
      add(0, F_GRAV_X);
    } else {
      add(0, F_DVDX_XX + 1);
      add(F_DVDX_YY, F_DVDX_YY + 1);
      add(F_DVDX_ZZ, F_DVDX_ZZ + 1);
    }
    add(F_GRAV_X, tensor ? (int)F_NUM_CARRIED : (int)F_HT_XX);
  } else {
    add(0, tensor ? (int)F_NUM_CARRIED : (int)F_HT_XX);
    add(F_NUM_CARRIED, tensor ? (int)F_VOL : (int)F_HIDEALT_XX);
    if (crk) add(F_VOL, F_NUM_PERMUTED);
  }
  // a few blocks leave the SMs idle: spread the fields over more
  const dim3 grid(gridFor(n, 256), n < kSplitPermute ? 9 : 1);
  permuteKernel<<<grid, 256, 0, s>>>(Fin, Fout, perm, origIn, origOut, listIn, listOut, cellIn, cellOut, n,
                                                sel, P, g, mirrors ? 1 : 0, sortedKeys, space, cellStart, cellEnd, prep);
  lc->add(1);
}
void launchItems(const uint32_t* sortedKeys, long n, int shift, uint32_t space, const int* cellEnd, int width,
                 int nItemsBound, Grid g, bool tensor, Fields32 P, int* items, int* chunkOf, int* counts, float4* box,
                 StepScratch* sc, cudaStream_t s, LaunchCounter* lc) {
  itemsKernel<<<gridFor(n, 256), 256, 0, s>>>(sortedKeys, n, shift, space, cellEnd, width, items, chunkOf, counts, sc);
  const unsigned gb = gridFor((long)nItemsBound * width, 128);
#define SPH_BOX(W, T) itemBoxKernel<W, T><<<gb, 128, 0, s>>>(items, sc, n, g, P, box, box + 2 * n)
#define SPH_BOXW(T) do { if (width == 8) SPH_BOX(8, T); else if (width == 16) SPH_BOX(16, T); else SPH_BOX(32, T); } while (0)
  if (tensor) SPH_BOXW(true);
  else SPH_BOXW(false);
#undef SPH_BOXW
#undef SPH_BOX
  lc->add(2);
}
// Band of the FP32 pre-filter on e2 = min(a_i, a_j)^2 r^2 around ext^2
// (a = 1/h).  Every cell-relative coordinate is within about one cell size C
// of its cell origin, so each FP32 separation component carries at most
// ~10 u C of rounding (u = 2^-24: the cell-relative positions, the mirror,
// the difference and the periodic offset), and near the threshold
// (a r ~ ext) |e2_fp32 - e2| <= ext^2 (20 sqrt(3) u C a / ext + 7 u).  The
// band used is four times that bound, evaluated with a = a_i >= min(a_i, a_j):
// delta_i = bandA a_i + bandB.  A node whose delta reaches 1/2 takes the exact
// test on every candidate.
// Items below which four warps share one: 30,011 nodes 92 us with four warps,
// 134 with one; 103,924 nodes 129 us with four, 89 with one.
constexpr int kWideItems = 2400;
static void neighborBand(const Grid& g, double ext2, float& bandA, float& bandB) {
  const double u = 1.0 / 16777216.0;
  const double cmax = std::max(g.cell[0], std::max(g.cell[1], g.cell[2]));
  const double ext = std::sqrt(ext2);
  bandA = (float)(4.0 * 20.0 * std::sqrt(3.0) * u * cmax / ext);
  bandB = (float)(4.0 * 7.0 * u);
}
// Tensor H (ASPH); the isotropic FP64 sweeps are in hydro64.cu.
void launchSumDensity(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                      cudaStream_t s, LaunchCounter* lc) {
  const size_t sm = sizeof(double) * 3 * (hp.tableN1 + 1);
  sumDensityKernel<<<gridFor(n, 128), 128, sm, s>>>(F, list, n, g, nl, t, hp);
  lc->add(1);
}
void launchGradh(Fields F, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp, cudaStream_t s,
                 LaunchCounter* lc) {
  const size_t sm = sizeof(double) * 6 * (hp.tableN1 + 1);
  gradhKernel<<<gridFor(n, 128), 128, sm, s>>>(F, n, g, nl, t, hp);
  lc->add(1);
}
void launchPairFP64(Fields F, const int* list, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                    double* pacc, cudaStream_t s, LaunchCounter* lc) {
  const size_t sm = sizeof(double) * 6 * (hp.tableN1 + 1);
  const int b = 128;
#define SPH_PAIR64(X, C) pairKernelFP64<X, C><<<gridFor(n, b), b, sm, s>>>(F, list, n, g, nl, t, hp, pacc)
  if (hp.xsph) {
    if (hp.compatible) SPH_PAIR64(true, true); else SPH_PAIR64(true, false);
  } else {
    if (hp.compatible) SPH_PAIR64(false, true); else SPH_PAIR64(false, false);
  }
#undef SPH_PAIR64
  lc->add(1);
}
void launchDt(Fields F, const int* list, long n, Grid g, NeighborLists nl, HydroParams hp,
              double maxNperh, double* dScratch, int nScratch, double* dOut,
              cudaStream_t s, LaunchCounter* lc) {
  const int nb = (int)gridFor(n, 128);
  (void)nScratch;
  dtKernel<<<nb, 128, 0, s>>>(F, list, n, g, nl, hp, maxNperh, dScratch);
  dtFinalKernel<<<1, 256, 0, s>>>(dScratch, nb, dOut);
  lc->add(2);
}
void launchRadius0(Fields F, long n, cudaStream_t s, LaunchCounter* lc) {
  radius0Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, n);
  lc->add(1);
}
void launchTensorExtent(Fields F, long n, cudaStream_t s, LaunchCounter* lc) {
  tensorExtentKernel<<<gridFor(n, 256), 256, 0, s>>>(F, n);
  lc->add(1);
}
void launchUpdate(Fields F, const int* list, long n, HydroParams hp, double mult, bool mid, bool gravity,
                  const Fields32* mirror, const Grid& g, const UpdateExtras& ex, cudaStream_t s, LaunchCounter* lc) {
  const int epsInc = (mid || !hp.compatible) ? 1 : 0;
  Fields32 P{};
  if (mirror) P = *mirror;
#define SPH_UPD(T, E, CRK, AE, FS, RO)                                                                              \
  updateKernel<T, E><<<gridFor(n, 256), 256, 0, s>>>(F, list, n, hp.lists, mult, mid ? 1 : 0, gravity ? 1 : 0,     \
                                                     epsInc, hp.hUpdate, hp.totalEnergy, CRK, P, g, AE, FS, RO, ex)
  if (hp.asph) {
    if (ex.end) SPH_UPD(true, true, 0, hp.asphEnd, hp.fixShape, hp.radialOnly);
    else SPH_UPD(true, false, 0, hp.asphEnd, hp.fixShape, hp.radialOnly);
  } else {
    if (ex.end) SPH_UPD(false, true, hp.crk, 0, 0, 0);
    else SPH_UPD(false, false, hp.crk, 0, 0, 0);
  }
#undef SPH_UPD
  lc->add(1);
}
void launchASPHEnd(Fields F, Fields32 P, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                   HydroParams hp, cudaStream_t s, LaunchCounter* lc) {
  const size_t smem = 3 * (size_t)(hp.tableN1 + 1) * sizeof(double);
  asphEndKernel<<<gridFor(n, 128), 128, smem, s>>>(F, P, list, n, g, nl, t, hp);
  lc->add(1);
}
void launchEOS(Fields F, const int* list, long n, const NodeListParams* lists, cudaStream_t s, LaunchCounter* lc) {
  eosKernel<<<gridFor(n, 256), 256, 0, s>>>(F, list, n, lists);
  lc->add(1);
}
void launchEndStep(Fields F, long n, Grid g, bool tensor, StepScratch* sc, cudaStream_t s, LaunchCounter* lc) {
  // at most 8 blocks per SM, each thread over several nodes: ten reductions and
  // atomics per block, not per node
  endStepKernel<<<std::min(gridFor(n, 256), 1216u), 256, 0, s>>>(F, n, g, tensor ? 1 : 0, sc);
  lc->add(1);
}
void launchConservation(Fields F, long n, bool gravity, double* dScratch, int nScratch, double* dOut, cudaStream_t s,
                        LaunchCounter* lc) {
  int nb = (int)std::min<long>((n + 255) / 256, nScratch / 7);
  if (nb < 1) nb = 1;
  conservationKernel<<<nb, 256, 0, s>>>(F, n, gravity ? 1 : 0, dScratch);
  conservationFinalKernel<<<1, 256, 0, s>>>(dScratch, nb, dOut);
  lc->add(2);
}
void launchExchangeGet(Fields F, const int* inv, const int* idx, long count, ExchangeFields ef, double* out,
                       cudaStream_t s, LaunchCounter* lc) {
  if (count <= 0) return;
  exchangeGetKernel<<<gridFor(count, 256), 256, 0, s>>>(F, inv, idx, count, ef, out);
  lc->add(1);
}
void launchExchangePut(Fields F, Fields32 P, const int* inv, long nOwn, long count, ExchangeFields ef,
                       const double* in, cudaStream_t s, LaunchCounter* lc) {
  if (count <= 0) return;
  exchangePutKernel<<<gridFor(count, 256), 256, 0, s>>>(F, P, inv, nOwn, count, ef, in);
  lc->add(1);
}

void launchGatherOut(Fields F, const int* orig, double* stage, int first, int ncomp, int stride, long n,
                     cudaStream_t s, LaunchCounter* lc) {
  gatherOutKernel<<<gridFor(n, 256), 256, 0, s>>>(F, orig, stage, first, ncomp, stride, n);
  lc->add(1);
}
void launchScatterIn(Fields F, const int* orig, const double* stage, int first, int ncomp, int stride, long n,
                     cudaStream_t s, LaunchCounter* lc) {
  scatterInKernel<<<gridFor(n, 256), 256, 0, s>>>(F, orig, stage, first, ncomp, stride, n);
  lc->add(1);
}
void launchInverseOrder(const int* orig, int* inv, long n, cudaStream_t s, LaunchCounter* lc) {
  inverseOrderKernel<<<gridFor(n, 256), 256, 0, s>>>(orig, inv, n);
  lc->add(1);
}
void launchScatterInHost(Fields F, const int* inv, const HostBatch& batch, long n, cudaStream_t s, LaunchCounter* lc) {
  if (batch.count == 0) return;
  scatterInHostKernel<<<dim3(gridFor(n * batch.maxStride, 256), batch.count), 256, 0, s>>>(F, inv, batch, n);
  lc->add(1);
}
void launchGatherOutHost(Fields F, const int* inv, const HostBatch& batch, long n, cudaStream_t s, LaunchCounter* lc) {
  if (batch.count == 0) return;
  gatherOutHostKernel<<<dim3(gridFor(n * batch.maxStride, 256), batch.count), 256, 0, s>>>(F, inv, batch, n);
  lc->add(1);
}
void launchGatherOutH(Fields F, const int* orig, double* stage, int field, long n, cudaStream_t s, LaunchCounter* lc) {
  gatherOutHKernel<<<gridFor(n, 256), 256, 0, s>>>(F, orig, stage, field, n);
  lc->add(1);
}
void launchCountsOut(const int* counts, const int* orig, double* stage, long n, cudaStream_t s, LaunchCounter* lc) {
  countsOutKernel<<<gridFor(n, 256), 256, 0, s>>>(counts, orig, stage, n);
  lc->add(1);
}

void launchNeighborsWarp(const Fields& F, Fields32 P, long n, const int* items, int nItems, StepScratch* sc,
                         int width, Grid g, const int* cellStart, const int* cellEnd, int* counts, uint32_t* nbr, int cap, double ext2, bool tensor, const float4* box, const int* chunkOf,
                         cudaStream_t s, LaunchCounter* lc) {
  float lo, hi;
  neighborBand(g, ext2, lo, hi);
  // four warps per item while the items alone would leave SMs idle (below
  // ~16 items per SM), one warp above
  const bool wide = nItems < kWideItems;
  const unsigned gb = wide ? (unsigned)nItems : (unsigned)((nItems + 3) / 4);
#define SPH_NBM(WR, CW, TE)                                                                                      \
  neighborMaskKernel<WR, CW, TE><<<gb, 128, 0, s>>>(F, P, items, nItems, width, g, cellStart, cellEnd, counts, \
                                                    WR ? nbr : nullptr, ext2, lo, hi, WR ? cap : 0, sc, box, box + 2 * n, chunkOf)
#define SPH_NBW(WR, TE) do { if (wide) SPH_NBM(WR, 4, TE); else SPH_NBM(WR, 1, TE); } while (0)
  if (nbr) { if (tensor) SPH_NBW(true, true); else SPH_NBW(true, false); }
  else { if (tensor) SPH_NBW(false, true); else SPH_NBW(false, false); }
#undef SPH_NBW
#undef SPH_NBM
  lc->add(1);
}

}  // namespace sph
