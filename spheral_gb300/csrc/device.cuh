// Device helpers shared by the FP64 (hydro.cu) and FP32 (hydro32.cu) sweeps.
#pragma once
#include "kernels.cuh"
#include <cfloat>
#include "tensor.cuh"

namespace sph {
namespace dev {

constexpr double kTiny30 = 1.0e-30;

// Kahan-compensated FP32 accumulation (explicit round-to-nearest so the
// compensation survives contraction); the pair leaves as the FP64 value s - c.
__device__ __forceinline__ void kahanAdd(float& s, float& c, float x) {
  const float y = __fsub_rn(x, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}
__device__ __forceinline__ double kahanValue(float s, float c) { return (double)s - (double)c; }
// The same accumulation, or a plain FP32 sum when `plain` (uniform per launch).
__device__ __forceinline__ void sumAdd(float& s, float& c, float x, int plain) {
  if (plain) s = __fadd_rn(s, x);
  else kahanAdd(s, c, x);
}

// eta from eta^2 in the FP32 sweeps: eta^2 times its reciprocal square root
// (the hardware approximation; eta^2 = 0 gives 0), as the pair kernel forms
// its eta_i and eta_j; the density/dt and grad-h sweeps use it too.
__device__ __forceinline__ float etaFromSq(float e2) { return __fmul_rn(e2, rsqrtf(fmaxf(e2, 1.0e-30f))); }

//------------------------------------------------------------------------------
// Lanes per node of the mixed-mode sweeps.  L consecutive lanes of a warp
// share one node: lane l takes the list slots l, l + L, ..., and the partial
// sums are combined by shuffles.
//------------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ float laneSum(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int L>
__device__ __forceinline__ float laneMax(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Compensated partial sums s - c: the rounding error of every addition of
// two partial sums goes into the compensation (TwoSum), so the total keeps
// the accuracy of the parts.
template <int L>
__device__ __forceinline__ void laneSumKahan(float& s, float& c) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o), c2 = __shfl_xor_sync(0xffffffffu, c, o);
    const float t = __fadd_rn(s, s2);
    const float b = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(s2, b));
    c = __fsub_rn(__fadd_rn(c, c2), err);
    s = t;
  }
}

// The cubic B-spline and its derivative in registers, without the volume
// normalisation A = 1/pi (kSplineA), which the sweeps apply once per node so
// that the rounding of A does not bias every term:
//   eta < 1: W/A = 1 - 3/2 eta^2 + 3/4 eta^3,  W'/A = -(3 - 9/4 eta) eta
//   eta < 2: W/A = 1/4 (2 - eta)^3,            W'/A = -3/4 (2 - eta)^2
// The interpolation table of this kernel (500 intervals) agrees with it to
// ~1e-9, far below FP32 rounding, and costs two shared-memory gathers with
// bank conflicts per lookup; the other kernels and caller tables use the
// packed table.
constexpr double kSplineA = 0.31830988618379067154;
__device__ __forceinline__ float bsplineGrad(float eta) {
  const float d = fmaxf(2.0f - eta, 0.0f);
  const float in = __fmul_rn(eta, __fmaf_rn(2.25f, eta, -3.0f));
  const float out = __fmul_rn(d, __fmul_rn(-0.75f, d));
  return eta < 1.0f ? in : out;
}
__device__ __forceinline__ float bsplineW(float eta) {
  const float d = fmaxf(2.0f - eta, 0.0f);
  const float in = __fmaf_rn(__fmul_rn(eta, eta), __fmaf_rn(0.75f, eta, -1.5f), 1.0f);
  const float out = __fmul_rn(__fmul_rn(d, d), __fmul_rn(0.25f, d));
  return eta < 1.0f ? in : out;
}
// x times A for one FP32 value per node (A as an unevaluated float pair).
__device__ __forceinline__ float timesSplineA(float x) {
  constexpr float hi = (float)kSplineA, lo = (float)(kSplineA - (double)(float)kSplineA);
  return __fmaf_rn(x, hi, __fmul_rn(x, lo));
}

__device__ __forceinline__ void resetVote(StepScratch* sc) {
  sc->voteKey = ~0ULL;
  for (int k = 0; k < kDtReasons; ++k) sc->votes[k] = ~0ULL;
  sc->voteEst = 0x7f7fffffu;   // FLT_MAX
}
__device__ __forceinline__ void resetScratch(StepScratch* sc) {
  for (int k = 0; k < 4; ++k) sc->bounds[k] = 0x7fffffffffffffffLL;
  for (int k = 4; k < 10; ++k) sc->bounds[k] = k < 7 ? (long long)0x8000000000000000ULL : 0LL;
  sc->bad = sc->sortTimeout = sc->maxCount = sc->items = 0;
  for (int k = 0; k < kEntrySums; ++k) sc->entries[k] = 0ULL;
  resetVote(sc);
}

__device__ __forceinline__ void lookupPacked(const float4* __restrict__ ta, const float2* __restrict__ tb, int N1,
                                             float invStep, float eta, float extent, float& w, float& gr) {
  if (eta < extent) {
    const int k = min(N1, (int)(eta * invStep));
    const float4 A = ta[k];
    const float2 B = tb[k];
    w = __fmaf_rn(__fmaf_rn(A.z, eta, A.y), eta, A.x);
    gr = __fmaf_rn(__fmaf_rn(B.y, eta, B.x), eta, A.w);
  } else {
    w = 0.0f;
    gr = 0.0f;
  }
}

// The packed table in shared memory with a zero interval behind it: an eta at
// or beyond the extent reads zeros, no branch.
constexpr int kTab32 = kMaxTable / 3 + 1;
__device__ __forceinline__ void loadTable32(float4* ta, float2* tb, const TableDev& t, int N1) {
  for (int k = threadIdx.x; k <= N1 + 1; k += blockDim.x) {
    ta[k] = k <= N1 ? t.p32a[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (tb) tb[k] = k <= N1 ? t.p32b[k] : make_float2(0.f, 0.f);
  }
}

// W and W' of the sweeps: KERN 1 the cubic B-spline over A in registers, 0
// the packed table.
template <int KERN>
struct Kernel32 {
  const float4* ta;
  const float2* tb;
  int N1;
  float invStep;
  __device__ __forceinline__ int index(float eta) const { return min(N1 + 1, (int)(eta * invStep)); }
  __device__ __forceinline__ float value(float eta) const {
    if (KERN) return bsplineW(eta);
    const float4 A = ta[index(eta)];
    return __fmaf_rn(__fmaf_rn(A.z, eta, A.y), eta, A.x);
  }
  __device__ __forceinline__ void both(float eta, float& w, float& g) const {
    if (KERN) {
      w = bsplineW(eta);
      g = bsplineGrad(eta);
    } else {
      const int k = index(eta);
      const float4 A = ta[k];
      const float2 B = tb[k];
      w = __fmaf_rn(__fmaf_rn(A.z, eta, A.y), eta, A.x);
      g = __fmaf_rn(__fmaf_rn(B.y, eta, B.x), eta, A.w);
    }
  }
  __device__ __forceinline__ float grad(float eta) const {
    if (KERN) return bsplineGrad(eta);
    const int k = index(eta);
    const float2 B = tb[k];
    return __fmaf_rn(__fmaf_rn(B.y, eta, B.x), eta, ta[k].w);
  }
};

// Block size of the light sweeps.  With one lane per node a block of 512
// consecutive nodes shares most of its neighbours, so more of its gathers hit
// L1 than those of four separate blocks of 128 (2.1 M nodes: density/dt 1162 ->
// 1029 us, energy 892 -> 860); small problems need the finer blocks to spread.
__host__ __device__ constexpr int sweepBlock(int lanes) { return lanes == 1 ? 512 : 128; }

// Lanes per node.  One lane per node leaves the GPU idle below ~300,000 nodes
// (152 SMs x 16-20 resident warps of 32 nodes), and several lanes cost the
// shuffles and the partly filled last slots.  The lines lie where the times cross
// (boxes of 57 and, in brackets, 115 neighbours), us with 1 / 2 / 4 / 8 / 16:
//   pair    2,744 18/16/14/14/16   13,824 20/20/18/28/39 (26/24/21/34/47)
//           39,304 36/37/41/57/96 (52/52/52/71/122; with walls or the limited Q
//           four lanes lead by 1 % of the step)   97,336 69/68/83/127/227 (96/95/109)
//   density 4,096 33/23/16/12/12   17,576 36/24/16/14/18   39,304 38/25/18/23/29
//           97,336 43/29/33/41/55   148,877 43/51/47/57/83
//   energy  5,832 25/13/10/10/10   13,824 25/14/11/12/19   39,304 27/18/18/25/35
//           (47/29/27/35/54)   64,000 29/33/37/49/74   148,877 49/55/61/78/121
constexpr long kCRKOneLane = 100000;   // from here one lane per node in the CRKSPH pair sweep
constexpr long kExactNodes = 150000;   // node count from which the mixed sweeps keep the earlier arithmetic
inline int lanesPair(long n) { return n >= 80000 ? 2 : 4; }
inline int lanesSweep(long n) { return n >= kExactNodes ? 1 : (n >= 20000 ? 4 : (n >= 6000 ? 8 : 16)); }
inline int lanesEnergy(long n) { return n >= kExactNodes ? 1 : (n >= 40000 ? 2 : (n >= 6000 ? 4 : 16)); }

#define SPH_BY_LANES(L, CALL)      \
  switch (L) {                     \
    case 1: CALL(1); break;        \
    case 4: CALL(4); break;        \
    case 8: CALL(8); break;        \
    default: CALL(16); break;      \
  }

// Velocity of a mirror image: the components along the mirrored axes flip
// (mir: per-axis bits of the entry's cell-offset code that cross a wall).
__device__ __forceinline__ void mirrorVel(uint32_t mir, float& vx, float& vy, float& vz) {
  if (mir) {
    if (mir & 3u) vx = -vx;
    if (mir & 12u) vy = -vy;
    if (mir & 48u) vz = -vz;
  }
}

// Warp-interleaved neighbour storage: slot q of node i lives at
// ((i / 32) * cap + q) * 32 + i % 32, so a warp reading slot q of its 32 nodes
// touches one contiguous 128-byte line.
__device__ __forceinline__ long long nbSlot(long i, int q, int cap) {
  return ((long long)(i >> 5) * cap + q) * 32 + (i & 31);
}

// FP32 pair accelerations: the three components of a list slot sit in three
// 32-wide planes per slot row, so a warp writing (reading) one component of
// slot q of its 32 nodes touches one 128-byte line.  paccSlot(nbSlot(..)) is
// the x component; y is 32 floats further, z 64.
__device__ __forceinline__ long long paccSlot(long long slot) { return (slot >> 5) * 96 + (slot & 31); }

// Walk the list slots of node i that belong to lane `sub` of its L lanes, in
// list order, U slots per iteration: load(j, rec) gathers a neighbour's
// record, slot(entry, rec) evaluates it.  The U gathers of an iteration are
// issued together and the next iteration's entries are loaded before they are
// used.
template <int L, int U, class Rec, class Load, class Slot>
__device__ __forceinline__ void laneSlots(const NeighborLists& nl, long i, int sub, int cnt, Load load, Slot slot) {
  constexpr int ST = 32 * L;
  const int mine = (cnt - sub + L - 1) / L;
  const uint32_t* __restrict__ nb = nl.nbr + nbSlot(i, 0, nl.cap) + 32 * sub;
  uint32_t nx[U];
#pragma unroll
  for (int u = 0; u < U; ++u) nx[u] = u < mine ? nb[u * ST] : 0u;
  int q = 0;
  for (; q + U <= mine; q += U) {
    uint32_t e[U];
    Rec rec[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = nx[u];
#pragma unroll
    for (int u = 0; u < U; ++u) load(e[u] & kIndexMask, rec[u]);
    nb += U * ST;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q + U + u < mine) nx[u] = nb[u * ST];
#pragma unroll
    for (int u = 0; u < U; ++u) slot(e[u], rec[u]);
  }
#pragma unroll
  for (int u = 0; u < U - 1; ++u)
    if (q + u < mine) {
      Rec rec;
      load(nx[u] & kIndexMask, rec);
      slot(nx[u], rec);
    }
}

__device__ __forceinline__ void unpackCell(uint32_t cc, int c[3]) {
  c[0] = (int)(cc & 1023u);
  c[1] = (int)((cc >> 10) & 1023u);
  c[2] = (int)((cc >> 20) & 1023u);
}

// Image code (2 bits per axis: 0 none, 1 low side, 2 high side) of a
// neighbour entry with cell-offset code dcode seen from home cell c.
__device__ __forceinline__ int imageCode(const Grid& g, const int c[3], int dcode) {
  int code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int d = (dcode >> (2 * a)) & 3;
    if (d == 1 && c[a] == 0) code |= 1 << (2 * a);
    else if (d == 2 && c[a] == g.nc[a] - 1) code |= 2 << (2 * a);
  }
  return code;
}

// Per-axis bits (dcode layout) of the offsets that cross a reflecting wall
// from home cell c: those neighbour entries are mirror images.
__device__ __forceinline__ uint32_t mirrorMask(const Grid& g, const int c[3]) {
  uint32_t m = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (c[a] == 0 && g.kindLo[a] == AXIS_REFLECT) m |= 1u << (2 * a);
    if (c[a] == g.nc[a] - 1 && g.kindHi[a] == AXIS_REFLECT) m |= 2u << (2 * a);
  }
  return m;
}

// Whether any wall of the grid reflects (host): the sweeps' forms without
// mirror images serve every other grid.
inline bool hasMirrors(const Grid& g) {
  for (int a = 0; a < 3; ++a)
    if (g.kindLo[a] == AXIS_REFLECT || g.kindHi[a] == AXIS_REFLECT) return true;
  return false;
}

// FP32 mirrors of the node stored at F.f[.][i], into slot k.  The conversions
// take the integer pipe (the FP64 pipe bounds the callers otherwise) and
// omega / (omega^2 + 1e-30) is formed in FP32.  full false: only what the
// neighbour search reads.
__device__ __forceinline__ void writeMirrors(const Fields& F, long i, const Fields32& P, long k, uint32_t cell,
                                             const Grid& g, bool full) {
  int c[3];
  unpackCell(cell, c);
  const double ox = g.lo[0] + smallIntToDouble(c[0]) * g.cell[0];
  const double oy = g.lo[1] + smallIntToDouble(c[1]) * g.cell[1];
  const double oz = g.lo[2] + smallIntToDouble(c[2]) * g.cell[2];
  P.posh[k] = make_float4(toFloatRN(F.f[F_X][i] - ox), toFloatRN(F.f[F_Y][i] - oy), toFloatRN(F.f[F_Z][i] - oz),
                          toFloatRN(F.f[F_HINV][i]));
  if (P.hten) writeTensorMirror(F, i, P, k);
  if (!full) return;
  P.velm[k] = make_float4(toFloatRN(F.f[F_VX][i]), toFloatRN(F.f[F_VY][i]), toFloatRN(F.f[F_VZ][i]),
                          toFloatRN(F.f[F_MASS][i]));
  const float om = toFloatRN(F.f[F_OMEGA][i]);
  P.thermo[k] = make_float4(toFloatRN(F.f[F_RHO][i]), toFloatRN(F.f[F_P][i]), toFloatRN(F.f[F_CS][i]),
                            om / (om * om + 1.0e-30f));
  if (P.vol) P.vol[k] = toFloatRN(F.f[F_VOL][i]);
}

// FP32 separation r_i - r_j' on cell-relative coordinates: r = (x_i - x_j')
// - d cell per axis, with x_j' = cell - x_j for a mirror image.  Periodic
// images need no box arithmetic: the cell offset d of the list entry carries the
// wrap.  The offset per axis (0, +c, -c for codes 0, 1, 2) comes by integer
// selection: the sweeps are bound by shared-memory / L1 wavefronts (~11 per 16-byte gather), so a table of the
// offsets in shared memory costs more than these instructions.
// MIR false: no wall of the grid reflects, so no entry is a mirror image.
__device__ __forceinline__ float cellOffset(uint32_t ent, int axis, float c) {
  const uint32_t f = (ent >> (kIndexBits + 2 * axis)) & 3u;
  return __uint_as_float((f ? __float_as_uint(c) : 0u) ^ ((f & 2u) << 30));
}
template <bool MIR = true>
__device__ __forceinline__ void relSepEntry(const float4& pi, const float4& pj, uint32_t ent, uint32_t mm, float cx,
                                            float cy, float cz, float& rx, float& ry, float& rz) {
  float xj = pj.x, yj = pj.y, zj = pj.z;
  if (MIR) {
    const uint32_t mir = (ent >> kIndexBits) & mm;
    if (mir) {
      if (mir & 3u) xj = cx - xj;
      if (mir & 12u) yj = cy - yj;
      if (mir & 48u) zj = cz - zj;
    }
  }
  rx = __fadd_rn(__fsub_rn(pi.x, xj), cellOffset(ent, 0, cx));
  ry = __fadd_rn(__fsub_rn(pi.y, yj), cellOffset(ent, 1, cy));
  rz = __fadd_rn(__fsub_rn(pi.z, zj), cellOffset(ent, 2, cz));
}

__device__ __forceinline__ void imagePos(const Grid& g, int code, double& x, double& y, double& z) {
  if (code) {
    x = imageCoord(x, code & 3, g.kindLo[0], g.kindHi[0], g.wallLo[0], g.wallHi[0]);
    y = imageCoord(y, (code >> 2) & 3, g.kindLo[1], g.kindHi[1], g.wallLo[1], g.wallHi[1]);
    z = imageCoord(z, (code >> 4) & 3, g.kindLo[2], g.kindHi[2], g.wallLo[2], g.wallHi[2]);
  }
}
__device__ __forceinline__ void imageVec(const Grid& g, int code, double& x, double& y, double& z) {
  if (code) {
    if (mirrored(code & 3, g.kindLo[0], g.kindHi[0])) x = -x;
    if (mirrored((code >> 2) & 3, g.kindLo[1], g.kindHi[1])) y = -y;
    if (mirrored((code >> 4) & 3, g.kindLo[2], g.kindHi[2])) z = -z;
  }
}

// Tensor seen through the image: a mirror along axis a is R = I - 2 e_a e_a,
// and R T R flips every component with exactly one index on a mirrored axis.
__device__ __forceinline__ void imageTensor(const Grid& g, int code, double* T) {
  if (code) {
    const double s[3] = {mirrored(code & 3, g.kindLo[0], g.kindHi[0]) ? -1.0 : 1.0,
                         mirrored((code >> 2) & 3, g.kindLo[1], g.kindHi[1]) ? -1.0 : 1.0,
                         mirrored((code >> 4) & 3, g.kindLo[2], g.kindHi[2]) ? -1.0 : 1.0};
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) T[3 * r + c] *= s[r] * s[c];
  }
}

// QuadraticInterpolatorView lookup shared by W and dW/deta
// (src/Utilities/QuadraticInterpolatorViewInline.hh:17-21,71-77).
__device__ __forceinline__ int tableIndex(double eta, int N1, double xstep) {
  const long k = (long)(fmax(0.0, eta) / xstep);
  return 3 * (int)min((long)N1, k);
}
__device__ __forceinline__ double tableEval(const double* c, int i0, double x) {
  return c[i0] + (c[i0 + 1] + c[i0 + 2] * x) * x;
}

__device__ __forceinline__ double blockSum(double v, double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  return v;
}


__device__ __forceinline__ double hermiteLookup(const double* __restrict__ v, const HydroParams& hp, double x) {
  // CubicHermiteInterpolatorView::operator() (CubicHermiteInterpolatorViewInline.hh:10-36)
  const int N = hp.hermN;
  if (x < hp.hermXmin) return v[0] + v[N] * (x - hp.hermXmin);
  if (x > hp.hermXmax) return v[N - 1] + v[2 * N - 1] * (x - hp.hermXmin);
  long k = (long)(fmax(0.0, x - hp.hermXmin) / hp.hermXstep);
  const int i0 = (int)min((long)(N - 2), k);
  const double t = fmax(0.0, fmin(1.0, (x - hp.hermXmin - i0 * hp.hermXstep) / hp.hermXstep));
  const double t2 = t * t, t3 = t * t2;
  return ((2.0 * t3 - 3.0 * t2 + 1.0) * v[i0] + (-2.0 * t3 + 3.0 * t2) * v[i0 + 1] +
          hp.hermXstep * ((t3 - 2.0 * t2 + t) * v[N + i0] + (t3 - t2) * v[N + i0 + 1]));
}

// Per-node completion shared by the FP64 and FP32 pair kernels: self terms,
// corrected velocity gradient, continuity, XSPH, and the IdealH update.
struct NodeAcc {
  double rhoSum, norm, dvx, dvy, dvz, deps, gx, gy, gz, maxQ, effQ, xw, xdx, xdy, xdz, m0, m1x, m1y, m1z;
  double D[9], M[9];
  double m2[6];   // ASPH second moment (xx xy xz yy yz zz)
};

// SPH finalize (SPH.cc:480-552): self terms, the corrected velocity gradient,
// continuity and XSPH; D returns the final DvDx.
__device__ __forceinline__ void finalizeHydro(Fields& F, long i, const NodeAcc& a, double mi, double rhoi,
                                              double vxi, double vyi, double vzi, double Hdeti, int numNb,
                                              const HydroParams& hp, double* D) {
  F.f[F_RHOSUM][i] = a.rhoSum + mi * hp.W0 * Hdeti;
  F.f[F_NORM][i] = a.norm + mi / rhoi * hp.W0 * Hdeti;
  double Mm[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) { D[k] = a.D[k]; Mm[k] = a.M[k]; }
  const double detM = (Mm[0] * Mm[4] * Mm[8] + Mm[1] * Mm[5] * Mm[6] + Mm[2] * Mm[3] * Mm[7] -
                       Mm[0] * Mm[5] * Mm[7] - Mm[1] * Mm[3] * Mm[8] - Mm[2] * Mm[4] * Mm[6]);
  if (hp.correctVelGrad && fabs(detM) > 1.0e-10 && numNb > 8) {
    // GeomTensor<3>::Inverse (src/Geometry/GeomTensorInline.hh:1885-1890)
    const double inv[9] = {(Mm[4] * Mm[8] - Mm[5] * Mm[7]) / detM, (Mm[2] * Mm[7] - Mm[1] * Mm[8]) / detM,
                           (Mm[1] * Mm[5] - Mm[2] * Mm[4]) / detM, (Mm[5] * Mm[6] - Mm[3] * Mm[8]) / detM,
                           (Mm[0] * Mm[8] - Mm[2] * Mm[6]) / detM, (Mm[2] * Mm[3] - Mm[0] * Mm[5]) / detM,
                           (Mm[3] * Mm[7] - Mm[4] * Mm[6]) / detM, (Mm[1] * Mm[6] - Mm[0] * Mm[7]) / detM,
                           (Mm[0] * Mm[4] - Mm[1] * Mm[3]) / detM};
    double R[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        R[3 * r + c] = D[3 * r] * inv[c] + D[3 * r + 1] * inv[3 + c] + D[3 * r + 2] * inv[6 + c];
#pragma unroll
    for (int k = 0; k < 9; ++k) { D[k] = R[k]; Mm[k] = inv[k]; }
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] /= rhoi;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) { F.f[F_DVDX_XX + k][i] = D[k]; F.f[F_M_XX + k][i] = Mm[k]; }
  F.f[F_GRADRHO_X][i] = a.gx / rhoi;
  F.f[F_GRADRHO_Y][i] = a.gy / rhoi;
  F.f[F_GRADRHO_Z][i] = a.gz / rhoi;
  const double trace = D[0] + D[4] + D[8];
  F.f[F_DRHODT][i] = -rhoi * trace;
  F.f[F_DVDT_X][i] = a.dvx;
  F.f[F_DVDT_Y][i] = a.dvy;
  F.f[F_DVDT_Z][i] = a.dvz;
  // evolveTotalEnergy: the total-energy rate m (v . DvDt + DepsDt) (SPH.cc:541)
  F.f[F_DEPSDT][i] = hp.totalEnergy ? mi * ((vxi * a.dvx + vyi * a.dvy + vzi * a.dvz) + a.deps) : a.deps;
  F.f[F_MAXQ][i] = a.maxQ;
  F.f[F_EFFQ][i] = a.effQ;
  double xw = a.xw;
  if (hp.xsph) {
    xw += Hdeti * mi / rhoi * hp.W0;
    const double ws = fmax(kTiny30, xw);
    F.f[F_DXDT_X][i] = vxi + a.xdx / ws;
    F.f[F_DXDT_Y][i] = vyi + a.xdy / ws;
    F.f[F_DXDT_Z][i] = vzi + a.xdz / ws;
  } else {
    F.f[F_DXDT_X][i] = vxi;
    F.f[F_DXDT_Y][i] = vyi;
    F.f[F_DXDT_Z][i] = vzi;
  }
  F.f[F_XSPHW][i] = xw;
  F.f[F_XSPHDV_X][i] = a.xdx;
  F.f[F_XSPHDV_Y][i] = a.xdy;
  F.f[F_XSPHDV_Z][i] = a.xdz;
}

__device__ __forceinline__ void finalizeNode(Fields& F, long i, int li, const NodeAcc& a, double mi, double rhoi,
                                             double vxi, double vyi, double vzi, double ai, int numNb,
                                             const HydroParams& hp, const double* __restrict__ herm) {
  double D[9];
  finalizeHydro(F, i, a, mi, rhoi, vxi, vyi, vzi, (ai * ai) * ai, numNb, hp, D);
  const double trace = D[0] + D[4] + D[8];
  // SPHSmoothingScale finalize (SPHSmoothingScale.cc:235-270)
  const NodeListParams L = hp.lists[li];
  const double m0s = fmax(0.0, a.m0);
  const double m0 = m0s < 0.0 ? -pow(-m0s, 0.3333333333333333) : pow(m0s, 0.3333333333333333);
  F.f[F_M0][i] = m0;
  F.f[F_M1_X][i] = a.m1x;
  F.f[F_M1_Y][i] = a.m1y;
  F.f[F_M1_Z][i] = a.m1z;
  F.f[F_DHDT][i] = ((-ai) / 3.0) * trace;
  const bool iso = fabs(m0 - 0.0) <= 1.0e-15 * fmax(1.0, fabs(m0));
  const double cur = iso ? 0.5 * L.nPerh : fmax(0.0, hermiteLookup(herm, hp, m0));
  const double s = fmin(4.0, fmax(0.25, L.nPerh / (cur + 1.0e-30)));
  const double aa = s < 1.0 ? 0.4 * (1.0 + s * s) : 0.4 * (1.0 + 1.0 / (s * s * s));
  const double hi0 = 1.0 / ai;
  const double hi1 = fmin(L.hmax, fmax(L.hmin, hi0 * (1.0 - aa + aa * s)));
  F.f[F_HIDEAL][i] = 1.0 / hi1;
}


// ASPHClassicSmoothingScale node part (ASPHClassicSmoothingScale.cc:180-291):
// tensor DH/Dt and Hideal (asphClassicHideal) from the moments.
__device__ __forceinline__ void finalizeNodeASPH(Fields& F, long i, int li, const NodeAcc& a, const Sym& Hi,
                                                 double mi, double rhoi, double vxi, double vyi, double vzi,
                                                 int numNb, const HydroParams& hp, const double* __restrict__ herm) {
  double D[9];
  finalizeHydro(F, i, a, mi, rhoi, vxi, vyi, vzi, symDet(Hi), numNb, hp, D);
  const NodeListParams L = hp.lists[li];
  storeSym(F, F_DHDTT_XX, i, smoothingScaleDerivative(Hi, D));
  if (hp.asphEnd) return;   // ASPHSmoothingScale: the ideal H comes at the end of the step
  const double m0 = rootnu3T(fmax(0.0, a.m0));
  F.f[F_M0][i] = m0;
  F.f[F_M1_X][i] = a.m1x;
  F.f[F_M1_Y][i] = a.m1y;
  F.f[F_M1_Z][i] = a.m1z;
  const Sym M2{a.m2[0], a.m2[1], a.m2[2], a.m2[3], a.m2[4], a.m2[5]};
  storeSym(F, F_M2_XX, i, M2);
  const bool isolated = fabs(m0) <= 1.0e-15 * fmax(1.0, fabs(m0));
  const double cur = isolated ? 0.5 * L.nPerh : fmax(0.0, hermiteLookup(herm, hp, m0));
  const double s = fmin(4.0, fmax(0.25, L.nPerh / cur));
  double ev[3];
  symEigenValues(M2, ev);
  storeSym(F, F_HIDEALT_XX, i,
           asphClassicHideal(M2, fmin(ev[0], fmin(ev[1], ev[2])) > 0.0, Hi, s, hp.fixShape != 0, L.hminInv,
                             L.hmaxInv, L.hminratio, hp.radialOnly != 0, F.f[F_X][i], F.f[F_Y][i], F.f[F_Z][i],
                             F.f[F_RAD0][i]));
}

// FP32 variant of finalizeNode for the mixed mode: the per-node completion
// (3x3 inverse, corrected gradient, IdealH lookup) in FP32, results stored in
// the FP64 fields.  GB300 runs FP64 at a small fraction of the FP32 rate, so
// per-node FP64 work is visible even next to a ~100-neighbour pair loop.
__device__ __forceinline__ float hermiteLookup32(const double* __restrict__ v, const HydroParams& hp, float x) {
  const int N = hp.hermN;
  const float xmin = (float)hp.hermXmin, xmax = (float)hp.hermXmax, st = (float)hp.hermXstep;
  if (x < xmin) return (float)v[0] + (float)v[N] * (x - xmin);
  if (x > xmax) return (float)v[N - 1] + (float)v[2 * N - 1] * (x - xmin);
  const int i0 = min(N - 2, (int)(fmaxf(0.0f, x - xmin) / st));
  const float t = fmaxf(0.0f, fminf(1.0f, (x - xmin - i0 * st) / st));
  const float t2 = t * t, t3 = t * t2;
  return ((2.0f * t3 - 3.0f * t2 + 1.0f) * (float)v[i0] + (-2.0f * t3 + 3.0f * t2) * (float)v[i0 + 1] +
          st * ((t3 - 2.0f * t2 + t) * (float)v[N + i0] + (t3 - t2) * (float)v[N + i0 + 1]));
}

struct NodeAcc32 {
  float rhoSum, norm, gx, gy, gz, maxQ, effQ, xw, xdx, xdy, xdz, m0, m1x, m1y, m1z;
  double dvx, dvy, dvz, deps;
  float D[9], M[9];
  float m2[6];      // TENSOR: ASPH second moment
  float4 h0, h1;    // TENSOR: the node's H mirror
};

// TENSOR: ASPHClassicSmoothingScale in FP32 (tensor DH/Dt, asphClassicHideal).
template <bool TENSOR>
__device__ __forceinline__ void finalizeNode32(Fields& F, long i, int li, const NodeAcc32& a, int numNb,
                                               const HydroParams& hp, const double* __restrict__ herm) {
  const float mi = (float)F.f[F_MASS][i], rhoi = (float)F.f[F_RHO][i], ai = (float)F.f[F_HINV][i];
  const float Hdeti = TENSOR ? a.h1.z : (ai * ai) * ai;
  const float W0 = (float)hp.W0;
  F.f[F_RHOSUM][i] = a.rhoSum + mi * W0 * Hdeti;
  F.f[F_NORM][i] = a.norm + mi / rhoi * W0 * Hdeti;
  float D[9], Mm[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) { D[k] = a.D[k]; Mm[k] = a.M[k]; }
  const float detM = (Mm[0] * Mm[4] * Mm[8] + Mm[1] * Mm[5] * Mm[6] + Mm[2] * Mm[3] * Mm[7] -
                      Mm[0] * Mm[5] * Mm[7] - Mm[1] * Mm[3] * Mm[8] - Mm[2] * Mm[4] * Mm[6]);
  const float irho = 1.0f / rhoi;
  if (hp.correctVelGrad && fabsf(detM) > 1.0e-10f && numNb > 8) {
    const float id = 1.0f / detM;
    const float inv[9] = {(Mm[4] * Mm[8] - Mm[5] * Mm[7]) * id, (Mm[2] * Mm[7] - Mm[1] * Mm[8]) * id,
                          (Mm[1] * Mm[5] - Mm[2] * Mm[4]) * id, (Mm[5] * Mm[6] - Mm[3] * Mm[8]) * id,
                          (Mm[0] * Mm[8] - Mm[2] * Mm[6]) * id, (Mm[2] * Mm[3] - Mm[0] * Mm[5]) * id,
                          (Mm[3] * Mm[7] - Mm[4] * Mm[6]) * id, (Mm[1] * Mm[6] - Mm[0] * Mm[7]) * id,
                          (Mm[0] * Mm[4] - Mm[1] * Mm[3]) * id};
    float R[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        R[3 * r + c] = D[3 * r] * inv[c] + D[3 * r + 1] * inv[3 + c] + D[3 * r + 2] * inv[6 + c];
#pragma unroll
    for (int k = 0; k < 9; ++k) { D[k] = R[k]; Mm[k] = inv[k]; }
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] *= irho;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) { F.f[F_DVDX_XX + k][i] = D[k]; F.f[F_M_XX + k][i] = Mm[k]; }
  F.f[F_GRADRHO_X][i] = a.gx * irho;
  F.f[F_GRADRHO_Y][i] = a.gy * irho;
  F.f[F_GRADRHO_Z][i] = a.gz * irho;
  const float trace = D[0] + D[4] + D[8];
  F.f[F_DRHODT][i] = -(double)rhoi * trace;
  F.f[F_DVDT_X][i] = a.dvx;
  F.f[F_DVDT_Y][i] = a.dvy;
  F.f[F_DVDT_Z][i] = a.dvz;
  F.f[F_DEPSDT][i] = hp.totalEnergy
                         ? (double)mi * ((F.f[F_VX][i] * a.dvx + F.f[F_VY][i] * a.dvy + F.f[F_VZ][i] * a.dvz) + a.deps)
                         : a.deps;
  F.f[F_MAXQ][i] = a.maxQ;
  F.f[F_EFFQ][i] = a.effQ;
  float xw = a.xw;
  const double vxi = F.f[F_VX][i], vyi = F.f[F_VY][i], vzi = F.f[F_VZ][i];
  if (hp.xsph) {
    xw += Hdeti * mi * irho * W0;
    const float ws = fmaxf(1.0e-30f, xw);
    F.f[F_DXDT_X][i] = vxi + a.xdx / ws;
    F.f[F_DXDT_Y][i] = vyi + a.xdy / ws;
    F.f[F_DXDT_Z][i] = vzi + a.xdz / ws;
  } else {
    F.f[F_DXDT_X][i] = vxi;
    F.f[F_DXDT_Y][i] = vyi;
    F.f[F_DXDT_Z][i] = vzi;
  }
  F.f[F_XSPHW][i] = xw;
  F.f[F_XSPHDV_X][i] = a.xdx;
  F.f[F_XSPHDV_Y][i] = a.xdy;
  F.f[F_XSPHDV_Z][i] = a.xdz;
  const NodeListParams L = hp.lists[li];
  const float m0 = cbrtf(fmaxf(0.0f, a.m0));
  if (!(TENSOR && hp.asphEnd)) {
    F.f[F_M0][i] = m0;
    F.f[F_M1_X][i] = a.m1x;
    F.f[F_M1_Y][i] = a.m1y;
    F.f[F_M1_Z][i] = a.m1z;
  }
  if (TENSOR) {
    const SymT<float> Hi{a.h0.x, a.h0.y, a.h0.z, a.h0.w, a.h1.x, a.h1.y};
    storeSym(F, F_DHDTT_XX, i, smoothingScaleDerivative(Hi, D));
    if (hp.asphEnd) return;   // ASPHSmoothingScale: the ideal H comes at the end of the step
    const SymT<float> M2{a.m2[0], a.m2[1], a.m2[2], a.m2[3], a.m2[4], a.m2[5]};
    storeSym(F, F_M2_XX, i, M2);
    const float nPerh = (float)L.nPerh;
    const bool isolated = fabsf(m0) <= 1.0e-15f * fmaxf(1.0f, fabsf(m0));
    const float cur = isolated ? 0.5f * nPerh : fmaxf(0.0f, hermiteLookup32(herm, hp, m0));
    const float s = fminf(4.0f, fmaxf(0.25f, nPerh / cur));
    // positive definite (Sylvester): every eigenvalue of M2 positive
    const bool pd = M2.xx > 0.0f && M2.xx * M2.yy - M2.xy * M2.xy > 0.0f && symDet(M2) > 0.0f;
    storeSym(F, F_HIDEALT_XX, i,
             asphClassicHideal(M2, pd, Hi, s, hp.fixShape != 0, (float)L.hminInv, (float)L.hmaxInv,
                               (float)L.hminratio, hp.radialOnly != 0, (float)F.f[F_X][i], (float)F.f[F_Y][i],
                               (float)F.f[F_Z][i], (float)F.f[F_RAD0][i]));
    return;
  }
  // FP32 forms of DHDt = -(H/3) tr(DvDx) and of the IdealH clamp
  // 1/clamp(h0 f, hmin, hmax) = clamp(H0 / f, 1/hmax, 1/hmin): no FP64 divide.
  F.f[F_DHDT][i] = (double)(-(ai * (1.0f / 3.0f)) * trace);
  const float nPerh = (float)L.nPerh;
  const bool iso = fabsf(m0) <= 1.0e-15f * fmaxf(1.0f, fabsf(m0));
  const float cur = iso ? 0.5f * nPerh : fmaxf(0.0f, hermiteLookup32(herm, hp, m0));
  const float s = fminf(4.0f, fmaxf(0.25f, nPerh / (cur + 1.0e-30f)));
  const float aa = s < 1.0f ? 0.4f * (1.0f + s * s) : 0.4f * (1.0f + 1.0f / (s * s * s));
  const double hid = (double)(ai / (1.0f - aa + aa * s));
  F.f[F_HIDEAL][i] = fmin(L.hminInv, fmax(L.hmaxInv, hid));
}

// A 32-byte record in one load (p a multiple of 32 bytes): for a gather half
// the L1 requests of two 16-byte loads.
struct Rec32B {
  float4 a, b;
};
__device__ __forceinline__ Rec32B load32B(const float4* p) {
  Rec32B r;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w)
      : "l"(p));
  return r;
}

// v12 = v0 + a dt/2 of the compatible-energy sweep, formed in FP64 and stored
// as an unevaluated float pair hi + lo.
__device__ __forceinline__ void halfStepVelocity(const Fields& F, long i, double ax, double ay, double az, double deps,
                                                 const HalfStep& half) {
  const double x = F.f[F_VX0][i] + ax * half.hdt;
  const double y = F.f[F_VY0][i] + ay * half.hdt;
  const double z = F.f[F_VZ0][i] + az * half.hdt;
  const float hx = (float)x, hy = (float)y, hz = (float)z;
  half.v[2 * i] = make_float4(hx, hy, hz, (float)deps);
  half.v[2 * i + 1] = make_float4((float)(x - hx), (float)(y - hy), (float)(z - hz), 0.0f);
}
// Per-node inputs of the isotropic pair sweep: (rho, Omega^-1 P / rho^2, -Cl c,
// 1 / (2 rho)), once per node instead of once per pair.
__device__ __forceinline__ float4 pairRecord(const float4& th, const PairForm& pf) {
  const float ir = __frcp_rn(th.x);
  float pr = __fmul_rn(__fmul_rn(__fmul_rn(th.w, th.y), ir), ir), hir = 0.5f * ir;
  if (pf.spline) { pr = timesSplineA(pr); hir = timesSplineA(hir); }
  return make_float4(th.x, pr, __fmul_rn(-pf.Cl, th.z), hir);
}
// The limited Q's DvDx for h = r/2: its symmetric part (xx yy zz xy | xz yz,
// off-diagonal pairs summed), or for the exact form (full) all nine components.
__device__ __forceinline__ void writeQGradient(const Fields32& P, long i, float* v, const PairForm& pf) {
  if (pf.full) {
    P.dvq[i] = make_float4(v[0], v[1], v[2], v[3]);
    P.dvq[P.stride + i] = make_float4(v[4], v[5], v[6], v[7]);
    P.dvq[2 * P.stride + i] = make_float4(v[8], 0.0f, 0.0f, 0.0f);
    return;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) v[k] *= 0.25f;
  P.dvq[i] = make_float4(v[0], v[4], v[8], v[1] + v[3]);
  P.dvq[P.stride + i] = make_float4(v[2] + v[6], v[5] + v[7], 0.0f, 0.0f);
}

// Node completion of the isotropic mixed pair loop: finalizeNode32 in terms
// of the loop's reduced sums.  The FP32 results go into the FP64 fields by
// integer conversions (the FP64 pipe is ~1/64 of the FP32 rate).
struct PairSums32 {
  float w, mw, ve, g0, m1x, m1y, m1z;      // sum w, m w, (V/2) e a^3 w, |g|, |g| r
  float D[9], M[6], gx, gy, gz, maxE;      // sum u v r^T, u r r^T (xx xy xz yy yz zz), u (rho_j - rho_i) r; max e
  float xw, xdx, xdy, xdz;                 // XSPH
  double dvx, dvy, dvz, deps;
};
// SPLINE: the sums carry W/A and W'/A of the cubic B-spline (the energy rate
// one factor of A already).
template <bool SPLINE>
__device__ __forceinline__ void finalizePair32(Fields& F, long i, int li, PairSums32& a, float ai, float mi,
                                               float rhoi, int numNb, const HydroParams& hp,
                                               const double* __restrict__ herm, const HalfStep& half) {
  auto put = [&](int f, float v) { F.f[f][i] = toDouble(v); };
  const float Hdeti = (ai * ai) * ai, W0 = (float)hp.W0;
  const float irho = 1.0f / rhoi;
  if (SPLINE) {
    a.w = timesSplineA(a.w); a.mw = timesSplineA(a.mw); a.g0 = timesSplineA(a.g0);
    a.m1x = timesSplineA(a.m1x); a.m1y = timesSplineA(a.m1y); a.m1z = timesSplineA(a.m1z);
  }
  put(F_RHOSUM, Hdeti * (a.mw + mi * W0));
  put(F_NORM, mi * irho * Hdeti * (a.w + W0));
  auto norm = [](float x) { return SPLINE ? timesSplineA(x) : x; };
  float D[9], Mm[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) D[k] = -norm(a.D[k]);
  Mm[0] = -norm(a.M[0]); Mm[1] = -norm(a.M[1]); Mm[2] = -norm(a.M[2]);
  Mm[3] = Mm[1];         Mm[4] = -norm(a.M[3]); Mm[5] = -norm(a.M[4]);
  Mm[6] = Mm[2];         Mm[7] = Mm[5];         Mm[8] = -norm(a.M[5]);
  const float detM = (Mm[0] * Mm[4] * Mm[8] + Mm[1] * Mm[5] * Mm[6] + Mm[2] * Mm[3] * Mm[7] -
                      Mm[0] * Mm[5] * Mm[7] - Mm[1] * Mm[3] * Mm[8] - Mm[2] * Mm[4] * Mm[6]);
  if (hp.correctVelGrad && fabsf(detM) > 1.0e-10f && numNb > 8) {
    const float id = 1.0f / detM;
    const float inv[9] = {(Mm[4] * Mm[8] - Mm[5] * Mm[7]) * id, (Mm[2] * Mm[7] - Mm[1] * Mm[8]) * id,
                          (Mm[1] * Mm[5] - Mm[2] * Mm[4]) * id, (Mm[5] * Mm[6] - Mm[3] * Mm[8]) * id,
                          (Mm[0] * Mm[8] - Mm[2] * Mm[6]) * id, (Mm[2] * Mm[3] - Mm[0] * Mm[5]) * id,
                          (Mm[3] * Mm[7] - Mm[4] * Mm[6]) * id, (Mm[1] * Mm[6] - Mm[0] * Mm[7]) * id,
                          (Mm[0] * Mm[4] - Mm[1] * Mm[3]) * id};
    float R[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        R[3 * r + c] = D[3 * r] * inv[c] + D[3 * r + 1] * inv[3 + c] + D[3 * r + 2] * inv[6 + c];
#pragma unroll
    for (int k = 0; k < 9; ++k) { D[k] = R[k]; Mm[k] = inv[k]; }
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] *= irho;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) { put(F_DVDX_XX + k, D[k]); put(F_M_XX + k, Mm[k]); }
  put(F_GRADRHO_X, irho * norm(a.gx)); put(F_GRADRHO_Y, irho * norm(a.gy)); put(F_GRADRHO_Z, irho * norm(a.gz));
  const float trace = D[0] + D[4] + D[8];
  put(F_DRHODT, -rhoi * trace);
  const double vxi = F.f[F_VX][i], vyi = F.f[F_VY][i], vzi = F.f[F_VZ][i];
  F.f[F_DVDT_X][i] = a.dvx;
  F.f[F_DVDT_Y][i] = a.dvy;
  F.f[F_DVDT_Z][i] = a.dvz;
  F.f[F_DEPSDT][i] =
      hp.totalEnergy ? toDouble(mi) * ((vxi * a.dvx + vyi * a.dvy + vzi * a.dvz) + a.deps) : a.deps;
  if (half.v) halfStepVelocity(F, i, a.dvx, a.dvy, a.dvz, F.f[F_DEPSDT][i], half);
  put(F_MAXQ, rhoi * a.maxE);
  put(F_EFFQ, 2.0f * rhoi * a.ve);
  float xw = a.xw;
  if (hp.xsph) {
    xw += Hdeti * mi * irho * W0;
    const float ws = fmaxf(1.0e-30f, xw);
    F.f[F_DXDT_X][i] = vxi + toDouble(a.xdx / ws);
    F.f[F_DXDT_Y][i] = vyi + toDouble(a.xdy / ws);
    F.f[F_DXDT_Z][i] = vzi + toDouble(a.xdz / ws);
  } else {
    F.f[F_DXDT_X][i] = vxi;
    F.f[F_DXDT_Y][i] = vyi;
    F.f[F_DXDT_Z][i] = vzi;
  }
  put(F_XSPHW, xw);
  put(F_XSPHDV_X, a.xdx); put(F_XSPHDV_Y, a.xdy); put(F_XSPHDV_Z, a.xdz);
  const NodeListParams L = hp.lists[li];
  const float m0 = cbrtf(fmaxf(0.0f, a.g0));
  put(F_M0, m0);
  put(F_M1_X, -ai * a.m1x); put(F_M1_Y, -ai * a.m1y); put(F_M1_Z, -ai * a.m1z);
  put(F_DHDT, -(ai * (1.0f / 3.0f)) * trace);
  const float nPerh = (float)L.nPerh;
  const bool iso = fabsf(m0) <= 1.0e-15f * fmaxf(1.0f, fabsf(m0));
  const float cur = iso ? 0.5f * nPerh : fmaxf(0.0f, hermiteLookup32(herm, hp, m0));
  const float s = fminf(4.0f, fmaxf(0.25f, nPerh / (cur + 1.0e-30f)));
  const float aa = s < 1.0f ? 0.4f * (1.0f + s * s) : 0.4f * (1.0f + 1.0f / (s * s * s));
  const double hid = toDouble(ai / (1.0f - aa + aa * s));
  F.f[F_HIDEAL][i] = fmin(L.hminInv, fmax(L.hmaxInv, hid));
}

//------------------------------------------------------------------------------
// Time-step vote; the bits of positive doubles order as integers.  FP32 limits
// travel as one 64-bit word, the reason code in the low mantissa bits that a
// widened float leaves zero.  FP64 limits need all their bits: one minimum per
// reason.
//------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long warpMin64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return v;
}
__device__ __forceinline__ unsigned long long dtKey(float v, int reason) {
  return (unsigned long long)__double_as_longlong(toDouble(v)) | (unsigned)reason;
}

// FP32 node limits of GenericHydro::dt (GenericHydro.cc:113-381): the smallest
// of them and of the pair limit, with its reason.  Every term is positive.
__device__ __forceinline__ float nodeDt32(float ns, float cs, float maxQ, float rho, float divv, float vmag,
                                          float amag, bool velDt, float pairDt, int& reason) {
  const float tiny = (float)DBL_EPSILON;
  float best = 3.0e38f;
  reason = -1;
  auto vote = [&](float v, int r) {
    if (v < best) { best = v; reason = r; }
  };
  vote(ns / (cs + tiny), 0);
  vote(ns / (sqrtf(maxQ / rho) + tiny), 1);
  vote(1.0f / (fabsf(divv) + tiny), 2);
  vote(0.1f * fmaxf(ns / (vmag + tiny), vmag / (amag + tiny)), 3);
  if (velDt) vote(ns / (vmag + 1.0e-10f), 4);
  vote(pairDt, 5);
  return best;
}

// The vote of GenericHydro::dt for one node in the precision of its FP64 limits.
// Each node first forms all its limits in FP32 (worst: the largest
// (max(a_i, a_j) |v_ij|)^2 of its pairs); only a node whose FP32 limit is within
// 1e-4 of the smallest seen so far (voteEst, which only falls) can hold the
// minimum and repeats its limits in FP64.  Whole warps call it.
template <bool TENSOR>
__device__ __forceinline__ void voteNode32(const Fields& F, const HydroParams& hp, const int* __restrict__ list, long i,
                                           bool votes, float lmaxi, const float4& vi, float worst, double maxNperh,
                                           StepScratch* __restrict__ sc) {
  const float bestPair = worst > 0.0f ? rsqrtf(worst) : 3.0e38f;
  float est = 3.0e38f;
  const NodeListParams Li = hp.lists[list[i]];
  if (votes) {
    const float ax = toFloatRN(F.f[F_DVDT_X][i]), ay = toFloatRN(F.f[F_DVDT_Y][i]), az = toFloatRN(F.f[F_DVDT_Z][i]);
    const float divv = toFloatRN(F.f[F_DVDX_XX][i] + F.f[F_DVDX_YY][i] + F.f[F_DVDX_ZZ][i]);
    int reason;
    est = nodeDt32(1.0f / (lmaxi * (float)Li.nPerh), toFloatRN(F.f[F_CS][i]), toFloatRN(F.f[F_MAXQ][i]),
                   toFloatRN(F.f[F_RHO][i]), divv, sqrtf(vi.x * vi.x + vi.y * vi.y + vi.z * vi.z),
                   sqrtf(ax * ax + ay * ay + az * az), hp.useVelMagDt != 0, bestPair / (float)maxNperh, reason);
  }
  const float wmin = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(est)));
  if ((threadIdx.x & 31) == 0 && wmin < 3.0e38f) atomicMin(&sc->voteEst, __float_as_uint(wmin));
  const float seen = __uint_as_float(*(volatile unsigned*)&sc->voteEst);
  // NaN compares false: a node with a NaN limit takes the FP64 limits too
  if (votes && !(est > fminf(seen, wmin) * 1.0001f)) {
    const double tiny = DBL_EPSILON;
    double best = DBL_MAX;
    int reason = -1;
    const double ai = F.f[TENSOR ? F_HLMAX : F_HINV][i];   // largest eigenvalue of H
    const double nodeScalei = 1.0 / ai / Li.nPerh;
    const double vxi = F.f[F_VX][i], vyi = F.f[F_VY][i], vzi = F.f[F_VZ][i];
    const double rhoi = F.f[F_RHO][i];
    const double csDt = nodeScalei / (F.f[F_CS][i] + tiny);
    if (csDt < best) { best = csDt; reason = 0; }
    const double csqDt = nodeScalei / (sqrt(F.f[F_MAXQ][i] / rhoi) + tiny);
    if (csqDt < best) { best = csqDt; reason = 1; }
    const double divvDt = 1.0 / (fabs(F.f[F_DVDX_XX][i] + F.f[F_DVDX_YY][i] + F.f[F_DVDX_ZZ][i]) + tiny);
    if (divvDt < best) { best = divvDt; reason = 2; }
    const double vmag = sqrt(vxi * vxi + vyi * vyi + vzi * vzi);
    const double ax = F.f[F_DVDT_X][i], ay = F.f[F_DVDT_Y][i], az = F.f[F_DVDT_Z][i];
    const double dtAcc = 0.1 * fmax(nodeScalei / (vmag + tiny), vmag / (sqrt(ax * ax + ay * ay + az * az) + tiny));
    if (dtAcc < best) { best = dtAcc; reason = 3; }
    if (hp.useVelMagDt) {
      const double velDt = nodeScalei / (vmag + 1.0e-10);
      if (velDt < best) { best = velDt; reason = 4; }
    }
    const double pairDt = (worst > 0.0f ? 1.0 / sqrt((double)worst) : 3.0e38) / maxNperh;
    if (pairDt < best) { best = pairDt; reason = 5; }
    if (reason >= 0) atomicMin(&sc->votes[reason], (unsigned long long)__double_as_longlong(best));
  }
}

}  // namespace dev
}  // namespace sph
