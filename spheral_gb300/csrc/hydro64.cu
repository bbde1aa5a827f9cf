// FP64 sweeps of libsphgpu for isotropic H (sm_103a): the density sum with the
// time-step vote, the grad-h correction, the SPH pair loop and the
// compatible-energy sweep.
//
// GB300 executes two FP64 operations per SM and clock (a warp instruction
// occupies the FP64 unit for 16 cycles), so these sweeps are bound by the
// number of FP64 instructions per pair; issue slots, integer work and loads
// are free beside it.  Hence:
//  * with H = a I both kernel gradients lie along the separation, and the
//    pair reduces to scalars times r (the form of the mixed sweep in
//    hydro32.cu): ~100 FP64 instructions per ordered pair instead of ~440
//    (KH slab, 94,500 nodes: pair loop 7.50 -> 2.75 ms, at 88 % of the FP64
//    unit; density and vote 1.85 -> 0.82 ms at 84 %);
//  * everything that depends on one node only (1/rho, Prho, Cl c) is formed
//    once per node into a record, read by aligned 16-byte loads;
//  * |r| and the viscosity's two quotients come from one reciprocal square
//    root and one reciprocal, each a hardware seed (~20 bits) with one
//    third-order Householder step;
//  * comparisons of positive values and index arithmetic use the integer pipe.
#include "device.cuh"
#include "recip64.cuh"

namespace sph {
namespace {
using namespace dev;

inline unsigned gridFor(long n, int b) { return (unsigned)((n + b - 1) / b); }

__device__ __forceinline__ long long bits(double x) { return __double_as_longlong(x); }
// max of two non-negative values
__device__ __forceinline__ double maxPos(double a, double b) { return bits(a) > bits(b) ? a : b; }
__device__ __forceinline__ double flipIf(double x, bool f) {
  return __longlong_as_double(bits(x) ^ (f ? (long long)0x8000000000000000ULL : 0LL));
}

// Per-node record: position and 1/h, velocity and mass, and the pair loop's
// (rho, Omega^-1 P / rho^2, -Cl c, 1 / (2 rho)).
struct __align__(32) Node64 {
  double2 xy, za, vxy, vzm, rp, ch;
};
struct __align__(32) Velocity64 {   // half-step velocity and DepsDt
  double2 xy, zd;
};

__global__ void nodes64Kernel(Fields F, long n, double Cl, int pairPart, Node64* __restrict__ rec) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  Node64& r = rec[i];
  r.xy = make_double2(F.f[F_X][i], F.f[F_Y][i]);
  r.za = make_double2(F.f[F_Z][i], F.f[F_HINV][i]);
  r.vxy = make_double2(F.f[F_VX][i], F.f[F_VY][i]);
  r.vzm = make_double2(F.f[F_VZ][i], F.f[F_MASS][i]);
  if (pairPart) {
    const double rho = F.f[F_RHO][i], om = F.f[F_OMEGA][i];
    r.rp = make_double2(rho, om / (om * om + kTiny30) * F.f[F_P][i] / (rho * rho));
    r.ch = make_double2(-Cl * F.f[F_CS][i], 0.5 / rho);
  }
}
__global__ void velocity64Kernel(Fields F, long n, double hdt, Velocity64* __restrict__ v) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  v[i].xy = make_double2(F.f[F_VX0][i] + F.f[F_DVDT_X][i] * hdt, F.f[F_VY0][i] + F.f[F_DVDT_Y][i] * hdt);
  v[i].zd = make_double2(F.f[F_VZ0][i] + F.f[F_DVDT_Z][i] * hdt, F.f[F_DEPSDT][i]);
}

// The kernel table in shared memory, per interval (g0 g1 | g2 w0 | w1 w2),
// with a zero interval behind it for eta beyond the extent.
struct Table64 {
  const double2* t;
  double inv, step, extent;
  int N1;
  // Interval of eta as eta / step truncated.  eta * (1/step) plus 1.5 2^32
  // leaves it as a fixed-point number with 20 fractional bits in the low
  // word; within 2^-20 of a knot the division decides, so the interval is
  // that of the reference lookup for every eta.
  __device__ __forceinline__ int index(double eta) const {
    if (bits(eta) >= bits(extent)) return N1 + 1;
    const unsigned lo = (unsigned)__double2loint(__dadd_rn(__dmul_rn(eta, inv), 6442450944.0));
    unsigned k = lo >> 20;
    if (((lo + 1u) & 0xfffffu) <= 2u) k = (unsigned)(eta / step);
    return (int)min(k, (unsigned)N1);
  }
  __device__ __forceinline__ double grad(int k, double eta) const {
    const double2 a = t[3 * k], b = t[3 * k + 1];
    return __fma_rn(__fma_rn(b.x, eta, a.y), eta, a.x);
  }
  __device__ __forceinline__ double value(int k, double eta) const {
    const double2 b = t[3 * k + 1], c = t[3 * k + 2];
    return __fma_rn(__fma_rn(c.y, eta, c.x), eta, b.y);
  }
};
__device__ __forceinline__ Table64 loadTable64(double2* sm, const TableDev& t, const HydroParams& hp) {
  const int nint = hp.tableN1 + 1;
  for (int k = threadIdx.x; k <= nint; k += blockDim.x) {
    const bool in = k < nint;
    sm[3 * k] = in ? make_double2(t.g[3 * k], t.g[3 * k + 1]) : make_double2(0.0, 0.0);
    sm[3 * k + 1] = in ? make_double2(t.g[3 * k + 2], t.w[3 * k]) : make_double2(0.0, 0.0);
    sm[3 * k + 2] = in ? make_double2(t.w[3 * k + 1], t.w[3 * k + 2]) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  return Table64{sm, 1.0 / hp.tableXstep, hp.tableXstep, hp.extent, hp.tableN1};
}
size_t tableBytes(const HydroParams& hp) { return 3 * (size_t)(hp.tableN1 + 2) * sizeof(double2); }

template <int L>
__device__ __forceinline__ double laneSum64(double v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int L>
__device__ __forceinline__ double laneMax64(double v) {   // non-negative values
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = maxPos(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// r = x_i - x_j through the image of the entry; r^2, 1/|r| and |r|.
__device__ __forceinline__ void separation64(const Grid& g, int code, double xi, double yi, double zi, const double2& xy,
                                             double z, double& rx, double& ry, double& rz, double& ir, double& rm) {
  double xj = xy.x, yj = xy.y, zj = z;
  imagePos(g, code, xj, yj, zj);
  rx = xi - xj; ry = yi - yj; rz = zi - zj;
  double r2 = __fma_rn(rz, rz, __fma_rn(ry, ry, __dmul_rn(rx, rx)));
  ir = rsqrt64(bits(r2) > bits(1.0e-290) ? r2 : 1.0e-290);   // coincident nodes: |r| = 0, finite 1/|r|
  rm = r2 * ir;
}

struct Sweep64 {
  double2 xy, za, vxy, vzm;
};

//------------------------------------------------------------------------------
// DENS: computeSPHSumMassDensity (src/SPH/computeSPHSumMassDensity.cc:15-87),
// gathered.  DT: GenericHydro::dt (src/Physics/GenericHydro.cc:113-381) on the
// same pass, with the new density; the pairwise limit min(h_i, h_j) / |v_ij|
// is 1 / sqrt(max (max(a_i, a_j) |v_ij|)^2).  One (value, reason) per block.
//------------------------------------------------------------------------------
template <bool DENS, bool DT, int L>
__global__ void __launch_bounds__(128) density64Kernel(Fields F, const Node64* __restrict__ rec,
                                                       const int* __restrict__ list, long n, Grid g, NeighborLists nl,
                                                       TableDev t, HydroParams hp, double maxNperh,
                                                       double* __restrict__ part) {
  extern __shared__ double2 sm64[];
  __shared__ double sv[4];
  __shared__ int sr[4];
  Table64 T{};
  if (DENS) T = loadTable64(sm64, t, hp);
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;   // whole warps run to the shuffles
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const Node64 me = rec[i];
  const double xi = me.xy.x, yi = me.xy.y, zi = me.za.x, ai = me.za.y, mi = me.vzm.y;
  const bool multi = hp.numLists > 1;
  const int li = list[i];
  double sum = 0.0, worst = 0.0;
  const int cnt = live ? nl.count[i] : 0;
  laneSlots<L, 1, Sweep64>(
      nl, i, sub, cnt,
      [&](uint32_t j, Sweep64& r) {
        const Node64& q = rec[j];
        if (DENS) r.xy = q.xy;
        r.za = q.za;
        if (DT) r.vxy = q.vxy;
        r.vzm = q.vzm;
      },
      [&](uint32_t ent, const Sweep64& r) {
        const int code = imageCode(g, hc, (int)(ent >> kIndexBits));
        const double aj = r.za.y;
        if (DENS) {
          double rx, ry, rz, ir, rm;
          separation64(g, code, xi, yi, zi, r.xy, r.za.x, rx, ry, rz, ir, rm);
          const double eta = aj * rm;
          const double w = T.value(T.index(eta), eta);
          const double m = (multi && list[ent & kIndexMask] != li) ? mi : r.vzm.y;
          sum = __fma_rn(m, ((aj * aj) * aj) * w, sum);
        }
        if (DT) {
          double vxj = r.vxy.x, vyj = r.vxy.y, vzj = r.vzm.x;
          imageVec(g, code, vxj, vyj, vzj);
          const double dx = me.vxy.x - vxj, dy = me.vxy.y - vyj, dz = me.vzm.x - vzj;
          const double am = maxPos(ai, aj);
          worst = maxPos(worst, (am * am) * __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx)));
        }
      });
  if (L > 1) {
    if (DENS) sum = laneSum64<L>(sum);
    if (DT) worst = laneMax64<L>(worst);
  }
  double best = DBL_MAX;
  int reason = -1;
  if (live && sub == 0) {
    double rhoi;
    if (DENS) {
      rhoi = mi * (((ai * ai) * ai) * hp.W0) + sum;
      F.f[F_RHO][i] = rhoi;
    }
    if (DT && !isGhost(hp, i)) {
      if (!DENS) rhoi = F.f[F_RHO][i];
      const double tiny = DBL_EPSILON;
      const double nodeScalei = 1.0 / ai / hp.lists[li].nPerh;
      auto vote = [&](double v, int r) {
        if (v < best) { best = v; reason = r; }
      };
      vote(nodeScalei / (F.f[F_CS][i] + tiny), 0);
      vote(nodeScalei / (sqrt(F.f[F_MAXQ][i] / rhoi) + tiny), 1);
      vote(1.0 / (fabs(F.f[F_DVDX_XX][i] + F.f[F_DVDX_YY][i] + F.f[F_DVDX_ZZ][i]) + tiny), 2);
      const double vx = me.vxy.x, vy = me.vxy.y, vz = me.vzm.x;
      const double vmag = sqrt(vx * vx + vy * vy + vz * vz);
      const double ax = F.f[F_DVDT_X][i], ay = F.f[F_DVDT_Y][i], az = F.f[F_DVDT_Z][i];
      vote(0.1 * fmax(nodeScalei / (vmag + tiny), vmag / (sqrt(ax * ax + ay * ay + az * az) + tiny)), 3);
      if (hp.useVelMagDt) vote(nodeScalei / (vmag + 1.0e-10), 4);
      if (cnt > 0) vote((1.0 / maxNperh) / fmax(kTiny30, sqrt(worst)), 5);
    }
  }
  if (!DT) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, best, o);
    const int r = __shfl_xor_sync(0xffffffffu, reason, o);
    if (v < best) { best = v; reason = r; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; sr[threadIdx.x >> 5] = reason; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w)
      if (sv[w] < best) { best = sv[w]; reason = sr[w]; }
    part[2 * blockIdx.x] = best;
    part[2 * blockIdx.x + 1] = (double)reason;
  }
}
__global__ void __launch_bounds__(1024) dtFinal64Kernel(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double sv[32], sr[32];
  double best = DBL_MAX, reason = -1.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    if (part[2 * b] < best) { best = part[2 * b]; reason = part[2 * b + 1]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, best, o), r = __shfl_xor_sync(0xffffffffu, reason, o);
    if (v < best) { best = v; reason = r; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; sr[threadIdx.x >> 5] = reason; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w)
      if (sv[w] < best) { best = sv[w]; reason = sr[w]; }
    out[0] = best;
    out[1] = reason;
  }
}

//------------------------------------------------------------------------------
// computeSPHOmegaGradhCorrection (src/SPH/computeSPHOmegaGradhCorrection.cc:15-116).
//------------------------------------------------------------------------------
template <int L>
__global__ void __launch_bounds__(128) gradh64Kernel(Fields F, const Node64* __restrict__ rec, long n, Grid g,
                                                     NeighborLists nl, TableDev t, HydroParams hp) {
  extern __shared__ double2 sm64[];
  const Table64 T = loadTable64(sm64, t, hp);
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const double xi = rec[i].xy.x, yi = rec[i].xy.y, zi = rec[i].za.x, ai = rec[i].za.y;
  double wsum = 0.0, gsum = 0.0;
  const int cnt = live ? nl.count[i] : 0;
  laneSlots<L, 1, Sweep64>(
      nl, i, sub, cnt,
      [&](uint32_t j, Sweep64& r) {
        r.xy = rec[j].xy;
        r.za = rec[j].za;
      },
      [&](uint32_t ent, const Sweep64& r) {
        double rx, ry, rz, ir, rm;
        separation64(g, imageCode(g, hc, (int)(ent >> kIndexBits)), xi, yi, zi, r.xy, r.za.x, rx, ry, rz, ir, rm);
        const double eta = ai * rm;
        const int k = T.index(eta);
        wsum += T.value(k, eta);
        gsum = __fma_rn(eta, T.grad(k, eta), gsum);
      });
  if (L > 1) {
    wsum = laneSum64<L>(wsum);
    gsum = laneSum64<L>(gsum);
  }
  if (!live || sub != 0) return;
  // Hdet cancels
  F.f[F_OMEGA][i] = cnt == 0 ? 1.0 : fmax(1.0e-30, -gsum / (3.0 * (wsum + hp.W0)));
}

//------------------------------------------------------------------------------
// SPH::evaluateDerivativesImpl (src/SPH/SPH.cc:294-552) with the
// (Limited)MonaghanGingoldViscosity and the SPHSmoothingScale moments + IdealH
// (SPHSmoothingScale.cc:154-272); the algebra of pairKernelIso32.
//------------------------------------------------------------------------------
template <bool XSPH, bool LIMQ, int L>
__global__ void __launch_bounds__(128) pair64Kernel(Fields F, const Node64* __restrict__ rec,
                                                    const int* __restrict__ list, long n, Grid g, NeighborLists nl,
                                                    TableDev t, HydroParams hp, double* __restrict__ pacc) {
  extern __shared__ double2 sm64[];
  const Table64 T = loadTable64(sm64, t, hp);
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const Node64 me = rec[i];
  const double xi = me.xy.x, yi = me.xy.y, zi = me.za.x, ai = me.za.y, vxi = me.vxy.x, vyi = me.vxy.y, vzi = me.vzm.x;
  const double mi = me.vzm.y, rhoi = me.rp.x;
  const double A4i = (ai * ai) * (ai * ai);
  const bool multi = hp.numLists > 1, tensile = hp.epsTensile != 0.0;
  const bool lin = hp.linearInExpansion != 0, quad = hp.quadraticInExpansion != 0;
  const int li = list[i];
  double Q[6];   // symmetric part of the Q's DvDx for h = r/2 (xx yy zz xy xz yz)
  auto loadQ = [&](long j, double* q) {
    q[0] = 0.25 * F.f[F_DVDXQ_XX][j]; q[1] = 0.25 * F.f[F_DVDXQ_YY][j]; q[2] = 0.25 * F.f[F_DVDXQ_ZZ][j];
    q[3] = 0.25 * (F.f[F_DVDXQ_XY][j] + F.f[F_DVDXQ_YX][j]);
    q[4] = 0.25 * (F.f[F_DVDXQ_XZ][j] + F.f[F_DVDXQ_ZX][j]);
    q[5] = 0.25 * (F.f[F_DVDXQ_YZ][j] + F.f[F_DVDXQ_ZY][j]);
  };
  if (LIMQ) loadQ(i, Q);
  double sw = 0.0, smw = 0.0, sve = 0.0, g0 = 0.0, m1x = 0.0, m1y = 0.0, m1z = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
  double maxE = 0.0, dvx = 0.0, dvy = 0.0, dvz = 0.0, deps = 0.0, xw = 0.0, xdx = 0.0, xdy = 0.0, xdz = 0.0;
  double D[9], M[6];
#pragma unroll
  for (int k = 0; k < 9; ++k) D[k] = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) M[k] = 0.0;
  const int cnt = live ? nl.count[i] : 0;
  double* out = hp.compatible ? pacc + paccSlot(nbSlot(i, 0, nl.cap) + 32 * sub) : nullptr;
  laneSlots<L, 1, Node64>(
      nl, i, sub, cnt, [&](uint32_t j, Node64& r) { r = rec[j]; },
      [&](uint32_t ent, const Node64& r) {
        const int code = imageCode(g, hc, (int)(ent >> kIndexBits));
        double rx, ry, rz, ir, rm;
        separation64(g, code, xi, yi, zi, r.xy, r.za.x, rx, ry, rz, ir, rm);
        double vxj = r.vxy.x, vyj = r.vxy.y, vzj = r.vzm.x;
        imageVec(g, code, vxj, vyj, vzj);
        const double aj = r.za.y, mj = r.vzm.y, rhoj = r.rp.x, hirj = r.ch.y;
        const double etai = ai * rm, etaj = aj * rm;
        const int ki = T.index(etai), kj = T.index(etaj);
        const double w = T.value(ki, etai), gi = T.grad(ki, etai), gj = T.grad(kj, etaj);
        const double vx = vxi - vxj, vy = vyi - vyj, vz = vzi - vzj;
        const double vr = __fma_rn(vz, rz, __fma_rn(vy, ry, vx * rx));
        double vq = vr;
        if (LIMQ) {
          double q[6];
          loadQ(ent & kIndexMask, q);
          if (code) {
            const bool fx = mirrored(code & 3, g.kindLo[0], g.kindHi[0]);
            const bool fy = mirrored((code >> 2) & 3, g.kindLo[1], g.kindHi[1]);
            const bool fz = mirrored((code >> 4) & 3, g.kindLo[2], g.kindHi[2]);
            q[3] = flipIf(q[3], fx != fy); q[4] = flipIf(q[4], fx != fz); q[5] = flipIf(q[5], fy != fz);
          }
          const double xx = rx * rx, yy = ry * ry, zz = rz * rz, xy = rx * ry, xz = rx * rz, yz = ry * rz;
          const double gri = Q[0] * xx + Q[1] * yy + Q[2] * zz + Q[3] * xy + Q[4] * xz + Q[5] * yz;
          const double grj = q[0] * xx + q[1] * yy + q[2] * zz + q[3] * xy + q[4] * xz + q[5] * yz;
          // van Leer factor of the smaller of q_i/q_j and q_j/q_i
          const double sum = gri + grj;
          double phi = 0.0;
          if ((bits(gri) ^ bits(grj)) >= 0 && fabs(sum) > 2.0e-30) {
            const double inv = 1.0 / sum;
            phi = 4.0 * (gri * inv) * (grj * inv);
          }
          const double etaij = bits(etai) < bits(etaj) ? etai : etaj;
          if (bits(etaij) < bits(hp.etaCrit)) {
            const double z = (etaij - hp.etaCrit) / hp.etaFold;
            phi *= exp(-(z * z));
          }
          vq = __fma_rn(-2.0 * phi, sum, vr);
        }
        // mu_i = a_i v.r / (eta_i^2 + eps2) and mu_j by one reciprocal
        const double di = __fma_rn(etai, etai, hp.eps2), dj = __fma_rn(etaj, etaj, hp.eps2);
        const double f = vq * rcp64(di * dj);
        const double mui = (ai * f) * dj, muj = (aj * f) * di;
        // strictly negative: coincident nodes have v.r = -0 or +0, and with eps2 = 0 a
        // quotient of 0/0 that no one-sided mu may take
        const bool neg = (unsigned long long)bits(vq) > 0x8000000000000000ULL;
        const double mni = neg ? mui : 0.0, mnj = neg ? muj : 0.0;
        double ei, ej;
        if (lin || quad) {
          const double qi = quad ? (neg ? mui * mui : -(mui * mui)) : mni * mni;
          const double qj = quad ? (neg ? muj * muj : -(muj * muj)) : mnj * mnj;
          ei = me.ch.x * (lin ? mui : mni) + hp.Cq * qi;
          ej = r.ch.x * (lin ? muj : mnj) + hp.Cq * qj;
        } else {
          ei = mni * __fma_rn(hp.Cq, mni, me.ch.x);
          ej = mnj * __fma_rn(hp.Cq, mnj, r.ch.x);
        }
        double pri = me.rp.y, prj = r.rp.y, wj = 0.0;
        if (XSPH || tensile) wj = T.value(kj, etaj);
        if (tensile) {   // P_eff = P (1 - epsT (W / W(1/nPerh))^4) in tension
          const double ti = w / hp.WnPerh, tj = wj / hp.WnPerh;
          if (pri < 0.0) pri *= 1.0 - hp.epsTensile * ((ti * ti) * (ti * ti));
          if (prj < 0.0) prj *= 1.0 - hp.epsTensile * ((tj * tj) * (tj * tj));
        }
        const double Ci = __fma_rn(ei, me.ch.y, pri), Cj = __fma_rn(ej, hirj, prj);
        const double aj2 = aj * aj;
        const double S = __fma_rn(Ci, A4i * gi, __dmul_rn(Cj, (aj2 * aj2) * gj)) * ir;
        const double gf = -mj * S;
        const double pax = gf * rx, pay = gf * ry, paz = gf * rz;
        dvx += pax; dvy += pay; dvz += paz;
        if (out) {
          out[0] = pax; out[32] = pay; out[64] = paz;
          out += 96 * L;
        }
        const double u = mj * (gi * ir);
        deps = __fma_rn(Ci, u * vr, deps);
        const double ux = u * rx, uy = u * ry, uz = u * rz;
        D[0] = __fma_rn(vx, ux, D[0]); D[1] = __fma_rn(vx, uy, D[1]); D[2] = __fma_rn(vx, uz, D[2]);
        D[3] = __fma_rn(vy, ux, D[3]); D[4] = __fma_rn(vy, uy, D[4]); D[5] = __fma_rn(vy, uz, D[5]);
        D[6] = __fma_rn(vz, ux, D[6]); D[7] = __fma_rn(vz, uy, D[7]); D[8] = __fma_rn(vz, uz, D[8]);
        M[0] = __fma_rn(rx, ux, M[0]); M[1] = __fma_rn(rx, uy, M[1]); M[2] = __fma_rn(rx, uz, M[2]);
        M[3] = __fma_rn(ry, uy, M[3]); M[4] = __fma_rn(ry, uz, M[4]); M[5] = __fma_rn(rz, uz, M[5]);
        const double dr = rhoj - rhoi;
        gx = __fma_rn(dr, ux, gx); gy = __fma_rn(dr, uy, gy); gz = __fma_rn(dr, uz, gz);
        const bool same = multi ? list[ent & kIndexMask] == li : true;
        if (same) {
          sw += w;
          smw = __fma_rn(mj, w, smw);
        }
        sve = __fma_rn(mj * hirj, ei * w, sve);
        if (bits(ei) > bits(maxE)) maxE = ei;   // signed order of the bits: negative e never replaces
        if (XSPH) {
          const double wx = mi * me.ch.y * ((ai * ai) * ai) * w + mj * hirj * (aj2 * aj) * wj;
          xw += wx;
          xdx -= wx * vx; xdy -= wx * vy; xdz -= wx * vz;
        }
        double wg = fabs(gi);
        if (!same) wg *= mj * rhoi / (mi * rhoj);
        g0 += wg;
        m1x = __fma_rn(wg, rx, m1x); m1y = __fma_rn(wg, ry, m1y); m1z = __fma_rn(wg, rz, m1z);
      });
  if (L > 1) {
    sw = laneSum64<L>(sw); smw = laneSum64<L>(smw); sve = laneSum64<L>(sve); g0 = laneSum64<L>(g0);
    m1x = laneSum64<L>(m1x); m1y = laneSum64<L>(m1y); m1z = laneSum64<L>(m1z);
    gx = laneSum64<L>(gx); gy = laneSum64<L>(gy); gz = laneSum64<L>(gz);
    dvx = laneSum64<L>(dvx); dvy = laneSum64<L>(dvy); dvz = laneSum64<L>(dvz); deps = laneSum64<L>(deps);
    maxE = laneMax64<L>(maxE);
    if (XSPH) { xw = laneSum64<L>(xw); xdx = laneSum64<L>(xdx); xdy = laneSum64<L>(xdy); xdz = laneSum64<L>(xdz); }
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] = laneSum64<L>(D[k]);
#pragma unroll
    for (int k = 0; k < 6; ++k) M[k] = laneSum64<L>(M[k]);
  }
  if (!live || sub != 0) return;
  const double Hdeti = (ai * ai) * ai;
  NodeAcc a;
  a.rhoSum = Hdeti * smw;
  a.norm = mi / rhoi * Hdeti * sw;
  a.dvx = dvx; a.dvy = dvy; a.dvz = dvz;
  a.deps = A4i * deps;
  a.gx = A4i * gx; a.gy = A4i * gy; a.gz = A4i * gz;
  a.maxQ = rhoi * maxE;
  a.effQ = 2.0 * rhoi * Hdeti * sve;
  a.xw = xw; a.xdx = xdx; a.xdy = xdy; a.xdz = xdz;
  a.m0 = g0; a.m1x = -ai * m1x; a.m1y = -ai * m1y; a.m1z = -ai * m1z;
#pragma unroll
  for (int k = 0; k < 9; ++k) a.D[k] = -A4i * D[k];
  a.M[0] = -A4i * M[0]; a.M[1] = -A4i * M[1]; a.M[2] = -A4i * M[2];
  a.M[3] = a.M[1];      a.M[4] = -A4i * M[3]; a.M[5] = -A4i * M[4];
  a.M[6] = a.M[2];      a.M[7] = a.M[5];      a.M[8] = -A4i * M[5];
  finalizeNode(F, i, li, a, mi, rhoi, vxi, vyi, vzi, ai, cnt, hp, t.herm);
}

//------------------------------------------------------------------------------
// SpecificThermalEnergyPolicy::update (src/Hydro/SpecificThermalEnergyPolicy.cc:110-173),
// gathered: node i takes its own share w_i du_ij of every pair.
//------------------------------------------------------------------------------
template <int L>
__global__ void __launch_bounds__(128) energy64Kernel(Fields F, const Velocity64* __restrict__ v12, long n, Grid g,
                                                      NeighborLists nl, const double* __restrict__ pacc, double dt) {
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;
  int hc[3];
  unpackCell(nl.cell[i], hc);
  const Velocity64 me = v12[i];
  double sum = 0.0;
  const double* pa = pacc + paccSlot(nbSlot(i, 0, nl.cap) + 32 * sub);
  laneSlots<L, 2, Velocity64>(
      nl, i, sub, live ? nl.count[i] : 0, [&](uint32_t j, Velocity64& r) { r = v12[j]; },
      [&](uint32_t ent, const Velocity64& r) {
        double vx = r.xy.x, vy = r.xy.y, vz = r.zd.x;
        imageVec(g, imageCode(g, hc, (int)(ent >> kIndexBits)), vx, vy, vz);
        const double du = __fma_rn(vz - me.zd.x, pa[64], __fma_rn(vy - me.xy.y, pa[32], (vx - me.xy.x) * pa[0]));
        pa += 96 * L;
        const bool neg = bits(du) < 0 && du != 0.0;
        const double si = flipIf(me.zd.y, neg), sj = flipIf(r.zd.y, neg);
        const double wi = bits(si) > bits(DBL_EPSILON) ? si : DBL_EPSILON;
        const double wj = bits(sj) > bits(DBL_EPSILON) ? sj : DBL_EPSILON;
        sum = __fma_rn(wi * rcp64(wi + wj), du, sum);   // both sides use the same reciprocal
      });
  if (L > 1) sum = laneSum64<L>(sum);
  if (!live || sub != 0) return;
  F.f[F_DEPS_COMPAT][i] = sum;
  F.f[F_EPS][i] = F.f[F_EPS0][i] + sum * dt;
}

// Lanes per node: enough warps to balance the SMs.  Pair sweep, us with 1 / 2 / 4 / 8:
// 8,000 nodes 353/189/182/214, 21,952 584/572/490/505, 39,304 835/742/738/854,
// 64,000 1137/1132/1123/1372, 148,877 2177/2255/2530/3035.
int lanes64(long n) { return n >= 60000 ? 1 : (n >= 30000 ? 2 : (n >= 8000 ? 4 : 8)); }

}  // namespace

size_t nodeRecordBytes64() { return sizeof(Node64); }

#define SPH_BY_LANES64(CALL)     \
  switch (lanes64(n)) {          \
    case 1: CALL(1); break;      \
    case 2: CALL(2); break;      \
    case 4: CALL(4); break;      \
    default: CALL(8); break;     \
  }

void launchDensityDt64(Fields F, void* nodeRec, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                       HydroParams hp, bool density, bool dt, double maxNperh, double* dScratch, double* dOut,
                       cudaStream_t s, LaunchCounter* lc) {
  Node64* rec = static_cast<Node64*>(nodeRec);
  nodes64Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, hp.Cl, 0, rec);
  const size_t sm = density ? tableBytes(hp) : 0;
#define SPH_D64(LA)                                                                                                     \
  do {                                                                                                                  \
    const unsigned nb = gridFor(n * LA, 128);                                                                           \
    if (density && dt) density64Kernel<true, true, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, maxNperh, dScratch); \
    else if (density) density64Kernel<true, false, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, maxNperh, dScratch); \
    else density64Kernel<false, true, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, maxNperh, dScratch);       \
    if (dt) dtFinal64Kernel<<<1, 1024, 0, s>>>(dScratch, (int)nb, dOut);                                                \
  } while (0)
  SPH_BY_LANES64(SPH_D64)
#undef SPH_D64
  lc->add(dt ? 3 : 2);
}

void launchGradh64(Fields F, void* nodeRec, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                   cudaStream_t s, LaunchCounter* lc) {
  Node64* rec = static_cast<Node64*>(nodeRec);
  nodes64Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, hp.Cl, 0, rec);
#define SPH_G64(LA) gradh64Kernel<LA><<<gridFor(n * LA, 128), 128, tableBytes(hp), s>>>(F, rec, n, g, nl, t, hp)
  SPH_BY_LANES64(SPH_G64)
#undef SPH_G64
  lc->add(2);
}

void launchPair64(Fields F, void* nodeRec, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                  HydroParams hp, double* pacc, cudaStream_t s, LaunchCounter* lc) {
  Node64* rec = static_cast<Node64*>(nodeRec);
  nodes64Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, hp.Cl, 1, rec);
  const size_t sm = tableBytes(hp);
#define SPH_P64(LA)                                                                                              \
  do {                                                                                                           \
    const unsigned nb = gridFor(n * LA, 128);                                                                    \
    if (hp.xsph) {                                                                                               \
      if (hp.limitedQ) pair64Kernel<true, true, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, pacc);    \
      else pair64Kernel<true, false, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, pacc);               \
    } else {                                                                                                     \
      if (hp.limitedQ) pair64Kernel<false, true, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, pacc);   \
      else pair64Kernel<false, false, LA><<<nb, 128, sm, s>>>(F, rec, list, n, g, nl, t, hp, pacc);              \
    }                                                                                                            \
  } while (0)
  SPH_BY_LANES64(SPH_P64)
#undef SPH_P64
  lc->add(2);
}

void launchEnergy64(Fields F, void* velRec, long n, Grid g, NeighborLists nl, const double* pacc, double dt,
                    cudaStream_t s, LaunchCounter* lc) {
  Velocity64* v12 = static_cast<Velocity64*>(velRec);
  velocity64Kernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, 0.5 * dt, v12);
#define SPH_E64(LA) energy64Kernel<LA><<<gridFor(n * LA, 128), 128, 0, s>>>(F, v12, n, g, nl, pacc, dt)
  SPH_BY_LANES64(SPH_E64)
#undef SPH_E64
  lc->add(2);
}

}  // namespace sph
