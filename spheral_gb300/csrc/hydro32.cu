// Mixed-precision sweeps of libsphgpu (sm_103a): the SPH pair loop, density
// sum, grad-h correction and pairwise dt limit in FP32 on cell-relative
// positions.  Time integration, the compatible-energy update, the per-node
// finalisation and all conserved tallies stay in FP64.
//
// Precision design.
//  * Positions are stored relative to the origin of each node's cell
//    (|x_rel| < one cell), so a pair separation is
//    (x_i,rel - x_j,rel) - d cell with d in {-1, 0, 1}: it keeps FP32 digits
//    relative to h instead of relative to the box size.
//  * The pair force Delta_ij is evaluated in a symmetric order,
//    (Prho_i gradW_i + Qacc_i) + (Prho_j gradW_j + Qacc_j), so the two ordered
//    slots (i, j) and (j, i) hold bitwise opposite values: momentum and the
//    compatible-energy split stay exactly antisymmetric despite FP32.
//  * The acceleration and energy-rate sums are Kahan compensated and leave
//    the kernel as the FP64 value s - c of the compensated pair (s, c).
#include "device.cuh"

namespace sph {
namespace {
using namespace dev;


__global__ void prepareKernel(Fields F, Fields32 P, long n, Grid g) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) writeMirrors(F, i, P, i, P.cell[i], g, true);
}

//------------------------------------------------------------------------------
// ASPH pair loop (src/SPH/SPH.cc:294-470) + smoothing-scale moments, FP32.
// Every operation that enters the pair force is deterministic and appears in
// the same order from both sides of the pair (explicit fma / rn intrinsics,
// MUFU reciprocal square root and fast division), so slot (j, i) holds the
// bitwise negation of slot (i, j).
//
// ASPH: H_i, H_j from the FP32 tensor mirror (eta = H r,
// grad W = gW H eta^, both in a fixed order so the pair force stays bitwise
// antisymmetric), the second moment of ASPHClassicSmoothingScale and its
// FP32 finalize.
//
// Two slots per iteration: their gathers are issued together, the next
// iteration's entries loaded ahead.  It serves what pairKernelTensor32 does not:
// XSPH, no compatible energy and the limited Q, with any of the other options.
// 405,224 nodes: XSPH 709 us, limited Q 994 (one slot ahead of another 906 and
// 1250; three slots at two blocks per SM 837 and 1258; two at four 877 and 1294).
template <bool XSPH, bool COMPAT, bool LIMQ>
__global__ void __launch_bounds__(128, 3) pairKernelFP32(Fields F, Fields32 P, const int* __restrict__ list, long n,
                                                      Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                                                      float* __restrict__ pacc) {
  __shared__ float4 ta[kMaxTable / 3];
  __shared__ float2 tb[kMaxTable / 3];
  const int nint = hp.pack32N1 + 1;
  for (int k = threadIdx.x; k < nint; k += blockDim.x) { ta[k] = t.p32a[k]; tb[k] = t.p32b[k]; }
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = mirrorMask(g, ci);
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i], vi = P.velm[i], thi = P.thermo[i];
  const int li = list[i];
  const float mi = vi.w, rhoi = thi.x, Pi = thi.y, csi = thi.z, sOi = thi.w;
  const float4 hi0 = P.hten[i], hi1 = P.hten[P.stride + i];
  const float Hdeti = hi1.z;
  const float extent = (float)hp.extent, invStep = (float)(1.0 / hp.pack32Xstep);
  const int N1 = hp.pack32N1;
  const float Cl = (float)hp.Cl, Cq = (float)hp.Cq, eps2 = (float)hp.eps2;
  const float epsT = (float)hp.epsTensile, WnPerh = (float)hp.WnPerh;
  float DQi[9];   // the limited Q's DvDx of node i
  if (LIMQ) {
    const float4 d0 = P.dvq[i], d1 = P.dvq[P.stride + i], d2 = P.dvq[2 * P.stride + i];
    DQi[0] = d0.x; DQi[1] = d0.y; DQi[2] = d0.z; DQi[3] = d0.w;
    DQi[4] = d1.x; DQi[5] = d1.y; DQi[6] = d1.z; DQi[7] = d1.w; DQi[8] = d2.x;
  }
  const float etaCrit = (float)hp.etaCrit, etaFold = (float)hp.etaFold;
  const float iri = __frcp_rn(rhoi);
  const float mrhoi = mi * iri;
  const float Prhoi0 = __fmul_rn(__fmul_rn(__fmul_rn(sOi, Pi), iri), iri);
  const float mClci = __fmul_rn(-Cl, csi);

  float rhoSum = 0.f, norm = 0.f, maxQ = 0.f, effQ = 0.f, xw = 0.f, xdx = 0.f, xdy = 0.f, xdz = 0.f;
  float sdx = 0.f, cdx = 0.f, sdy = 0.f, cdy = 0.f, sdz = 0.f, cdz = 0.f, se = 0.f, ce = 0.f;
  float gx = 0.f, gy = 0.f, gz = 0.f, m0 = 0.f, m1x = 0.f, m1y = 0.f, m1z = 0.f;
  float D[9], M[9], m2[6];
#pragma unroll
  for (int k = 0; k < 9; ++k) { D[k] = 0.f; M[k] = 0.f; }
#pragma unroll
  for (int k = 0; k < 6; ++k) m2[k] = 0.f;

  const int cnt = nl.count[i];
  // One neighbour slot: the pair's contributions to node i's sums (and the
  // pair acceleration of the compatible-energy sweep at list slot k).
  auto slot = [&](uint32_t ent, const float4& pj, const float4& vj4, const float4& thj, float4 hj0, float4 hj1,
                  long long k) {
    const int j = (int)(ent & kIndexMask), dcode = (int)(ent >> kIndexBits);
    float rx, ry, rz;
    relSepEntry(pi, pj, ent, mm, cx, cy, cz, rx, ry, rz);
    float vxj = vj4.x, vyj = vj4.y, vzj = vj4.z;
    mirrorVel((uint32_t)dcode & mm, vxj, vyj, vzj);
    const float mj = vj4.w, rhoj = thj.x, Pj = thj.y, csj = thj.z, sOj = thj.w;
    const bool same = list[j] == li;
    {   // H_j through the mirrors of the entry
      const uint32_t mq = (uint32_t)dcode & mm;
      if (mq) {
        const float sx = (mq & 3u) ? -1.f : 1.f, sy = (mq & 12u) ? -1.f : 1.f, sz = (mq & 48u) ? -1.f : 1.f;
        hj0.y *= sx * sy;
        hj0.z *= sx * sz;
        hj1.x *= sy * sz;
      }
    }
    const float Hdetj = hj1.z;
    const float irj = __frcp_rn(rhoj);

    float eix, eiy, eiz, ejx, ejy, ejz;
    symDot32(hi0, hi1, rx, ry, rz, eix, eiy, eiz);
    symDot32(hj0, hj1, rx, ry, rz, ejx, ejy, ejz);
    const float e2i = __fmaf_rn(eiz, eiz, __fmaf_rn(eiy, eiy, __fmul_rn(eix, eix)));
    const float e2j = __fmaf_rn(ejz, ejz, __fmaf_rn(ejy, ejy, __fmul_rn(ejx, ejx)));
    const float ri = rsqrtf(fmaxf(e2i, 1.0e-30f)), rj = rsqrtf(fmaxf(e2j, 1.0e-30f));
    const float etai = __fmul_rn(e2i, ri), etaj = __fmul_rn(e2j, rj);
    float Wi, gi, Wj, gj;
    lookupPacked(ta, tb, N1, invStep, etai, extent, Wi, gi);
    lookupPacked(ta, tb, N1, invStep, etaj, extent, Wj, gj);
    const float WSPHi = fabsf(gi);
    Wi *= Hdeti;
    Wj *= Hdetj;
    // gradW = gW H eta/|eta|
    float gwix, gwiy, gwiz, gwjx, gwjy, gwjz;
    const float fi = __fmul_rn(__fmul_rn(Hdeti, gi), ri);
    const float fj = __fmul_rn(__fmul_rn(Hdetj, gj), rj);
    float hx, hy, hz;
    symDot32(hi0, hi1, eix, eiy, eiz, hx, hy, hz);
    gwix = __fmul_rn(fi, hx); gwiy = __fmul_rn(fi, hy); gwiz = __fmul_rn(fi, hz);
    symDot32(hj0, hj1, ejx, ejy, ejz, hx, hy, hz);
    gwjx = __fmul_rn(fj, hx); gwjy = __fmul_rn(fj, hy); gwjz = __fmul_rn(fj, hz);

    if (same) {
      rhoSum += mj * Wi;
      norm += mrhoi * Wi;
    }
    const float vx = vi.x - vxj, vy = vi.y - vyj, vz = vi.z - vzj;
    float vqx = vx, vqy = vy, vqz = vz;
    if (LIMQ) {
      // LimitedMonaghanGingoldViscosity.cc:171-200 in a form symmetric in
      // (i, j): v_q = v_ij - phi (DvDx_i + DvDx_j) x_ij with x_ij = r/2, so
      // the pair force stays bitwise antisymmetric.
      const float4 d0 = P.dvq[j], d1 = P.dvq[P.stride + j], d2 = P.dvq[2 * P.stride + j];
      float Dj[9] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w, d2.x};
      const uint32_t mq = (uint32_t)dcode & mm;
      if (mq) {
        const float sg[3] = {(mq & 3u) ? -1.f : 1.f, (mq & 12u) ? -1.f : 1.f, (mq & 48u) ? -1.f : 1.f};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) Dj[3 * r + cc] *= sg[r] * sg[cc];
      }
      const float hx = 0.5f * rx, hy = 0.5f * ry, hz = 0.5f * rz;
      const float aix = __fmaf_rn(DQi[2], hz, __fmaf_rn(DQi[1], hy, __fmul_rn(DQi[0], hx)));
      const float aiy = __fmaf_rn(DQi[5], hz, __fmaf_rn(DQi[4], hy, __fmul_rn(DQi[3], hx)));
      const float aiz = __fmaf_rn(DQi[8], hz, __fmaf_rn(DQi[7], hy, __fmul_rn(DQi[6], hx)));
      const float ajx = __fmaf_rn(Dj[2], hz, __fmaf_rn(Dj[1], hy, __fmul_rn(Dj[0], hx)));
      const float ajy = __fmaf_rn(Dj[5], hz, __fmaf_rn(Dj[4], hy, __fmul_rn(Dj[3], hx)));
      const float ajz = __fmaf_rn(Dj[8], hz, __fmaf_rn(Dj[7], hy, __fmul_rn(Dj[6], hx)));
      const float gri = __fmaf_rn(aiz, hz, __fmaf_rn(aiy, hy, __fmul_rn(aix, hx)));
      const float grj = __fmaf_rn(ajz, hz, __fmaf_rn(ajy, hy, __fmul_rn(ajx, hx)));
      const float rri = __fdiv_rn(gri, (grj < 0.f ? -1.f : 1.f) * fmaxf(1.0e-30f, fabsf(grj)));
      const float rrj = __fdiv_rn(grj, (gri < 0.f ? -1.f : 1.f) * fmaxf(1.0e-30f, fabsf(gri)));
      const float xl = fminf(rri, rrj);
      float phi = xl > 0.f ? __fdiv_rn(4.0f * xl, __fmul_rn(1.0f + xl, 1.0f + xl)) : 0.f;   // van Leer
      const float etaij = fminf(etai, etaj);
      if (etaij < etaCrit) {
        const float z = __fdiv_rn(etaij - etaCrit, etaFold);
        phi *= expf(-(z * z));
      }
      vqx = __fsub_rn(vx, __fmul_rn(phi, __fadd_rn(aix, ajx)));
      vqy = __fsub_rn(vy, __fmul_rn(phi, __fadd_rn(aiy, ajy)));
      vqz = __fsub_rn(vz, __fmul_rn(phi, __fadd_rn(aiz, ajz)));
    }
    const float mui = __fdividef(__fmaf_rn(vqz, eiz, __fmaf_rn(vqy, eiy, __fmul_rn(vqx, eix))), __fadd_rn(e2i, eps2));
    const float muj = __fdividef(__fmaf_rn(vqz, ejz, __fmaf_rn(vqy, ejy, __fmul_rn(vqx, ejx))), __fadd_rn(e2j, eps2));
    const float mni = fminf(0.f, mui), mnj = fminf(0.f, muj);
    const float li_ = hp.linearInExpansion ? mui : mni;
    const float lj_ = hp.linearInExpansion ? muj : mnj;
    const float qi_ = hp.quadraticInExpansion ? -(mui < 0.f ? -1.f : 1.f) * mui * mui : mni * mni;
    const float qj_ = hp.quadraticInExpansion ? -(muj < 0.f ? -1.f : 1.f) * muj * muj : mnj * mnj;
    const float ei = __fmaf_rn(Cq, qi_, __fmul_rn(mClci, li_));
    const float ej = __fmaf_rn(Cq, qj_, __fmul_rn(__fmul_rn(-Cl, csj), lj_));
    const float qai = __fmul_rn(0.5f, __fmul_rn(ei, iri)), qaj = __fmul_rn(0.5f, __fmul_rn(ej, irj));
    const float Qi = rhoi * ei;
    maxQ = fmaxf(maxQ, Qi);
    effQ += mj * Qi * Wi * irj;
    float Prhoi = Prhoi0, Prhoj = __fmul_rn(__fmul_rn(__fmul_rn(sOj, Pj), irj), irj);
    if (epsT != 0.f) {
      const float ti = Wi / (Hdeti * WnPerh), tj = Wj / (Hdetj * WnPerh);
      Prhoi = __fmul_rn(__fmul_rn(__fmul_rn(sOi, Pi + epsT * (ti * ti * ti * ti) * (Pi < 0.f ? -Pi : 0.f)), iri), iri);
      Prhoj = __fmul_rn(__fmul_rn(__fmul_rn(sOj, Pj + epsT * (tj * tj * tj * tj) * (Pj < 0.f ? -Pj : 0.f)), irj), irj);
    }
    // symmetric-order pair force: (Prho_i + Q_i/2) gradW_i + (Prho_j + Q_j/2) gradW_j
    const float ci_ = __fadd_rn(Prhoi, qai), cj_ = __fadd_rn(Prhoj, qaj);
    const float ddx = __fadd_rn(__fmul_rn(ci_, gwix), __fmul_rn(cj_, gwjx));
    const float ddy = __fadd_rn(__fmul_rn(ci_, gwiy), __fmul_rn(cj_, gwjy));
    const float ddz = __fadd_rn(__fmul_rn(ci_, gwiz), __fmul_rn(cj_, gwjz));
    const float pax = __fmul_rn(-mj, ddx), pay = __fmul_rn(-mj, ddy), paz = __fmul_rn(-mj, ddz);
    sumAdd(sdx, cdx, pax, hp.plainSums);
    sumAdd(sdy, cdy, pay, hp.plainSums);
    sumAdd(sdz, cdz, paz, hp.plainSums);
    if (COMPAT) {
      float* out = pacc + paccSlot(k);
      out[0] = pax;
      out[32] = pay;
      out[64] = paz;
    }
    const float vg = vx * gwix + vy * gwiy + vz * gwiz;
    sumAdd(se, ce, mj * (Prhoi + qai) * vg, hp.plainSums);
    const float mvx = mj * vx, mvy = mj * vy, mvz = mj * vz;
    D[0] -= mvx * gwix; D[1] -= mvx * gwiy; D[2] -= mvx * gwiz;
    D[3] -= mvy * gwix; D[4] -= mvy * gwiy; D[5] -= mvy * gwiz;
    D[6] -= mvz * gwix; D[7] -= mvz * gwiy; D[8] -= mvz * gwiz;
    if (XSPH) {
      const float wx = 0.5f * (mrhoi * Wi + mj * irj * Wj);
      xw += wx;
      xdx -= wx * vx; xdy -= wx * vy; xdz -= wx * vz;
    }
    const float gr = mj * (rhoj - rhoi);
    gx += gr * gwix; gy += gr * gwiy; gz += gr * gwiz;
    const float mrx = mj * rx, mry = mj * ry, mrz = mj * rz;
    M[0] -= mrx * gwix; M[1] -= mrx * gwiy; M[2] -= mrx * gwiz;
    M[3] -= mry * gwix; M[4] -= mry * gwiy; M[5] -= mry * gwiz;
    M[6] -= mrz * gwix; M[7] -= mrz * gwiy; M[8] -= mrz * gwiz;
    const float fw = same ? 1.0f : mj * rhoi / (mi * rhoj);
    const float fwW = fw * WSPHi;
    m0 += fwW;
    m1x -= fwW * eix; m1y -= fwW * eiy; m1z -= fwW * eiz;
    {   // ASPHClassicSmoothingScale second moment: WSPH^2 r r / |r|^5
      const float ir = rsqrtf(fmaxf(rx * rx + ry * ry + rz * rz, 1.0e-30f));
      const float ir2 = ir * ir;
      const float w = fwW * WSPHi * (ir2 * ir2 * ir);
      m2[0] += w * (rx * rx); m2[1] += w * (rx * ry); m2[2] += w * (rx * rz);
      m2[3] += w * (ry * ry); m2[4] += w * (ry * rz); m2[5] += w * (rz * rz);
    }
  };
  constexpr int U = 2;
  uint32_t nx[U];
  if (U <= cnt) {
#pragma unroll
    for (int u = 0; u < U; ++u) nx[u] = nl.nbr[nbSlot(i, u, nl.cap)];
  }
  int q = 0;
  for (; q + U <= cnt; q += U) {
    const long long k0 = nbSlot(i, q, nl.cap);
    uint32_t e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = nx[u];
    if (q + 2 * U <= cnt) {
#pragma unroll
      for (int u = 0; u < U; ++u) nx[u] = nl.nbr[k0 + 32 * (U + u)];
    }
    float4 pp[U], vv[U], tt[U], aa[U], bb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int jj = (int)(e[u] & kIndexMask);
      pp[u] = P.posh[jj]; vv[u] = P.velm[jj]; tt[u] = P.thermo[jj];
      aa[u] = P.hten[jj]; bb[u] = P.hten[P.stride + jj];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) slot(e[u], pp[u], vv[u], tt[u], aa[u], bb[u], k0 + 32 * u);
  }
  for (; q < cnt; ++q) {
    const long long k = nbSlot(i, q, nl.cap);
    const uint32_t ent = nl.nbr[k];
    const int jj = (int)(ent & kIndexMask);
    slot(ent, P.posh[jj], P.velm[jj], P.thermo[jj], P.hten[jj], P.hten[P.stride + jj], k);
  }
  NodeAcc32 a;
  a.rhoSum = rhoSum; a.norm = norm;
  a.dvx = kahanValue(sdx, cdx); a.dvy = kahanValue(sdy, cdy); a.dvz = kahanValue(sdz, cdz);
  a.deps = kahanValue(se, ce);
  a.gx = gx; a.gy = gy; a.gz = gz; a.maxQ = maxQ; a.effQ = effQ;
  a.xw = xw; a.xdx = xdx; a.xdy = xdy; a.xdz = xdz;
  a.m0 = m0; a.m1x = m1x; a.m1y = m1y; a.m1z = m1z;
#pragma unroll
  for (int k = 0; k < 9; ++k) { a.D[k] = D[k]; a.M[k] = M[k]; }
#pragma unroll
  for (int k = 0; k < 6; ++k) a.m2[k] = m2[k];
  a.h0 = hi0;
  a.h1 = hi1;
  finalizeNode32<true>(F, i, li, a, cnt, hp, t.herm);
}

//------------------------------------------------------------------------------
// SPH pair loop for isotropic H (src/SPH/SPH.cc:294-470) + SPHSmoothingScale
// moments, FP32.  With H = a I both kernel gradients lie along the separation,
// grad W = a^4 W'(a |r|) r / |r|, so the pair reduces to scalars times r:
//
//   u     = m_j a_i^4 W'_i / |r|        (velocity gradient, M, grad rho)
//   mu    = a min(v . r, 0) / (a^2 r^2 + eps2),  e = mu (Cq mu - Cl c)
//   C     = Prho + e / (2 rho)          (both sides)
//   g     = -m_j (C_i a_i^4 W'_i + C_j a_j^4 W'_j) / |r|,  a_ij = g r.
//
// The scalar in brackets is formed from commutative operations on values both
// sides of the pair compute alike, and r is bitwise antisymmetric, so for
// equal masses slot (j, i) holds the bitwise negation of slot (i, j).
//
// The limited Q's velocity correction enters only through v . r:
// v_q . r = v . r - 2 phi (q_i + q_j), q = h^T DvDx h, h = r/2, so the Q's
// DvDx is read as its symmetric part, and the van Leer factor of the ratios
// q_i/q_j and q_j/q_i is 4 q_i q_j / (q_i + q_j)^2 for q_i q_j > 0, else 0.
//
// L lanes per node, U slots per iteration (their gathers issued together, the
// next iteration's entries loaded ahead).  KERN 1: cubic B-spline in
// registers, its normalisation A carried by Prho and 1 / (2 rho) (pairInputs32)
// and applied to the other sums per node; 0: packed table.  LEAN 1: one NodeList,
// compensated sums, no tensile correction and the standard Q expansion fixed at
// compile time; 2: the same with plain sums; 0: read from hp.
//------------------------------------------------------------------------------
template <bool XSPH, bool COMPAT, bool LIMQ, int LEAN, bool MIR, int KERN, int L, int U, int MINB>
__global__ void __launch_bounds__(128, MINB) pairKernelIso32(Fields F, Fields32 P, const int* __restrict__ list, long n,
                                                             Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                                                             float* __restrict__ pacc, HalfStep half) {
  constexpr int NT = KERN ? 1 : kTab32;
  __shared__ float4 ta[NT];
  __shared__ float2 tb[NT];
  if (!KERN) loadTable32(ta, tb, t, hp.pack32N1);
  __syncthreads();
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  if (L == 1 && !live) return;
  const long i = live ? node : n - 1;   // whole groups run to the shuffles
  const Kernel32<KERN> K{ta, tb, hp.pack32N1, (float)(1.0 / hp.pack32Xstep)};
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i], vi = P.velm[i], ki = P.pk[i];
  const bool multi = !LEAN && hp.numLists > 1;
  const int li = multi ? list[i] : 0;
  const float ai = pi.w, mi = vi.w, rhoi = ki.x, Prhoi = ki.y, mClci = ki.z, hiri = ki.w;
  const float ai2 = ai * ai, A4i = __fmul_rn(ai2, ai2), Hdeti = ai2 * ai;
  const float Cq = (float)hp.Cq, eps2 = (float)hp.eps2;
  const float epsT = (float)hp.epsTensile, iWnPerh = 1.0f / (float)hp.WnPerh;
  const float etaCrit = (float)hp.etaCrit, iFold = 1.0f / (float)hp.etaFold;
  float4 qa = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 qb = make_float2(0.f, 0.f);
  if (LIMQ) {
    qa = P.dvq[i];
    const float4 q1 = P.dvq[P.stride + i];
    qb = make_float2(q1.x, q1.y);
  }
  PairSums32 a;
  a.w = a.mw = a.ve = a.g0 = a.m1x = a.m1y = a.m1z = a.gx = a.gy = a.gz = a.maxE = 0.f;
  a.xw = a.xdx = a.xdy = a.xdz = 0.f;
#pragma unroll
  for (int k = 0; k < 9; ++k) a.D[k] = 0.f;
#pragma unroll
  for (int k = 0; k < 6; ++k) a.M[k] = 0.f;
  float sdx = 0.f, cdx = 0.f, sdy = 0.f, cdy = 0.f, sdz = 0.f, cdz = 0.f, se = 0.f, ce = 0.f;
  const int plain = LEAN ? LEAN == 2 : hp.plainSums;

  auto slot = [&](uint32_t ent, const float4& pj, const float4& vj4, const float4& kj, const float4& q0,
                  const float4& q1, float* out) {
    const uint32_t dcode = ent >> kIndexBits;
    float rx, ry, rz;
    relSepEntry<MIR>(pi, pj, ent, mm, cx, cy, cz, rx, ry, rz);
    float vxj = vj4.x, vyj = vj4.y, vzj = vj4.z;
    if (MIR) mirrorVel(dcode & mm, vxj, vyj, vzj);
    const float aj = pj.w, mj = vj4.w, rhoj = kj.x, Prhoj = kj.y, mClcj = kj.z, hirj = kj.w;
    const bool same = multi ? (list[ent & kIndexMask] == li) : true;
    const float r2 = __fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmul_rn(rx, rx)));
    const float ir = rsqrtf(fmaxf(r2, 1.0e-36f));
    const float rm = __fmul_rn(r2, ir);
    const float etai = __fmul_rn(ai, rm), etaj = __fmul_rn(aj, rm);
    float w, gi;
    K.both(etai, w, gi);
    float wj = 0.f, gj;
    if (XSPH) K.both(etaj, wj, gj);
    else gj = K.grad(etaj);
    const float aj2 = __fmul_rn(aj, aj);
    const float Gi = __fmul_rn(A4i, gi), Gj = __fmul_rn(__fmul_rn(aj2, aj2), gj);
    const float vx = vi.x - vxj, vy = vi.y - vyj, vz = vi.z - vzj;
    const float vr = __fmaf_rn(vz, rz, __fmaf_rn(vy, ry, __fmul_rn(vx, rx)));
    float vq = vr;
    if (LIMQ) {
      float jxy = q0.w, jxz = q1.x, jyz = q1.y;
      const uint32_t mq = dcode & mm;
      if (MIR && mq) {
        const float sx = (mq & 3u) ? -1.f : 1.f, sy = (mq & 12u) ? -1.f : 1.f, sz = (mq & 48u) ? -1.f : 1.f;
        jxy *= sx * sy; jxz *= sx * sz; jyz *= sy * sz;
      }
      const float xx = __fmul_rn(rx, rx), yy = __fmul_rn(ry, ry), zz = __fmul_rn(rz, rz);
      const float xy = __fmul_rn(rx, ry), xz = __fmul_rn(rx, rz), yz = __fmul_rn(ry, rz);
      const float gri = __fmaf_rn(qb.y, yz, __fmaf_rn(qb.x, xz, __fmaf_rn(qa.w, xy,
                        __fmaf_rn(qa.z, zz, __fmaf_rn(qa.y, yy, __fmul_rn(qa.x, xx))))));
      const float grj = __fmaf_rn(jyz, yz, __fmaf_rn(jxz, xz, __fmaf_rn(jxy, xy,
                        __fmaf_rn(q0.z, zz, __fmaf_rn(q0.y, yy, __fmul_rn(q0.x, xx))))));
      // phi = 4 x (1 - x) with x = q_i / (q_i + q_j), as a symmetric product
      const float sum = __fadd_rn(gri, grj);
      const float inv = __frcp_rn(sum);
      float phi = __fmul_rn(4.0f, __fmul_rn(__fmul_rn(gri, inv), __fmul_rn(grj, inv)));
      if (!(phi > 0.f) || fabsf(sum) < 2.0e-30f) phi = 0.f;
      const float etaij = fminf(etai, etaj);
      if (etaij < etaCrit) {
        const float z = __fmul_rn(etaij - etaCrit, iFold);
        phi *= expf(-(z * z));
      }
      vq = __fmaf_rn(-2.0f * phi, sum, vr);
    }
    // a (a r^2): eta carries the error of the reciprocal root twice, and a^2 one
    // rounding that all nodes of the same h share
    const float di = __fmaf_rn(__fmul_rn(ai, r2), ai, eps2), dj = __fmaf_rn(__fmul_rn(aj, r2), aj, eps2);
    float ei, ej;
    if (LEAN) {
      // the quotient of coincident nodes is 0/0 with eps2 = 0: fminf makes it 0
      const float mni = fminf(0.f, __fdividef(__fmul_rn(ai, vq), di)), mnj = fminf(0.f, __fdividef(__fmul_rn(aj, vq), dj));
      ei = __fmul_rn(mni, __fmaf_rn(Cq, mni, mClci));
      ej = __fmul_rn(mnj, __fmaf_rn(Cq, mnj, mClcj));
    } else {
      const float mui = __fdividef(__fmul_rn(ai, vq), di), muj = __fdividef(__fmul_rn(aj, vq), dj);
      const float mni = fminf(0.f, mui), mnj = fminf(0.f, muj);
      const float li_ = hp.linearInExpansion ? mui : mni, lj_ = hp.linearInExpansion ? muj : mnj;
      const float qi_ = hp.quadraticInExpansion ? -(mui < 0.f ? -1.f : 1.f) * mui * mui : mni * mni;
      const float qj_ = hp.quadraticInExpansion ? -(muj < 0.f ? -1.f : 1.f) * muj * muj : mnj * mnj;
      ei = __fmaf_rn(Cq, qi_, __fmul_rn(mClci, li_));
      ej = __fmaf_rn(Cq, qj_, __fmul_rn(mClcj, lj_));
    }
    float pri = Prhoi, prj = Prhoj;
    if (!LEAN && epsT != 0.f) {   // P_eff = P (1 - epsT (W / W(1/nPerh))^4) in tension
      float wjt = wj;
      if (!XSPH) { float gt; K.both(etaj, wjt, gt); }
      const float ti = w * iWnPerh, tj = wjt * iWnPerh;
      if (pri < 0.f) pri = __fmul_rn(pri, 1.0f - epsT * ((ti * ti) * (ti * ti)));
      if (prj < 0.f) prj = __fmul_rn(prj, 1.0f - epsT * ((tj * tj) * (tj * tj)));
    }
    const float Ci = __fmaf_rn(ei, hiri, pri), Cj = __fmaf_rn(ej, hirj, prj);
    const float S = __fmul_rn(__fadd_rn(__fmul_rn(Ci, Gi), __fmul_rn(Cj, Gj)), ir);
    const float gf = __fmul_rn(-mj, S);
    const float pax = __fmul_rn(gf, rx), pay = __fmul_rn(gf, ry), paz = __fmul_rn(gf, rz);
    if (COMPAT) { out[0] = pax; out[32] = pay; out[64] = paz; }
    sumAdd(sdx, cdx, pax, plain);
    sumAdd(sdy, cdy, pay, plain);
    sumAdd(sdz, cdz, paz, plain);
    const float u = (mj * Gi) * ir;   // a^4 first: m r^2 alone leaves FP32 in CGS units of a star
    sumAdd(se, ce, __fmul_rn(Ci, __fmul_rn(u, vr)), plain);
    const float ux = u * rx, uy = u * ry, uz = u * rz;
    a.D[0] += vx * ux; a.D[1] += vx * uy; a.D[2] += vx * uz;
    a.D[3] += vy * ux; a.D[4] += vy * uy; a.D[5] += vy * uz;
    a.D[6] += vz * ux; a.D[7] += vz * uy; a.D[8] += vz * uz;
    a.M[0] += rx * ux; a.M[1] += rx * uy; a.M[2] += rx * uz;
    a.M[3] += ry * uy; a.M[4] += ry * uz; a.M[5] += rz * uz;
    const float dr = rhoj - rhoi;
    a.gx += dr * ux; a.gy += dr * uy; a.gz += dr * uz;
    if (same) {
      a.w += w;
      a.mw += mj * w;
    }
    a.ve += (mj * hirj) * (ei * (Hdeti * w));
    a.maxE = fmaxf(a.maxE, ei);
    if (XSPH) {
      const float wx = 0.5f * (2.0f * mi * hiri * (ai2 * ai) * w + 2.0f * mj * hirj * (aj2 * aj) * wj);
      a.xw += wx;
      a.xdx -= wx * vx; a.xdy -= wx * vy; a.xdz -= wx * vz;
    }
    float wg = fabsf(gi);
    if (!same) wg *= mj * rhoi / (mi * rhoj);
    a.g0 += wg;
    a.m1x += wg * rx; a.m1y += wg * ry; a.m1z += wg * rz;
  };
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const int cnt = live ? nl.count[i] : 0;
  const int mine = (cnt - sub + L - 1) / L;   // slots of this lane
  const long long s0 = nbSlot(i, 0, nl.cap) + 32 * sub;
  const uint32_t* __restrict__ nb = nl.nbr + s0;
  float* out = COMPAT ? pacc + paccSlot(s0) : nullptr;
  constexpr int ST = 32 * L;
  uint32_t nx[U];
#pragma unroll
  for (int u = 0; u < U; ++u) nx[u] = u < mine ? nb[u * ST] : 0u;
  int q = 0;
  for (; q + U <= mine; q += U) {
    uint32_t e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = nx[u];
    float4 pp[U], vv[U], kk[U], q0[U], q1[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t j = e[u] & kIndexMask;
      pp[u] = P.posh[j]; vv[u] = P.velm[j]; kk[u] = P.pk[j];
      q0[u] = LIMQ ? P.dvq[j] : zero4;
      q1[u] = LIMQ ? P.dvq[P.stride + j] : zero4;
    }
    nb += U * ST;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q + U + u < mine) nx[u] = nb[u * ST];
#pragma unroll
    for (int u = 0; u < U; ++u) slot(e[u], pp[u], vv[u], kk[u], q0[u], q1[u], out + 3 * u * ST);
    if (COMPAT) out += 3 * U * ST;
  }
  if (U > 1) {
#pragma unroll
    for (int u = 0; u < U - 1; ++u) {
      if (q + u < mine) {
        const uint32_t j = nx[u] & kIndexMask;
        slot(nx[u], P.posh[j], P.velm[j], P.pk[j], LIMQ ? P.dvq[j] : zero4, LIMQ ? P.dvq[P.stride + j] : zero4,
             out + 3 * u * ST);
      }
    }
  }
  if (L > 1) {
    a.w = laneSum<L>(a.w); a.mw = laneSum<L>(a.mw); a.ve = laneSum<L>(a.ve); a.g0 = laneSum<L>(a.g0);
    a.m1x = laneSum<L>(a.m1x); a.m1y = laneSum<L>(a.m1y); a.m1z = laneSum<L>(a.m1z);
#pragma unroll
    for (int k = 0; k < 9; ++k) a.D[k] = laneSum<L>(a.D[k]);
#pragma unroll
    for (int k = 0; k < 6; ++k) a.M[k] = laneSum<L>(a.M[k]);
    a.gx = laneSum<L>(a.gx); a.gy = laneSum<L>(a.gy); a.gz = laneSum<L>(a.gz);
    a.maxE = laneMax<L>(a.maxE);
    if (XSPH) {
      a.xw = laneSum<L>(a.xw); a.xdx = laneSum<L>(a.xdx); a.xdy = laneSum<L>(a.xdy); a.xdz = laneSum<L>(a.xdz);
    }
    laneSumKahan<L>(sdx, cdx); laneSumKahan<L>(sdy, cdy); laneSumKahan<L>(sdz, cdz); laneSumKahan<L>(se, ce);
    if (sub != 0 || !live) return;
  }
  a.dvx = kahanValue(sdx, cdx); a.dvy = kahanValue(sdy, cdy); a.dvz = kahanValue(sdz, cdz);
  a.deps = kahanValue(se, ce);
  finalizePair32<KERN == 1>(F, i, list[i], a, ai, mi, rhoi, cnt, hp, t.herm, half);
}

//------------------------------------------------------------------------------
// The same pair loop in the arithmetic of the earlier releases: W and W' from
// the table at |a r| of each side, grad W_i and grad W_j as vectors, the pair
// force added componentwise, one lane per node.  A node whose energy rate
// cancels to rounding takes its share of a pair's work by the sign of that
// rounding (SpecificThermalEnergyPolicy's weights), a 1e-3 change of its
// energy; some node of a large run is always that close, so large runs keep
// these roundings (kExactNodes) and small ones take the cheaper form above.
// Per-node values (rho, Prho, -Cl c, 1/rho) come from the record, mirror
// tests and table branches are gone and the accelerations go out in planes.
// Bound by the L1 data pipe and issue (65 % of the slots at 12 warps per SM);
// writes 12 and reads 4 bytes of DRAM per slot, 0.6 ms at 2.1 M nodes of 119.
// 2.1 M nodes: 2685 -> 2058 us.
//------------------------------------------------------------------------------
template <bool LIMQ, bool MIR, bool SPLINE, bool PLAIN, int U, int MINB>
__global__ void __launch_bounds__(128, MINB) pairKernelLean32(Fields F, Fields32 P, const int* __restrict__ list,
                                                              long n, Grid g, NeighborLists nl, TableDev t,
                                                              HydroParams hp, float* __restrict__ pacc, HalfStep half) {
  __shared__ float4 tg[kTab32];   // (g0, g1, g2, w0)
  __shared__ float2 tw[SPLINE ? 1 : kTab32];
  for (int k = threadIdx.x; k <= hp.pack32N1 + 1; k += blockDim.x) {
    const bool in = k <= hp.pack32N1;
    const float4 A = in ? t.p32a[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 B = in ? t.p32b[k] : make_float2(0.f, 0.f);
    tg[k] = make_float4(A.w, B.x, B.y, A.x);
    if (!SPLINE) tw[k] = make_float2(A.y, A.z);
  }
  __syncthreads();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int N1 = hp.pack32N1;
  const float invStep = (float)(1.0 / hp.pack32Xstep);
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i], vi = P.velm[i], ki = P.pk[i];
  const float ai = pi.w, mi = vi.w, rhoi = ki.x, Prhoi = ki.y, mClci = ki.z, hiri = ki.w;
  const float Hdeti = ai * ai * ai;
  const float Cq = (float)hp.Cq, eps2 = (float)hp.eps2;
  const float etaCrit = (float)hp.etaCrit, etaFold = (float)hp.etaFold;
  float DQi[9];   // the limited Q's DvDx of node i
  if (LIMQ) {
    const float4 d0 = P.dvq[i], d1 = P.dvq[P.stride + i], d2 = P.dvq[2 * P.stride + i];
    DQi[0] = d0.x; DQi[1] = d0.y; DQi[2] = d0.z; DQi[3] = d0.w;
    DQi[4] = d1.x; DQi[5] = d1.y; DQi[6] = d1.z; DQi[7] = d1.w; DQi[8] = d2.x;
  }
  float sw = 0.f, smw = 0.f, sve = 0.f, maxE = 0.f;
  float sdx = 0.f, cdx = 0.f, sdy = 0.f, cdy = 0.f, sdz = 0.f, cdz = 0.f, se = 0.f, ce = 0.f;
  float gx = 0.f, gy = 0.f, gz = 0.f, m0 = 0.f, m1x = 0.f, m1y = 0.f, m1z = 0.f;
  float D[9], M[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) { D[k] = 0.f; M[k] = 0.f; }
  const int cnt = nl.count[i];
  float* out = pacc + paccSlot(nbSlot(i, 0, nl.cap));
  struct Rec {
    float4 p, v, k, d0, d1, d2;
  };
  laneSlots<1, U, Rec>(
      nl, i, 0, cnt,
      [&](uint32_t j, Rec& r) {
        r.p = P.posh[j];
        r.v = P.velm[j];
        r.k = P.pk[j];
        if (LIMQ) { r.d0 = P.dvq[j]; r.d1 = P.dvq[P.stride + j]; r.d2 = P.dvq[2 * P.stride + j]; }
      },
      [&](uint32_t ent, const Rec& q) {
        const uint32_t dcode = ent >> kIndexBits;
        float rx, ry, rz;
        relSepEntry<MIR>(pi, q.p, ent, mm, cx, cy, cz, rx, ry, rz);
        float vxj = q.v.x, vyj = q.v.y, vzj = q.v.z;
        if (MIR) mirrorVel(dcode & mm, vxj, vyj, vzj);
        const float aj = q.p.w, mj = q.v.w, rhoj = q.k.x, Prhoj = q.k.y, mClcj = q.k.z, hirj = q.k.w;
        const float Hdetj = aj * aj * aj;
        const float eix = ai * rx, eiy = ai * ry, eiz = ai * rz;
        const float ejx = aj * rx, ejy = aj * ry, ejz = aj * rz;
        const float e2i = __fmaf_rn(eiz, eiz, __fmaf_rn(eiy, eiy, __fmul_rn(eix, eix)));
        const float e2j = __fmaf_rn(ejz, ejz, __fmaf_rn(ejy, ejy, __fmul_rn(ejx, ejx)));
        const float ri = rsqrtf(fmaxf(e2i, 1.0e-30f)), rj = rsqrtf(fmaxf(e2j, 1.0e-30f));
        const float etai = __fmul_rn(e2i, ri), etaj = __fmul_rn(e2j, rj);
        const int ti = min(N1 + 1, (int)(etai * invStep));
        const float4 Gi = tg[ti], Gj = tg[min(N1 + 1, (int)(etaj * invStep))];
        const float gi = __fmaf_rn(__fmaf_rn(Gi.z, etai, Gi.y), etai, Gi.x);
        const float gj = __fmaf_rn(__fmaf_rn(Gj.z, etaj, Gj.y), etaj, Gj.x);
        // W feeds only massDensitySum, normalization and effViscousPressure
        float w;
        if (SPLINE) w = bsplineW(etai);
        else w = __fmaf_rn(__fmaf_rn(tw[ti].y, etai, tw[ti].x), etai, Gi.w);
        const float fi = __fmul_rn(__fmul_rn(__fmul_rn(Hdeti, gi), ai), ri);
        const float fj = __fmul_rn(__fmul_rn(__fmul_rn(Hdetj, gj), aj), rj);
        const float gwix = fi * eix, gwiy = fi * eiy, gwiz = fi * eiz;
        const float gwjx = fj * ejx, gwjy = fj * ejy, gwjz = fj * ejz;
        const float vx = vi.x - vxj, vy = vi.y - vyj, vz = vi.z - vzj;
        float vqx = vx, vqy = vy, vqz = vz;
        if (LIMQ) {
          // LimitedMonaghanGingoldViscosity.cc:171-200 in a form symmetric in
          // (i, j): v_q = v_ij - phi (DvDx_i + DvDx_j) x_ij with x_ij = r/2
          float Dj[9] = {q.d0.x, q.d0.y, q.d0.z, q.d0.w, q.d1.x, q.d1.y, q.d1.z, q.d1.w, q.d2.x};
          const uint32_t mq = dcode & mm;
          if (MIR && mq) {
            const float sg[3] = {(mq & 3u) ? -1.f : 1.f, (mq & 12u) ? -1.f : 1.f, (mq & 48u) ? -1.f : 1.f};
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
              for (int cc = 0; cc < 3; ++cc) Dj[3 * r + cc] *= sg[r] * sg[cc];
          }
          const float hx = 0.5f * rx, hy = 0.5f * ry, hz = 0.5f * rz;
          const float aix = __fmaf_rn(DQi[2], hz, __fmaf_rn(DQi[1], hy, __fmul_rn(DQi[0], hx)));
          const float aiy = __fmaf_rn(DQi[5], hz, __fmaf_rn(DQi[4], hy, __fmul_rn(DQi[3], hx)));
          const float aiz = __fmaf_rn(DQi[8], hz, __fmaf_rn(DQi[7], hy, __fmul_rn(DQi[6], hx)));
          const float ajx = __fmaf_rn(Dj[2], hz, __fmaf_rn(Dj[1], hy, __fmul_rn(Dj[0], hx)));
          const float ajy = __fmaf_rn(Dj[5], hz, __fmaf_rn(Dj[4], hy, __fmul_rn(Dj[3], hx)));
          const float ajz = __fmaf_rn(Dj[8], hz, __fmaf_rn(Dj[7], hy, __fmul_rn(Dj[6], hx)));
          const float gri = __fmaf_rn(aiz, hz, __fmaf_rn(aiy, hy, __fmul_rn(aix, hx)));
          const float grj = __fmaf_rn(ajz, hz, __fmaf_rn(ajy, hy, __fmul_rn(ajx, hx)));
          const float rri = __fdiv_rn(gri, (grj < 0.f ? -1.f : 1.f) * fmaxf(1.0e-30f, fabsf(grj)));
          const float rrj = __fdiv_rn(grj, (gri < 0.f ? -1.f : 1.f) * fmaxf(1.0e-30f, fabsf(gri)));
          const float xl = fminf(rri, rrj);
          float phi = xl > 0.f ? __fdiv_rn(4.0f * xl, __fmul_rn(1.0f + xl, 1.0f + xl)) : 0.f;   // van Leer
          const float etaij = fminf(etai, etaj);
          if (etaij < etaCrit) {
            const float z = __fdiv_rn(etaij - etaCrit, etaFold);
            phi *= expf(-(z * z));
          }
          vqx = __fsub_rn(vx, __fmul_rn(phi, __fadd_rn(aix, ajx)));
          vqy = __fsub_rn(vy, __fmul_rn(phi, __fadd_rn(aiy, ajy)));
          vqz = __fsub_rn(vz, __fmul_rn(phi, __fadd_rn(aiz, ajz)));
        }
        const float mui = __fdividef(__fmaf_rn(vqz, eiz, __fmaf_rn(vqy, eiy, __fmul_rn(vqx, eix))), __fadd_rn(e2i, eps2));
        const float muj = __fdividef(__fmaf_rn(vqz, ejz, __fmaf_rn(vqy, ejy, __fmul_rn(vqx, ejx))), __fadd_rn(e2j, eps2));
        const float mni = fminf(0.f, mui), mnj = fminf(0.f, muj);
        const float ei = __fmaf_rn(Cq, __fmul_rn(mni, mni), __fmul_rn(mClci, mni));
        const float ej = __fmaf_rn(Cq, __fmul_rn(mnj, mnj), __fmul_rn(mClcj, mnj));
        // (Prho_i + Q_i/2) gradW_i + (Prho_j + Q_j/2) gradW_j: commutative
        // operations only, so slot (j, i) holds the bitwise negation
        const float ci_ = __fadd_rn(Prhoi, __fmul_rn(ei, hiri)), cj_ = __fadd_rn(Prhoj, __fmul_rn(ej, hirj));
        const float ddx = __fadd_rn(__fmul_rn(ci_, gwix), __fmul_rn(cj_, gwjx));
        const float ddy = __fadd_rn(__fmul_rn(ci_, gwiy), __fmul_rn(cj_, gwjy));
        const float ddz = __fadd_rn(__fmul_rn(ci_, gwiz), __fmul_rn(cj_, gwjz));
        const float pax = __fmul_rn(-mj, ddx), pay = __fmul_rn(-mj, ddy), paz = __fmul_rn(-mj, ddz);
        out[0] = pax; out[32] = pay; out[64] = paz;
        out += 96;
        sumAdd(sdx, cdx, pax, PLAIN);
        sumAdd(sdy, cdy, pay, PLAIN);
        sumAdd(sdz, cdz, paz, PLAIN);
        const float vg = vx * gwix + vy * gwiy + vz * gwiz;
        sumAdd(se, ce, __fmul_rn(__fmul_rn(mj, ci_), vg), PLAIN);
        const float mvx = mj * vx, mvy = mj * vy, mvz = mj * vz;
        D[0] -= mvx * gwix; D[1] -= mvx * gwiy; D[2] -= mvx * gwiz;
        D[3] -= mvy * gwix; D[4] -= mvy * gwiy; D[5] -= mvy * gwiz;
        D[6] -= mvz * gwix; D[7] -= mvz * gwiy; D[8] -= mvz * gwiz;
        const float mrx = mj * rx, mry = mj * ry, mrz = mj * rz;
        M[0] -= mrx * gwix; M[1] -= mrx * gwiy; M[2] -= mrx * gwiz;
        M[3] -= mry * gwix; M[4] -= mry * gwiy; M[5] -= mry * gwiz;
        M[6] -= mrz * gwix; M[7] -= mrz * gwiy; M[8] -= mrz * gwiz;
        const float gr = mj * (rhoj - rhoi);
        gx += gr * gwix; gy += gr * gwiy; gz += gr * gwiz;
        sw += w;
        smw += mj * w;
        sve += (mj * hirj) * (ei * (Hdeti * w));
        maxE = fmaxf(maxE, ei);
        const float wg = fabsf(gi);
        m0 += wg;
        m1x -= wg * eix; m1y -= wg * eiy; m1z -= wg * eiz;
      });
  if (SPLINE) { sw = timesSplineA(sw); smw = timesSplineA(smw); sve = timesSplineA(sve); }
  NodeAcc32 a;
  a.rhoSum = Hdeti * smw; a.norm = mi * (2.0f * hiri) * Hdeti * sw;
  a.dvx = kahanValue(sdx, cdx); a.dvy = kahanValue(sdy, cdy); a.dvz = kahanValue(sdz, cdz);
  a.deps = kahanValue(se, ce);
  a.gx = gx; a.gy = gy; a.gz = gz; a.maxQ = rhoi * maxE; a.effQ = 2.0f * rhoi * sve;
  a.xw = a.xdx = a.xdy = a.xdz = 0.f;
  a.m0 = m0; a.m1x = m1x; a.m1y = m1y; a.m1z = m1z;
#pragma unroll
  for (int k = 0; k < 9; ++k) { a.D[k] = D[k]; a.M[k] = M[k]; }
  finalizeNode32<false>(F, i, list[i], a, cnt, hp, t.herm);
  if (half.v) halfStepVelocity(F, i, a.dvx, a.dvy, a.dvz, F.f[F_DEPSDT][i], half);
}

//------------------------------------------------------------------------------
// The ASPH pair loop (tensor H) of the lean path, in the arithmetic of
// pairKernelFP32: the same values in every sum the state reads.  What
// bounds both is the L1 data pipe: five 16-byte gathers per slot and the table.
// Here one 16-byte entry per side holds W' (W, which feeds only massDensitySum,
// normalization and effViscousPressure, is the spline in registers or the
// second table), and what depends on one node comes formed (Fields32::pk).
// L lanes per node, U slots per iteration.  OPT: several NodeLists, plain sums,
// the tensile correction and the Q's expansion options are read from hp.
//------------------------------------------------------------------------------
struct PairRecTensor {
  float4 p, v, k, a, b;
};
template <bool OPT, bool MIR, bool SPLINE, int L, int U, int MINB>
__global__ void __launch_bounds__(128, MINB) pairKernelTensor32(Fields F, Fields32 P, const int* __restrict__ list,
                                                                long n, Grid g, NeighborLists nl, TableDev t,
                                                                HydroParams hp, float* __restrict__ pacc,
                                                                HalfStep half) {
  __shared__ float4 tg[kTab32];   // (g0, g1, g2, w0)
  __shared__ float2 tw[SPLINE ? 1 : kTab32];
  for (int k = threadIdx.x; k <= hp.pack32N1 + 1; k += blockDim.x) {
    const bool in = k <= hp.pack32N1;
    const float4 A = in ? t.p32a[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 B = in ? t.p32b[k] : make_float2(0.f, 0.f);
    tg[k] = make_float4(A.w, B.x, B.y, A.x);
    if (!SPLINE) tw[k] = make_float2(A.y, A.z);
  }
  __syncthreads();
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  if (L == 1 && !live) return;
  const long i = live ? node : n - 1;
  const int N1 = hp.pack32N1;
  const float invStep = (float)(1.0 / hp.pack32Xstep);
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i], vi = P.velm[i], ki = P.pk[i], hi0 = P.hten[i], hi1 = P.hten[P.stride + i];
  const float mi = vi.w, rhoi = ki.x, Prhoi = ki.y, mClci = ki.z, hiri = ki.w, Hdeti = hi1.z;
  const float Cq = (float)hp.Cq, eps2 = (float)hp.eps2;
  const bool multi = OPT && hp.numLists > 1;
  const int li = multi ? list[i] : 0, plain = OPT ? hp.plainSums : 0;
  const float epsT = OPT ? (float)hp.epsTensile : 0.f, iWnPerh = 1.0f / (float)hp.WnPerh;
  float sw = 0.f, smw = 0.f, sve = 0.f, maxE = 0.f;
  float sdx = 0.f, cdx = 0.f, sdy = 0.f, cdy = 0.f, sdz = 0.f, cdz = 0.f, se = 0.f, ce = 0.f;
  float gx = 0.f, gy = 0.f, gz = 0.f, m0 = 0.f, m1x = 0.f, m1y = 0.f, m1z = 0.f;
  float D[9], M[9], m2[6];
#pragma unroll
  for (int k = 0; k < 9; ++k) { D[k] = 0.f; M[k] = 0.f; }
#pragma unroll
  for (int k = 0; k < 6; ++k) m2[k] = 0.f;
  const int cnt = live ? nl.count[i] : 0;
  float* out = pacc + paccSlot(nbSlot(i, 0, nl.cap) + 32 * sub);
  laneSlots<L, U, PairRecTensor>(
      nl, i, sub, cnt,
      [&](uint32_t j, PairRecTensor& r) {
        r.p = P.posh[j];
        r.v = P.velm[j];
        r.k = P.pk[j];
        r.a = P.hten[j];
        r.b = P.hten[P.stride + j];
      },
      [&](uint32_t ent, const PairRecTensor& q) {
        float rx, ry, rz;
        relSepEntry<MIR>(pi, q.p, ent, mm, cx, cy, cz, rx, ry, rz);
        float vxj = q.v.x, vyj = q.v.y, vzj = q.v.z;
        float4 hj0 = q.a, hj1 = q.b;
        if (MIR) {   // velocity and H_j through the mirrors of the entry
          const uint32_t mq = (ent >> kIndexBits) & mm;
          mirrorVel(mq, vxj, vyj, vzj);
          if (mq) {
            const float sx = (mq & 3u) ? -1.f : 1.f, sy = (mq & 12u) ? -1.f : 1.f, sz = (mq & 48u) ? -1.f : 1.f;
            hj0.y *= sx * sy;
            hj0.z *= sx * sz;
            hj1.x *= sy * sz;
          }
        }
        const float mj = q.v.w, rhoj = q.k.x, Prhoj = q.k.y, mClcj = q.k.z, hirj = q.k.w;
        float eix, eiy, eiz, ejx, ejy, ejz;
        symDot32(hi0, hi1, rx, ry, rz, eix, eiy, eiz);
        symDot32(hj0, hj1, rx, ry, rz, ejx, ejy, ejz);
        const float e2i = __fmaf_rn(eiz, eiz, __fmaf_rn(eiy, eiy, __fmul_rn(eix, eix)));
        const float e2j = __fmaf_rn(ejz, ejz, __fmaf_rn(ejy, ejy, __fmul_rn(ejx, ejx)));
        const float ri = rsqrtf(fmaxf(e2i, 1.0e-30f)), rj = rsqrtf(fmaxf(e2j, 1.0e-30f));
        const float etai = __fmul_rn(e2i, ri), etaj = __fmul_rn(e2j, rj);
        const int ti = min(N1 + 1, (int)(etai * invStep));
        const float4 Gi = tg[ti], Gj = tg[min(N1 + 1, (int)(etaj * invStep))];
        const float gi = __fmaf_rn(__fmaf_rn(Gi.z, etai, Gi.y), etai, Gi.x);
        const float gj = __fmaf_rn(__fmaf_rn(Gj.z, etaj, Gj.y), etaj, Gj.x);
        float w;
        if (SPLINE) w = bsplineW(etai);
        else w = __fmaf_rn(__fmaf_rn(tw[ti].y, etai, tw[ti].x), etai, Gi.w);
        const float fi = __fmul_rn(__fmul_rn(Hdeti, gi), ri), fj = __fmul_rn(__fmul_rn(hj1.z, gj), rj);
        float hx, hy, hz;
        symDot32(hi0, hi1, eix, eiy, eiz, hx, hy, hz);
        const float gwix = __fmul_rn(fi, hx), gwiy = __fmul_rn(fi, hy), gwiz = __fmul_rn(fi, hz);
        symDot32(hj0, hj1, ejx, ejy, ejz, hx, hy, hz);
        const float gwjx = __fmul_rn(fj, hx), gwjy = __fmul_rn(fj, hy), gwjz = __fmul_rn(fj, hz);
        const float vx = vi.x - vxj, vy = vi.y - vyj, vz = vi.z - vzj;
        const float mui = __fdividef(__fmaf_rn(vz, eiz, __fmaf_rn(vy, eiy, __fmul_rn(vx, eix))), __fadd_rn(e2i, eps2));
        const float muj = __fdividef(__fmaf_rn(vz, ejz, __fmaf_rn(vy, ejy, __fmul_rn(vx, ejx))), __fadd_rn(e2j, eps2));
        const float mni = fminf(0.f, mui), mnj = fminf(0.f, muj);
        float lmi = mni, lmj = mnj, qmi = __fmul_rn(mni, mni), qmj = __fmul_rn(mnj, mnj);
        float pri = Prhoi, prj = Prhoj;
        if (OPT) {
          if (hp.linearInExpansion) { lmi = mui; lmj = muj; }
          if (hp.quadraticInExpansion) {
            qmi = __fmul_rn(fabsf(mui), -mui);
            qmj = __fmul_rn(fabsf(muj), -muj);
          }
          if (epsT != 0.f) {   // P_eff = P (1 - epsT (W / W(1/nPerh))^4) in tension
            const int tj = min(N1 + 1, (int)(etaj * invStep));
            const float wj = __fmaf_rn(__fmaf_rn(tw[tj].y, etaj, tw[tj].x), etaj, Gj.w);
            const float si = w * iWnPerh, sj = wj * iWnPerh;
            if (pri < 0.f) pri = __fmul_rn(pri, 1.0f - epsT * ((si * si) * (si * si)));
            if (prj < 0.f) prj = __fmul_rn(prj, 1.0f - epsT * ((sj * sj) * (sj * sj)));
          }
        }
        const float ei = __fmaf_rn(Cq, qmi, __fmul_rn(mClci, lmi));
        const float ej = __fmaf_rn(Cq, qmj, __fmul_rn(mClcj, lmj));
        const float ci_ = __fadd_rn(pri, __fmul_rn(ei, hiri)), cj_ = __fadd_rn(prj, __fmul_rn(ej, hirj));
        const float ddx = __fadd_rn(__fmul_rn(ci_, gwix), __fmul_rn(cj_, gwjx));
        const float ddy = __fadd_rn(__fmul_rn(ci_, gwiy), __fmul_rn(cj_, gwjy));
        const float ddz = __fadd_rn(__fmul_rn(ci_, gwiz), __fmul_rn(cj_, gwjz));
        const float pax = __fmul_rn(-mj, ddx), pay = __fmul_rn(-mj, ddy), paz = __fmul_rn(-mj, ddz);
        out[0] = pax; out[32] = pay; out[64] = paz;
        out += 96 * L;
        sumAdd(sdx, cdx, pax, plain);
        sumAdd(sdy, cdy, pay, plain);
        sumAdd(sdz, cdz, paz, plain);
        const float vg = vx * gwix + vy * gwiy + vz * gwiz;
        sumAdd(se, ce, __fmul_rn(__fmul_rn(mj, ci_), vg), plain);
        const float mvx = mj * vx, mvy = mj * vy, mvz = mj * vz;
        D[0] -= mvx * gwix; D[1] -= mvx * gwiy; D[2] -= mvx * gwiz;
        D[3] -= mvy * gwix; D[4] -= mvy * gwiy; D[5] -= mvy * gwiz;
        D[6] -= mvz * gwix; D[7] -= mvz * gwiy; D[8] -= mvz * gwiz;
        const float mrx = mj * rx, mry = mj * ry, mrz = mj * rz;
        M[0] -= mrx * gwix; M[1] -= mrx * gwiy; M[2] -= mrx * gwiz;
        M[3] -= mry * gwix; M[4] -= mry * gwiy; M[5] -= mry * gwiz;
        M[6] -= mrz * gwix; M[7] -= mrz * gwiy; M[8] -= mrz * gwiz;
        const float gr = mj * (rhoj - rhoi);
        gx += gr * gwix; gy += gr * gwiy; gz += gr * gwiz;
        const bool same = multi ? list[ent & kIndexMask] == li : true;
        if (same) {
          sw += w;
          smw += mj * w;
        }
        sve += (mj * hirj) * (ei * (Hdeti * w));
        maxE = fmaxf(maxE, ei);
        const float wf = fabsf(gi);
        const float wg = same ? wf : wf * (mj * rhoi / (mi * rhoj));
        m0 += wg;
        m1x -= wg * eix; m1y -= wg * eiy; m1z -= wg * eiz;
        // ASPHClassicSmoothingScale second moment: WSPH^2 r r / |r|^5
        const float ir = rsqrtf(fmaxf(rx * rx + ry * ry + rz * rz, 1.0e-30f));
        const float ir2 = ir * ir;
        const float w2 = wg * wf * (ir2 * ir2 * ir);
        m2[0] += w2 * (rx * rx); m2[1] += w2 * (rx * ry); m2[2] += w2 * (rx * rz);
        m2[3] += w2 * (ry * ry); m2[4] += w2 * (ry * rz); m2[5] += w2 * (rz * rz);
      });
  if (L > 1) {
    laneSumKahan<L>(sdx, cdx); laneSumKahan<L>(sdy, cdy); laneSumKahan<L>(sdz, cdz); laneSumKahan<L>(se, ce);
    sw = laneSum<L>(sw); smw = laneSum<L>(smw); sve = laneSum<L>(sve); maxE = laneMax<L>(maxE);
    gx = laneSum<L>(gx); gy = laneSum<L>(gy); gz = laneSum<L>(gz);
    m0 = laneSum<L>(m0); m1x = laneSum<L>(m1x); m1y = laneSum<L>(m1y); m1z = laneSum<L>(m1z);
#pragma unroll
    for (int k = 0; k < 9; ++k) { D[k] = laneSum<L>(D[k]); M[k] = laneSum<L>(M[k]); }
#pragma unroll
    for (int k = 0; k < 6; ++k) m2[k] = laneSum<L>(m2[k]);
    if (sub != 0 || !live) return;
  }
  if (SPLINE) { sw = timesSplineA(sw); smw = timesSplineA(smw); sve = timesSplineA(sve); }
  NodeAcc32 a;
  a.rhoSum = Hdeti * smw; a.norm = mi * (2.0f * hiri) * Hdeti * sw;
  a.dvx = kahanValue(sdx, cdx); a.dvy = kahanValue(sdy, cdy); a.dvz = kahanValue(sdz, cdz);
  a.deps = kahanValue(se, ce);
  a.gx = gx; a.gy = gy; a.gz = gz; a.maxQ = rhoi * maxE; a.effQ = 2.0f * rhoi * sve;
  a.xw = a.xdx = a.xdy = a.xdz = 0.f;
  a.m0 = m0; a.m1x = m1x; a.m1y = m1y; a.m1z = m1z;
#pragma unroll
  for (int k = 0; k < 9; ++k) { a.D[k] = D[k]; a.M[k] = M[k]; }
#pragma unroll
  for (int k = 0; k < 6; ++k) a.m2[k] = m2[k];
  a.h0 = hi0;
  a.h1 = hi1;
  finalizeNode32<true>(F, i, list[i], a, cnt, hp, t.herm);
  if (half.v) halfStepVelocity(F, i, a.dvx, a.dvy, a.dvz, F.f[F_DEPSDT][i], half);
}

// The pair sweep's per-node inputs, where the update has not written them.
__global__ void pairInputs32(Fields F, Fields32 P, long n, PairForm pf) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  P.pk[i] = pairRecord(P.thermo[i], pf);
  if (pf.limited) {
    float v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = toFloatRN(F.f[F_DVDXQ_XX + k][i]);
    writeQGradient(P, i, v, pf);
  }
}

// H_j through the mirrors of an entry (FP32 tensor mirror): the off-diagonal
// components flip once per mirrored index.
__device__ __forceinline__ void mirrorTensor32(uint32_t mq, float4& h0, float4& h1) {
  if (mq) {
    const float sx = (mq & 3u) ? -1.f : 1.f, sy = (mq & 12u) ? -1.f : 1.f, sz = (mq & 48u) ? -1.f : 1.f;
    h0.y *= sx * sy;
    h0.z *= sx * sz;
    h1.x *= sy * sz;
  }
}

struct SweepRec {   // a neighbour's record in the density / dt / grad-h sweeps
  float4 p, v, h0, h1;
};

//------------------------------------------------------------------------------
// Density sum (computeSPHSumMassDensity.cc:15-87, gathered) and, with DT, the
// time-step vote of the same step (GenericHydro.cc:113-381: pairwise velocity
// limit on the same neighbour data, node limits with the new density), in one
// pass over the lists.  KERN 1: cubic B-spline in registers, else the table.
// LEAN: one NodeList and compensated sums fixed at compile time.  L lanes per
// node, U slots per iteration.  dtOut receives the smallest dtKey.
//------------------------------------------------------------------------------
template <bool TENSOR, bool DT, bool LEAN, bool MIR, int KERN, int L, int U>
__global__ void __launch_bounds__(sweepBlock(L)) densityKernel32(Fields F, Fields32 P, const int* __restrict__ list, long n,
                                                       Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                                                       float maxNperh, unsigned long long* __restrict__ dtOut) {
  constexpr int NT = KERN ? 1 : kTab32;
  __shared__ float4 ta[NT];
  __shared__ unsigned long long sv[sweepBlock(L) / 32];
  if (!KERN) loadTable32(ta, nullptr, t, hp.pack32N1);
  __syncthreads();
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;   // whole warps run to the shuffles
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i], vi = P.velm[i];
  const bool multi = !LEAN && hp.numLists > 1;
  const int li = multi ? list[i] : 0;
  const Kernel32<KERN> K{ta, nullptr, hp.pack32N1, (float)(1.0 / hp.pack32Xstep)};
  float s = 0.f, c = 0.f, worst = 0.0f;
  // the node scale of GenericHydro::dt: 1/h, the largest eigenvalue of H
  const float lmaxi = TENSOR ? P.hten[P.stride + i].w : pi.w;
  const int cnt = live ? nl.count[i] : 0;
  laneSlots<L, U, SweepRec>(
      nl, i, sub, cnt,
      [&](uint32_t j, SweepRec& r) {
        r.p = P.posh[j];
        r.v = P.velm[j];
        if (TENSOR) { r.h0 = P.hten[j]; r.h1 = P.hten[P.stride + j]; }
      },
      [&](uint32_t ent, SweepRec& r) {
        const uint32_t dcode = ent >> kIndexBits;
        float rx, ry, rz;
        relSepEntry<MIR>(pi, r.p, ent, mm, cx, cy, cz, rx, ry, rz);
        float eta, Hdj, lmaxj;
        if (TENSOR) {   // |H_j r|
          if (MIR) mirrorTensor32(dcode & mm, r.h0, r.h1);
          eta = etaFromSq(eta2Sym32(r.h0, r.h1, rx, ry, rz));
          Hdj = r.h1.z;
          lmaxj = r.h1.w;
        } else {
          const float aj = r.p.w;
          eta = aj * etaFromSq(rx * rx + ry * ry + rz * rz);
          Hdj = aj * aj * aj;
          lmaxj = aj;
        }
        const float w = K.value(eta);
        const bool same = multi ? list[ent & kIndexMask] == li : true;
        sumAdd(s, c, (same ? r.v.w : vi.w) * (Hdj * w), LEAN ? 0 : hp.plainSums);
        if (DT) {
          float vxj = r.v.x, vyj = r.v.y, vzj = r.v.z;
          if (MIR) mirrorVel(dcode & mm, vxj, vyj, vzj);
          const float dx = vi.x - vxj, dy = vi.y - vyj, dz = vi.z - vzj;
          // min over pairs of min(h_i, h_j)/|v_ij| = 1/sqrt(max over pairs of
          // (max(a_i, a_j) |v_ij|)^2): no division or root per pair
          const float am = fmaxf(lmaxi, lmaxj);
          worst = fmaxf(worst, (am * am) * (dx * dx + dy * dy + dz * dz));
        }
      });
  if (L > 1) {
    laneSumKahan<L>(s, c);
    if (DT) worst = laneMax<L>(worst);
  }
  unsigned long long key = ~0ULL;
  if (live && sub == 0) {
    const double Hdeti = TENSOR ? symDet(loadSym(F, F_HT_XX, i)) : (F.f[F_HINV][i] * F.f[F_HINV][i]) * F.f[F_HINV][i];
    const double rho = F.f[F_MASS][i] * (Hdeti * hp.W0) + (KERN ? kSplineA * kahanValue(s, c) : kahanValue(s, c));
    F.f[F_RHO][i] = rho;
    const float rhof = toFloatRN(rho);
    P.thermo[i].x = rhof;
    if (DT && !isGhost(hp, i)) {   // halo copies do not vote
      // FP32 node limits (the vote only picks the minimum; FP64 divide and
      // square root sequences would dominate the sweep otherwise)
      const NodeListParams Li = hp.lists[multi ? li : list[i]];
      const float ax = toFloatRN(F.f[F_DVDT_X][i]), ay = toFloatRN(F.f[F_DVDT_Y][i]), az = toFloatRN(F.f[F_DVDT_Z][i]);
      const float divv = toFloatRN(F.f[F_DVDX_XX][i] + F.f[F_DVDX_YY][i] + F.f[F_DVDX_ZZ][i]);
      int reason;
      const float best = nodeDt32(1.0f / (lmaxi * (float)Li.nPerh), P.thermo[i].z, toFloatRN(F.f[F_MAXQ][i]), rhof,
                                  divv, sqrtf(vi.x * vi.x + vi.y * vi.y + vi.z * vi.z),
                                  sqrtf(ax * ax + ay * ay + az * az), hp.useVelMagDt != 0,
                                  (worst > 0.0f ? rsqrtf(worst) : 3.0e38f) / maxNperh, reason);
      if (reason >= 0) key = dtKey(best, reason);
    }
  }
  if (DT) {
    key = warpMin64(key);
    if ((threadIdx.x & 31) == 0) sv[threadIdx.x >> 5] = key;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < sweepBlock(L) / 32; ++w) key = sv[w] < key ? sv[w] : key;
      if (key != ~0ULL) atomicMin(dtOut, key);
    }
  }
}

//------------------------------------------------------------------------------
// Grad-h correction, FP32 sums (computeSPHOmegaGradhCorrection.cc:15-116).
//------------------------------------------------------------------------------
// LEAN: compensated sums fixed at compile time.
template <bool TENSOR, bool LEAN, bool MIR, int KERN, int L, int U>
__global__ void __launch_bounds__(sweepBlock(L)) gradhKernel32(Fields F, Fields32 P, long n, Grid g, NeighborLists nl,
                                                     TableDev t, HydroParams hp, PairForm pf) {
  constexpr int NT = KERN ? 1 : kTab32;
  __shared__ float4 ta[NT];
  __shared__ float2 tb[NT];
  if (!KERN) loadTable32(ta, tb, t, hp.pack32N1);
  __syncthreads();
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  if (L == 1 && !live) return;
  const long i = live ? node : n - 1;
  const Kernel32<KERN> K{ta, tb, hp.pack32N1, (float)(1.0 / hp.pack32Xstep)};
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float cx = g.cellf[0], cy = g.cellf[1], cz = g.cellf[2];
  const float4 pi = P.posh[i];
  const float ai = pi.w;
  float4 hi0 = make_float4(0.f, 0.f, 0.f, 0.f), hi1 = hi0;
  if (TENSOR) { hi0 = P.hten[i]; hi1 = P.hten[P.stride + i]; }
  float ws = 0.f, wc = 0.f, gs = 0.f, gc = 0.f;
  const int cnt = live ? nl.count[i] : 0;
  laneSlots<L, U, float4>(
      nl, i, sub, cnt, [&](uint32_t j, float4& p) { p = P.posh[j]; },
      [&](uint32_t ent, const float4& p) {
        float rx, ry, rz;
        relSepEntry<MIR>(pi, p, ent, mm, cx, cy, cz, rx, ry, rz);
        float eta;
        if (TENSOR) eta = etaFromSq(eta2Sym32(hi0, hi1, rx, ry, rz));
        else if (KERN) eta = ai * etaFromSq(__fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmul_rn(rx, rx))));
        else {
          const float ex = ai * rx, ey = ai * ry, ez = ai * rz;
          eta = etaFromSq(__fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex))));
        }
        float w, gr;
        K.both(eta, w, gr);
        sumAdd(ws, wc, w, LEAN ? 0 : hp.plainSums);
        sumAdd(gs, gc, __fmul_rn(eta, gr), LEAN ? 0 : hp.plainSums);
      });
  if (L > 1) {
    laneSumKahan<L>(ws, wc);
    laneSumKahan<L>(gs, gc);
    if (sub != 0 || !live) return;
  }
  // Omega = -sum eta dW/deta / (3 (sum W + W0)) (Hdet cancels), in FP32 from
  // the compensated sums
  float omega = 1.0f;
  if (cnt > 0) omega = fmaxf(1.0e-30f, -(gs - gc) / (3.0f * ((ws - wc) + (KERN ? 1.0f : (float)hp.W0))));
  F.f[F_OMEGA][i] = toDouble(omega);
  const float iom = omega / (omega * omega + 1.0e-30f);
  P.thermo[i].w = iom;
  if (pf.on) {
    float4 th = P.thermo[i];
    th.w = iom;
    P.pk[i] = pairRecord(th, pf);
  }
}

//------------------------------------------------------------------------------
// GenericHydro::dt with the pairwise velocity limit in FP32 and the node
// limits in FP64 (voteNode32).
//------------------------------------------------------------------------------
template <bool TENSOR, bool MIR, int L, int U>
__global__ void __launch_bounds__(128) dtKernel32(Fields F, Fields32 P, const int* __restrict__ list, long n, Grid g,
                                                  NeighborLists nl, HydroParams hp, double maxNperh,
                                                  StepScratch* __restrict__ sc) {
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  const long i = live ? node : n - 1;
  int ci[3];
  unpackCell(P.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float4 vi = P.velm[i];
  const float lmaxi = TENSOR ? P.hten[P.stride + i].w : P.posh[i].w;
  float worst = 0.0f;
  laneSlots<L, U, float4>(
      nl, i, sub, live ? nl.count[i] : 0,
      [&](uint32_t j, float4& v) {
        v = P.velm[j];
        v.w = TENSOR ? P.hten[P.stride + j].w : P.posh[j].w;
      },
      [&](uint32_t ent, const float4& v) {
        float vxj = v.x, vyj = v.y, vzj = v.z;
        if (MIR) mirrorVel((ent >> kIndexBits) & mm, vxj, vyj, vzj);
        const float dx = vi.x - vxj, dy = vi.y - vyj, dz = vi.z - vzj;
        const float am = fmaxf(lmaxi, v.w);
        worst = fmaxf(worst, (am * am) * (dx * dx + dy * dy + dz * dz));
      });
  if (L > 1) worst = laneMax<L>(worst);
  voteNode32<TENSOR>(F, hp, list, i, live && sub == 0 && !isGhost(hp, i), lmaxi, vi, worst, maxNperh, sc);
}

__global__ void dtInitKernel(StepScratch* __restrict__ sc) { resetVote(sc); }

//------------------------------------------------------------------------------
// Compatible-energy sweep of the mixed mode (SpecificThermalEnergyPolicy.cc:110-173).
// v12 = v0 + a dt/2 is formed once per node in FP64 from the beginning-of-step
// velocity; the per-pair work
// du_ij = (v12_j - v12_i) . pacc_ij uses the FP64 velocity difference rounded
// to FP32 and the FP32 pair acceleration; the weighted shares are summed and
// applied to the specific energy in FP64.
//------------------------------------------------------------------------------
__global__ void halfStepVelocityKernel(Fields F, long n, HalfStep half) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  halfStepVelocity(F, i, F.f[F_DVDT_X][i], F.f[F_DVDT_Y][i], F.f[F_DVDT_Z][i], F.f[F_DEPSDT][i], half);
}

// B: slots per batch (the gathers and pair-acceleration reads in flight per
// thread); every B adds in the same slot order, so the result is the same.
// L lanes per node.
template <bool MIR, int B, int L>
__global__ void __launch_bounds__(sweepBlock(L)) energyKernel32(Fields F, long n, Grid g, NeighborLists nl,
                                                      const float4* __restrict__ v12,
                                                      const float* __restrict__ pacc, double dt) {
  const long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = node < n;
  if (L == 1 && !live) return;
  const long i = live ? node : n - 1;
  int ci[3];
  unpackCell(nl.cell[i], ci);
  const uint32_t mm = MIR ? mirrorMask(g, ci) : 0u;
  const float4 hi = v12[2 * i], lo = v12[2 * i + 1];
  const float d0i = hi.w;
  const float feps = (float)DBL_EPSILON;
  float s = 0.0f, c = 0.0f;
  // One slot: du = (v_j - v_i) . a_ij with the half-step velocities as
  // hi + lo float pairs, split by the DepsDt0 weights.
  auto slot = [&](uint32_t ent, float4 hj, float4 lj, float p0, float p1, float p2) {
    const uint32_t dcode = ent >> kIndexBits;
    float hx = hj.x, hy = hj.y, hz = hj.z, lx = lj.x, ly = lj.y, lz = lj.z;
    const uint32_t mir = dcode & mm;
    if (MIR && mir) {
      if (mir & 3u) { hx = -hx; lx = -lx; }
      if (mir & 12u) { hy = -hy; ly = -ly; }
      if (mir & 48u) { hz = -hz; lz = -lz; }
    }
    // (hi_j - hi_i) + (lo_j - lo_i): the FP64 difference to FP32 rounding
    const float wx = __fadd_rn(__fsub_rn(hx, hi.x), __fsub_rn(lx, lo.x));
    const float wy = __fadd_rn(__fsub_rn(hy, hi.y), __fsub_rn(ly, lo.y));
    const float wz = __fadd_rn(__fsub_rn(hz, hi.z), __fsub_rn(lz, lo.z));
    const float du = __fmaf_rn(wz, p2, __fmaf_rn(wy, p1, __fmul_rn(wx, p0)));
    const float weighti = fmaxf(feps, du < 0.0f ? -d0i : d0i);
    const float weightj = fmaxf(feps, du < 0.0f ? -hj.w : hj.w);
    // The split of du between i and j: both sides divide by the same sum with
    // IEEE rounding, so the two shares add up to du with unbiased rounding
    // errors.  (An approximate reciprocal here, even after a Newton step,
    // leaves a one-signed error on every pair, which accumulates into a
    // steady energy drift.)
    kahanAdd(s, c, __fmul_rn(__fdiv_rn(weighti, __fadd_rn(weighti, weightj)), du));
  };
  // Batches of B slots: all their loads are issued before any is used, so B
  // gathers and pair-acceleration reads are in flight together.  The entries
  // of the next batch are loaded while this batch's gathers are in flight.
  const int cnt = live ? nl.count[i] : 0;
  const int mine = (cnt - sub + L - 1) / L;   // slots of this lane
  const long long s0 = nbSlot(i, 0, nl.cap) + 32 * sub;
  const uint32_t* __restrict__ nb = nl.nbr + s0;
  const float* __restrict__ pa = pacc + paccSlot(s0);
  constexpr int ST = 32 * L;
  uint32_t en[B];
#pragma unroll
  for (int u = 0; u < B; ++u) en[u] = u < mine ? nb[u * ST] : 0u;
  int q = 0;
  for (; q + B <= mine; q += B) {
    uint32_t e[B];
    Rec32B v[B];
    float p[B][3];
#pragma unroll
    for (int u = 0; u < B; ++u) e[u] = en[u];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const uint32_t j = e[u] & kIndexMask;
      v[u] = load32B(v12 + 2 * (size_t)j);
#pragma unroll
      for (int k = 0; k < 3; ++k) p[u][k] = pa[3 * u * ST + 32 * k];
    }
    nb += B * ST;
    pa += 3 * B * ST;
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (q + B + u < mine) en[u] = nb[u * ST];
#pragma unroll
    for (int u = 0; u < B; ++u) slot(e[u], v[u].a, v[u].b, p[u][0], p[u][1], p[u][2]);
  }
  for (; q < mine; ++q, nb += ST, pa += 3 * ST) {
    const uint32_t ent = nb[0];
    const uint32_t j = ent & kIndexMask;
    const Rec32B v = load32B(v12 + 2 * (size_t)j);
    slot(ent, v.a, v.b, pa[0], pa[32], pa[64]);
  }
  if (L > 1) {
    laneSumKahan<L>(s, c);
    if (sub != 0 || !live) return;
  }
  const double sum = kahanValue(s, c);
  F.f[F_DEPS_COMPAT][i] = sum;
  F.f[F_EPS][i] = F.f[F_EPS0][i] + sum * dt;
}

inline unsigned gridFor(long n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

void launchPrepareFP32(Fields F, Fields32 F32, long n, Grid g, cudaStream_t s, LaunchCounter* lc) {
  prepareKernel<<<gridFor(n, 256), 256, 0, s>>>(F, F32, n, g);
  lc->add(1);
}

constexpr int kDensU = 2, kGradhU = 4;   // slots per iteration of the density and grad-h sweeps
// The lean path: one NodeList, compensated sums, the standard Q, no tensile
// correction, compatible energy, no XSPH.  From kExactNodes on, and in every
// domain of a decomposed run (the two sides of a pair across a cut are evaluated
// by domains of different node counts), it keeps the earlier arithmetic; else the
// reduced one, with the spline in registers.
static bool leanPair(const HydroParams& hp) {
  return hp.epsTensile == 0.0 && !hp.linearInExpansion && !hp.quadraticInExpansion && !hp.xsph && hp.compatible && hp.numLists == 1;
}
static bool exactPair(long n, const HydroParams& hp) { return leanPair(hp) && (n >= kExactNodes || hp.decomposed); }
static bool reducedPair(long n, const HydroParams& hp) { return leanPair(hp) && !exactPair(n, hp) && hp.cubicSpline; }
// and with tensor H: none of the run-time options either
static bool leanTensor(const HydroParams& hp) { return leanPair(hp) && !hp.plainSums && !hp.limitedQ; }
// The options read at run time (pairKernelIso32's LEAN 0 and the tensor forms).
// Isotropic: one lane per node with two slots in flight where its blocks fill
// their one wave (three blocks of 128 on each of 152 SMs) or several, else four
// lanes.  The tensile correction at 21,952 / 50,653 / 97,336 / 405,224 nodes:
// one lane 41 / 52 / 108 / 321 us, four 31 / 67 / 102 / 457.
static int lanesGeneral(long n) { return n >= kExactNodes || (n >= 40000 && n <= 58368) ? 1 : 4; }
// Tensor H, us with 1 / 2 / 4 / 8 lanes: 10,648 nodes 47/39/37/60, 17,576 47/39/62/87,
// 21,952 55/47/68/107, 29,791 56/72/90/139, 97,336 136/169/231/390.
static int lanesTensor(long n) { return n >= 25000 ? 1 : (n >= 15000 ? 2 : 4); }
constexpr long kTensorVariants = 100000;   // from here the variants are worth timing
bool pairVariantsDiffer32(long n, const HydroParams& hp) {
  if (hp.crk) return n >= kCRKOneLane && !hp.xsph && hp.compatible;
  if (hp.asph) return !hp.xsph && hp.compatible && !hp.limitedQ && n >= (leanTensor(hp) ? kTensorVariants : 20000);
  return exactPair(n, hp) && hp.cubicSpline && !hp.limitedQ;
}
PairForm pairForm32(long n, const HydroParams& hp) {
  PairForm f;
  f.on = 1;
  f.Cl = (float)hp.Cl;
  f.spline = !hp.asph && reducedPair(n, hp) ? 1 : 0;
  f.limited = hp.limitedQ;
  f.full = exactPair(n, hp) ? 1 : 0;
  return f;
}

// variant (isotropic, from kExactNodes on, standard Q): five slots per iteration
// at three blocks per SM (even) or four at two (odd).  Few warps with many
// gathers each keep the neighbours' lines in L1: 2.1 M nodes 2081 / 2093 us,
// four at three 2188, six at two 2222.
void launchPairFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                    HydroParams hp, float* pacc, int variant, bool inputs, const HalfStep& half, cudaStream_t s,
                    LaunchCounter* lc) {
  const int b = 128;
  if (hp.asph) {
    const unsigned gb = gridFor(n, b);
    // Lean path, one lane per node (303,912 nodes): variants 0 to 3 are two slots
    // per iteration at three blocks per SM (579 us), one at four (593), two at four
    // (578), three at two (567); below 100,000 nodes variant 0 (79,507 nodes:
    // 125 us), and several lanes per node below 25,000.  The run-time options: one
    // lane from 20,000 nodes on (two NodeLists, 21,952 nodes: 73 us, four lanes 76;
    // 50,653: 93 and 145), four below (10,648: 41).
    if (!hp.xsph && hp.compatible && !hp.limitedQ) {
      if (!inputs) pairInputs32<<<gridFor(n, 256), 256, 0, s>>>(F, F32, n, pairForm32(n, hp));
#define SPH_TEN(OP, MI, SP, LA, U, MB) \
  pairKernelTensor32<OP, MI, SP, LA, U, MB><<<gridFor(n * LA, b), b, 0, s>>>(F, F32, list, n, g, nl, t, hp, pacc, half)
#define SPH_TENL(MI, LA, U, MB) do { if (hp.cubicSpline) SPH_TEN(false, MI, true, LA, U, MB); else SPH_TEN(false, MI, false, LA, U, MB); } while (0)
#define SPH_TENM(LA, U, MB) do { if (hasMirrors(g)) SPH_TENL(true, LA, U, MB); else SPH_TENL(false, LA, U, MB); } while (0)
      const int L = lanesTensor(n);
      if (!leanTensor(hp)) {
        if (n < 20000) SPH_TEN(true, true, false, 4, 2, 3);
        else if (variant == 1) SPH_TEN(true, true, false, 1, 3, 2);
        else if (variant == 2) SPH_TEN(true, true, false, 1, 2, 4);
        else if (variant == 3) SPH_TEN(true, true, false, 1, 1, 4);
        else SPH_TEN(true, true, false, 1, 2, 3);
      } else if (L == 1) {
        const int v = n >= kTensorVariants ? variant : 0;
        if (v == 1) SPH_TENM(1, 1, 4);
        else if (v == 2) SPH_TENM(1, 2, 4);
        else if (v == 3) SPH_TENM(1, 3, 2);
        else SPH_TENM(1, 2, 3);
      } else if (L == 2) SPH_TENM(2, 2, 3);
      else SPH_TENM(4, 2, 3);
#undef SPH_TENM
#undef SPH_TENL
#undef SPH_TEN
      lc->add(inputs ? 1 : 2);
      return;
    }
#define SPH_TENG(X, C)                                                                                          \
  do {                                                                                                          \
    if (hp.limitedQ) pairKernelFP32<X, C, true><<<gridFor(n, b), b, 0, s>>>(F, F32, list, n, g, nl, t, hp, pacc); \
    else pairKernelFP32<X, C, false><<<gridFor(n, b), b, 0, s>>>(F, F32, list, n, g, nl, t, hp, pacc);            \
  } while (0)
    if (hp.xsph) { if (hp.compatible) SPH_TENG(true, true); else SPH_TENG(true, false); }
    else { if (hp.compatible) SPH_TENG(false, true); else SPH_TENG(false, false); }
#undef SPH_TENG
    if (half.v) halfStepVelocityKernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, half);
    lc->add(half.v ? 2 : 1);
    return;
  }
  const bool exact = exactPair(n, hp), fast = reducedPair(n, hp);
  if (!inputs) pairInputs32<<<gridFor(n, 256), 256, 0, s>>>(F, F32, n, pairForm32(n, hp));
  const int L = lanesPair(n);
#define SPH_ISO(X, C, Q, LE, MI, K, LA, U, MB) \
  pairKernelIso32<X, C, Q, LE, MI, K, LA, U, MB><<<gridFor(n * LA, b), b, 0, s>>>(F, F32, list, n, g, nl, t, hp, pacc, half)
  if (exact) {
#define SPH_LEAN(Q, MI, SP, PL, U, MB) \
  pairKernelLean32<Q, MI, SP, PL, U, MB><<<gridFor(n, b), b, 0, s>>>(F, F32, list, n, g, nl, t, hp, pacc, half)
#define SPH_LEANP(MI, PL)                                                                      \
  do {                                                                                         \
    if (hp.limitedQ) { if (hp.cubicSpline) SPH_LEAN(true, MI, true, PL, 2, 3); else SPH_LEAN(true, MI, false, PL, 2, 3); } \
    else if (!hp.cubicSpline) SPH_LEAN(false, MI, false, PL, 2, 3);                            \
    else if (variant & 1) SPH_LEAN(false, MI, true, PL, 4, 2);                                 \
    else SPH_LEAN(false, MI, true, PL, 5, 3);                                                  \
  } while (0)
    if (hasMirrors(g)) { if (hp.plainSums) SPH_LEANP(true, true); else SPH_LEANP(true, false); }
    else { if (hp.plainSums) SPH_LEANP(false, true); else SPH_LEANP(false, false); }
#undef SPH_LEANP
#undef SPH_LEAN
  } else if (fast) {
#define SPH_ISOL(Q, LE, MI)                                                               \
  if (L == 2) SPH_ISO(false, true, Q, LE, MI, 1, 2, 2, 4);                                \
  else SPH_ISO(false, true, Q, LE, MI, 1, 4, 2, 4);
    if (hp.plainSums) {
      if (hp.limitedQ) { SPH_ISOL(true, 2, true) } else { SPH_ISOL(false, 2, true) }
    } else if (hasMirrors(g)) {
      if (hp.limitedQ) { SPH_ISOL(true, 1, true) } else { SPH_ISOL(false, 1, true) }
    } else {
      if (hp.limitedQ) { SPH_ISOL(true, 1, false) } else { SPH_ISOL(false, 1, false) }
    }
#undef SPH_ISOL
  } else {
#define SPH_ISOG(X, C, Q)                                                              \
  do {                                                                                 \
    if (lanesGeneral(n) == 1) SPH_ISO(X, C, Q, 0, true, 0, 1, 2, 3);                   \
    else SPH_ISO(X, C, Q, 0, true, 0, 4, 1, 3);                                        \
  } while (0)
#define SPH_ISOQ(X, C) do { if (hp.limitedQ) SPH_ISOG(X, C, true); else SPH_ISOG(X, C, false); } while (0)
    if (hp.xsph) { if (hp.compatible) SPH_ISOQ(true, true); else SPH_ISOQ(true, false); }
    else { if (hp.compatible) SPH_ISOQ(false, true); else SPH_ISOQ(false, false); }
#undef SPH_ISOQ
#undef SPH_ISOG
  }
#undef SPH_ISO
  lc->add(inputs ? 1 : 2);
}

// Slots per iteration of the density and grad-h sweeps: see densityKernel32.
static void launchDensity32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                            const HydroParams& hp, bool dt, double maxNperh, unsigned long long* key, cudaStream_t s) {
  const int L = lanesSweep(n);
#define SPH_DENS(T, D, LE, MI, K, LA, U) \
  densityKernel32<T, D, LE, MI, K, LA, U><<<gridFor(n * LA, sweepBlock(LA)), sweepBlock(LA), 0, s>>>(F, F32, list, n, g, nl, t, hp, (float)maxNperh, key)
  // lean: one NodeList and compensated sums fixed at compile time
  const bool lean = hp.numLists == 1 && !hp.plainSums;
  if (dt && lean && (n >= kExactNodes || hp.asph)) {
#define SPH_DX(LA)                                                          \
  do {                                                                      \
    if (hp.asph) SPH_DENS(true, true, true, true, 0, LA, 2);                \
    else if (hasMirrors(g)) SPH_DENS(false, true, true, true, 0, LA, kDensU); \
    else SPH_DENS(false, true, true, false, 0, LA, kDensU);                 \
  } while (0)
    SPH_BY_LANES(L, SPH_DX)
#undef SPH_DX
  } else if (dt && lean && hp.cubicSpline) {
#define SPH_DL(LA)                                                          \
  do {                                                                      \
    if (hasMirrors(g)) SPH_DENS(false, true, true, true, 1, LA, kDensU);    \
    else SPH_DENS(false, true, true, false, 1, LA, kDensU);                 \
  } while (0)
    SPH_BY_LANES(L, SPH_DL)
#undef SPH_DL
  } else if (L == 1 && !hp.asph) {   // 2,000,376 nodes, two NodeLists: 633 us, four lanes 801; tensor H: 313 against 255
    if (dt) SPH_DENS(false, true, false, true, 0, 1, 2); else SPH_DENS(false, false, false, true, 0, 1, 2);
  } else if (dt) {
    if (hp.asph) SPH_DENS(true, true, false, true, 0, 4, 1); else SPH_DENS(false, true, false, true, 0, 4, 2);
  } else {
    if (hp.asph) SPH_DENS(true, false, false, true, 0, 4, 1); else SPH_DENS(false, false, false, true, 0, 4, 2);
  }
#undef SPH_DENS
}

void launchSumDensityFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                          HydroParams hp, cudaStream_t s, LaunchCounter* lc) {
  launchDensity32(F, F32, list, n, g, nl, t, hp, false, 1.0, nullptr, s);
  lc->add(1);
}

void launchGradhFP32(Fields F, Fields32 F32, long n, Grid g, NeighborLists nl, TableDev t, HydroParams hp,
                     const PairForm& pf, cudaStream_t s, LaunchCounter* lc) {
  const int L = lanesSweep(n);
#define SPH_GH(T, LE, MI, K, LA, U) gradhKernel32<T, LE, MI, K, LA, U><<<gridFor(n * LA, sweepBlock(LA)), sweepBlock(LA), 0, s>>>(F, F32, n, g, nl, t, hp, pf)
  if (!hp.plainSums && (n >= kExactNodes || hp.asph)) {
#define SPH_GX(LA)                                                    \
  do {                                                                \
    if (hp.asph) SPH_GH(true, true, true, 0, LA, 2);                  \
    else if (hasMirrors(g)) SPH_GH(false, true, true, 0, LA, kGradhU); \
    else SPH_GH(false, true, false, 0, LA, kGradhU);                  \
  } while (0)
    SPH_BY_LANES(L, SPH_GX)
#undef SPH_GX
  } else if (!hp.plainSums && hp.cubicSpline) {
#define SPH_GL(LA)                                                    \
  do {                                                                \
    if (hasMirrors(g)) SPH_GH(false, true, true, 1, LA, kGradhU);     \
    else SPH_GH(false, true, false, 1, LA, kGradhU);                  \
  } while (0)
    SPH_BY_LANES(L, SPH_GL)
#undef SPH_GL
  } else if (hp.asph) {
    SPH_GH(true, false, true, 0, 4, 2);
  } else if (L == 1) {
    SPH_GH(false, false, true, 0, 1, kGradhU);
  } else {
    SPH_GH(false, false, true, 0, 4, 2);
  }
#undef SPH_GH
  lc->add(1);
}

void launchDtReset(StepScratch* sc, cudaStream_t s, LaunchCounter* lc) {
  dtInitKernel<<<1, 1, 0, s>>>(sc);
  lc->add(1);
}
void launchDtFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, HydroParams hp,
                  double maxNperh, StepScratch* sc, cudaStream_t s, LaunchCounter* lc) {
  dtInitKernel<<<1, 1, 0, s>>>(sc);
  const int L = lanesSweep(n);
#define SPH_DT(LA)                                                                                                     \
  do {                                                                                                                 \
    if (hp.asph) dtKernel32<true, true, LA, 2><<<gridFor(n * LA, 128), 128, 0, s>>>(F, F32, list, n, g, nl, hp, maxNperh, sc); \
    else dtKernel32<false, true, LA, 2><<<gridFor(n * LA, 128), 128, 0, s>>>(F, F32, list, n, g, nl, hp, maxNperh, sc);        \
  } while (0)
  SPH_BY_LANES(L, SPH_DT)
#undef SPH_DT
  lc->add(2);
}

void launchCompatibleEnergyFP32(Fields F, long n, Grid g, NeighborLists nl, const float* pacc, float4* v12,
                                double dt, int variant, bool half, cudaStream_t s,
                                LaunchCounter* lc) {
  if (half) halfStepVelocityKernel<<<gridFor(n, 256), 256, 0, s>>>(F, n, HalfStep{v12, 0.5 * dt});
  const int L = lanesEnergy(n);
#define SPH_EN(B, LA)                                                                                                    \
  if (hasMirrors(g)) energyKernel32<true, B, LA><<<gridFor(n * LA, sweepBlock(LA)), sweepBlock(LA), 0, s>>>(F, n, g, nl, v12, pacc, dt); \
  else energyKernel32<false, B, LA><<<gridFor(n * LA, sweepBlock(LA)), sweepBlock(LA), 0, s>>>(F, n, g, nl, v12, pacc, dt)
#define SPH_ENL(B)                 \
  switch (L) {                     \
    case 1: SPH_EN(B, 1); break;   \
    case 2: SPH_EN(B, 2); break;   \
    case 4: SPH_EN(B, 4); break;   \
    default: SPH_EN(B, 16); break; \
  }
  if (variant == 1) { SPH_ENL(8) } else if (variant == 2) { SPH_ENL(2) } else { SPH_ENL(4) }
#undef SPH_ENL
#undef SPH_EN
  lc->add(half ? 2 : 1);
}

void launchDensityDtFP32(Fields F, Fields32 F32, const int* list, long n, Grid g, NeighborLists nl, TableDev t,
                         HydroParams hp, double maxNperh, StepScratch* sc, bool reset, cudaStream_t s,
                         LaunchCounter* lc) {
  if (reset) dtInitKernel<<<1, 1, 0, s>>>(sc);
  launchDensity32(F, F32, list, n, g, nl, t, hp, true, maxNperh, &sc->voteKey, s);
  lc->add(reset ? 2 : 1);
}

}  // namespace sph
