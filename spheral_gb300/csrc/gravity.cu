// Octree gravity of libsphgpu: the TreeGravity build and walk
// (src/Gravity/TreeGravity.cc:362-480, 819-932; TreeGravityInline.hh:38-165)
// as a linear octree over Morton-sorted nodes.
//
// The reference inserts nodes one at a time into per-level hash maps: a cell
// is created holding a single node and split when a second node arrives,
// down to level 20 where nodes accumulate in one leaf.  The resulting tree
// does not depend on the insertion order: the cell (l, key) exists when it
// holds a node and its parent holds at least two (or l == 0); it is a leaf
// when it holds one node or l == 20.  Here every node gets the reference's
// level-20 integer coordinates (same floating-point expression), the nodes
// are sorted by the 60-bit Morton key of those coordinates, and the cells are
// read off the sorted keys:
//
//   cpl(k)  = deepest level at which sorted nodes k-1 and k share a cell
//             (-1 for k = 0 and k = n);
//   the cells that start at node k are the levels cpl(k)+1 .. leaf(k),
//   leaf(k) = min(20, max(cpl(k), cpl(k+1)) + 1).
//
// Listing those chains in node order gives the cells in depth-first
// pre-order; each cell stores the index of the first cell after its subtree
// (`skip`), so the walk needs no stack.  Monopoles (mass, centre of mass) are
// summed bottom-up, level by level.
//
// Walk.  The reference walks level by level per node and, per cell, applies
// the far-field monopole when r^2 > cellsize^2 / theta^2 + |xcm - centre|^2,
// sums the leaf's nodes directly when the cell is a leaf, and descends
// otherwise (TreeGravity.cc:845-905).  The per-node set of far cells and
// opened leaves does not depend on the visiting order, so here the 32 nodes
// of a warp (neighbours in Morton order) walk the pre-order cell array
// together: a lane that applies a cell (far or leaf) skips that cell's
// subtree; the warp descends into a cell while any lane still needs it open.
// (In the FP64 walk a warp walks for 8 nodes and queues the interactions.)
// Forces and potentials are evaluated in FP64; so is the decision wherever FP32
// could take it differently, with the reference's expression (no fused
// multiply-add).  Summation order is pre-order, split over the lanes of a node,
// instead of level order.
//
// Mixed precision (the mixed-mode package).  GB300's FP64 pipe is thin, so
// the mixed walk evaluates each interaction in FP32 on double-float
// (hi + lo) coordinates -- the separation (hi_c - hi_i) + (lo_c - lo_i)
// carries FP32 relative precision at any distance -- and sums the terms with
// compensated (Kahan) FP32 accumulators that leave the kernel as the FP64
// value s - c.
//
// Decisions.  Both walks compare an FP32 r^2 with FP32 thresholds and retake the
// decision in FP64 with the reference's expression inside a guard band, so the
// set of far cells and opened leaves is the reference's.  The double-float
// coordinates count from the corner of the bounding box: they are exact to
// 2^-49 of its length L wherever the system lies, a separation to 2^-46 L, and
// the band is twice that in r and 4e-6 in r^2 for the FP32 roundings.
#include "kernels.cuh"
#include "packed32.cuh"
#include "recip64.cuh"
#include "sort.cuh"
#include "../../include/sphgpu.h"

#include <cfloat>
#include <cstdio>
#include <cstring>
#include <string>

namespace sph {

namespace {

constexpr int kMaxLevel = 20;   // num1dbits - 1 (TreeGravity.hh: num1dbits = 21)
constexpr int kThreads = 256;

inline int blocksFor(long n, int t) { return (int)((n + t - 1) / t); }

// 64 bytes: one cell read by a whole warp is two 32-byte sectors.
struct __align__(32) TreeCell {
  double x, y, z, M;   // centre of mass and mass (Mglobal on one process)
  double r2cc;         // |xcm - geometric centre|^2 (rcm2cc2)
  double spare;
  int skip;            // first pre-order index after this cell's subtree
  int start;           // first node (tree order)
  int count;           // nodes in the cell
  int lvl;             // level | leaf << 8
};
static_assert(sizeof(TreeCell) == 64, "TreeCell layout");

struct __align__(32) Sums4 {
  double x, y, z, w;   // sums of m x, m y, m z and m
};

// Node in tree order: position and mass.
struct __align__(32) TreeNode {
  double x, y, z, m;
};

__device__ __forceinline__ TreeNode loadNode(const TreeNode* __restrict__ p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return TreeNode{a.x, a.y, b.x, b.y};
}

// What a walk reads of a cell it visits: the double-float centre of mass (from
// the box corner) in pairs for the packed operations, the mass, and the decision
// thresholds.  With r2 the FP32 squared separation, r2 > hi: the cell's monopole applies (a far
// cell, or a one-node leaf, whose monopole is its node); r2 < lo: it does not
// (an internal cell is opened, a one-node leaf is the node itself); between
// them FP64 decides.
struct __align__(16) TreeCell32 {
  float xh, yh, xl, yl;
  float zh, zl, hi, lo;
  float M;
  int skip, start, cnt;   // cnt: nodes of a leaf, 0 for an internal cell
};
static_assert(sizeof(TreeCell32) == 48, "TreeCell32 layout");

struct __align__(32) TreeNode32 {
  float xh, yh, zh, m;
  float xl, yl, zl, pad;
};

__device__ __forceinline__ void splitDF(double x, float& h, float& l) {
  h = (float)x;
  l = (float)(x - (double)h);
}

struct GBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t b) {
    if (b <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    const cudaError_t e = cudaMalloc(&p, b);
    if (e == cudaSuccess) bytes = b;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T> T* as() const { return static_cast<T*>(p); }
};

__device__ __forceinline__ uint64_t spread3(uint64_t v) {
  // 20-bit integer -> every third bit of a 60-bit word.
  v &= 0xFFFFFull;
  v = (v | (v << 32)) & 0x001F00000000FFFFull;
  v = (v | (v << 16)) & 0x001F0000FF0000FFull;
  v = (v | (v << 8)) & 0x100F00F00F00F00Full;
  v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

__device__ __forceinline__ uint64_t compact3(uint64_t v) {
  v &= 0x1249249249249249ull;
  v = (v | (v >> 2)) & 0x10C30C30C30C30C3ull;
  v = (v | (v >> 4)) & 0x100F00F00F00F00Full;
  v = (v | (v >> 8)) & 0x001F0000FF0000FFull;
  v = (v | (v >> 16)) & 0x001F00000000FFFFull;
  v = (v | (v >> 32)) & 0xFFFFFull;
  return v;
}

// TreeGravity::buildCellKey at the deepest level: min(ncell-1, (x - xmin) /
// boxLength * ncell) truncated, ncell = 2^20.
__device__ __forceinline__ uint64_t cellCoord(double x, double xmin, double L) {
  const double u = __dmul_rn(__ddiv_rn(__dsub_rn(x, xmin), L), 1048576.0);
  const uint64_t c = (uint64_t)u;
  return c < 1048575ull ? c : 1048575ull;
}

//------------------------------------------------------------------------------
// Bounding box (TreeGravity::initialize: xmin, xmax, boxLength).
//------------------------------------------------------------------------------
__global__ void boxPartialKernel(Fields F, long n, double* __restrict__ part) {
  __shared__ double sm[6][kThreads / 32];
  double v[6] = {DBL_MAX, DBL_MAX, DBL_MAX, DBL_MAX, DBL_MAX, DBL_MAX};   // min x,y,z, -max x,y,z
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double x = F.f[F_X][i], y = F.f[F_Y][i], z = F.f[F_Z][i];
    v[0] = fmin(v[0], x); v[1] = fmin(v[1], y); v[2] = fmin(v[2], z);
    v[3] = fmin(v[3], -x); v[4] = fmin(v[4], -y); v[5] = fmin(v[5], -z);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = fmin(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if (lane == 0) sm[k][warp] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = DBL_MAX;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = fmin(r, sm[threadIdx.x][w]);
    part[blockIdx.x * 6 + threadIdx.x] = r;
  }
}

// box = {xmin, ymin, zmin, boxLength, boxLength^2, -, -, -};
// also resets the dt-vote slot and the per-level opening thresholds.
__global__ void boxFinalKernel(const double* __restrict__ part, int nb, double opening, double* __restrict__ box,
                               double* __restrict__ thr, unsigned long long* __restrict__ dtBits) {
  __shared__ double v[6];
  __shared__ double sL2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;   // a warp per component
  if (warp < 6) {
    double r = DBL_MAX;
    for (int b = lane; b < nb; b += 32) r = fmin(r, part[b * 6 + warp]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = fmin(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (lane == 0) v[warp] = r;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double xmin = v[0], ymin = v[1], zmin = v[2];
    const double xmax = -v[3], ymax = -v[4], zmax = -v[5];
    // boxLength = max(xmax - xmin, max(ymax - ymin, zmax - zmin))
    const double L = fmax(__dsub_rn(xmax, xmin), fmax(__dsub_rn(ymax, ymin), __dsub_rn(zmax, zmin)));
    sL2 = __dmul_rn(L, L);
    box[0] = xmin; box[1] = ymin; box[2] = zmin; box[3] = L; box[4] = sL2;
    *dtBits = __double_as_longlong(DBL_MAX);
  }
  __syncthreads();
  if (threadIdx.x <= kMaxLevel) {
    // cellsize2 / opening2 with cellsize2 = boxLength2 / 2^(2 level)
    const double cs2 = __ddiv_rn(sL2, (double)(1ull << (2 * threadIdx.x)));
    thr[threadIdx.x] = __ddiv_rn(cs2, __dmul_rn(opening, opening));
  }
}

//------------------------------------------------------------------------------
// Morton keys of the level-20 cell coordinates (60 bits).
//------------------------------------------------------------------------------
__global__ void treeKeyKernel(Fields F, long n, const double* __restrict__ box, uint64_t* __restrict__ key64,
                              int* __restrict__ vals) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double L = box[3];
  uint64_t key = 0;
  if (L > 0.0) {
    const uint64_t ix = cellCoord(F.f[F_X][i], box[0], L);
    const uint64_t iy = cellCoord(F.f[F_Y][i], box[1], L);
    const uint64_t iz = cellCoord(F.f[F_Z][i], box[2], L);
    key = spread3(ix) | (spread3(iy) << 1) | (spread3(iz) << 2);
  }
  key64[i] = key;
  vals[i] = (int)i;
}

// Tree-ordered node data.  Indices of a sort that gave up waiting stay in
// range; the evaluation then fails on the sort's flag.
__global__ void treeNodesKernel(Fields F, const int* __restrict__ vals, long n, const double* __restrict__ box,
                                TreeNode* __restrict__ tpos, TreeNode32* __restrict__ tpos32) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int i = (int)min((unsigned)vals[k], (unsigned)(n - 1));
  const double x = F.f[F_X][i], y = F.f[F_Y][i], z = F.f[F_Z][i], m = F.f[F_MASS][i];
  tpos[k] = TreeNode{x, y, z, m};
  if (tpos32) {
    TreeNode32 t;
    splitDF(x - box[0], t.xh, t.xl);
    splitDF(y - box[1], t.yh, t.yl);
    splitDF(z - box[2], t.zh, t.zl);
    t.m = (float)m;
    t.pad = 0.0f;
    tpos32[k] = t;
  }
}

__device__ __forceinline__ int sharedLevels(const uint64_t* __restrict__ skey, long n, long k) {
  if (k <= 0 || k >= n) return -1;
  const uint64_t x = skey[k] ^ skey[k - 1];
  if (x == 0) return kMaxLevel;
  const int b = 63 - __clzll((long long)x);
  return kMaxLevel - 1 - b / 3;
}

__device__ __forceinline__ int leafLevel(int c0, int c1) {
  const int m = (c0 > c1 ? c0 : c1) + 1;
  return m < kMaxLevel ? m : kMaxLevel;
}

__global__ void chainCountKernel(const uint64_t* __restrict__ skey, long n, int* __restrict__ nc) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c0 = sharedLevels(skey, n, k), c1 = sharedLevels(skey, n, k + 1);
  nc[k] = leafLevel(c0, c1) - c0;
}

// First node after k whose level-l cell differs from k's (sorted keys).
__device__ __forceinline__ long cellEnd(const uint64_t* __restrict__ skey, long n, long k, int l) {
  const int sh = 3 * (kMaxLevel - l);
  const uint64_t p = skey[k] >> sh;
  long lo = k + 1, hi = n;
  while (lo < hi) {
    const long mid = (lo + hi) >> 1;
    if ((skey[mid] >> sh) == p) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void cellBuildKernel(const uint64_t* __restrict__ skey, long n, const long long* __restrict__ off,
                                long long numCells, TreeCell* __restrict__ cells) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c0 = sharedLevels(skey, n, k), c1 = sharedLevels(skey, n, k + 1);
  const int lf = leafLevel(c0, c1);
  const long long base = off[k];
  for (int l = c0 + 1; l <= lf; ++l) {
    const long e = (l == lf && l < kMaxLevel) ? k + 1 : cellEnd(skey, n, k, l);
    TreeCell c;
    c.x = c.y = c.z = c.M = c.r2cc = c.spare = 0.0;
    c.skip = (int)(e < n ? off[e] : numCells);
    c.start = (int)k;
    c.count = (int)(e - k);
    c.lvl = l | ((l == lf) ? 256 : 0);
    cells[base + (l - c0 - 1)] = c;
  }
}

// Parent and number of daughters of every cell.
__global__ void linkKernel(const TreeCell* __restrict__ cells, long long numCells, int* __restrict__ parent,
                           int* __restrict__ pending) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= numCells) return;
  if (c == 0) parent[0] = -1;
  if (cells[c].lvl >> 8) return;
  const int end = cells[c].skip;
  int m = 0;
  for (int ch = (int)c + 1; ch < end; ch = cells[ch].skip) { parent[ch] = (int)c; ++m; }
  pending[c] = m;
}

// The guard band of the FP32 r^2 around a squared distance d2, in a box of
// length L: r^2 above hi is above d2, below lo below it.  Values near underflow
// are left to FP64.
__device__ __forceinline__ void guardBand(float d2, float L, float& hi, float& lo) {
  constexpr float kBand = 4.0e-6f, kTiny = 1.0e-30f, kAbs = 2.842171e-14f;   // 2^-45
  const float d = sqrtf(d2), up = d + kAbs * L, down = fmaxf(d - kAbs * L, 0.0f);
  hi = fmaxf((up * up) * (1.0f + kBand), kTiny);
  lo = (down * down) * (1.0f - kBand);
  if (!(lo > kTiny)) lo = -1.0f;
}
// The walks' thresholds (TreeCell32) from the squared opening distance and,
// for a one-node leaf, the separation limit 1e-10 eps^2 below which the node
// does not act.
__device__ __forceinline__ void setThresholds(TreeCell32& o, double open2, double soft2, float L) {
  guardBand((float)open2, L, o.hi, o.lo);
  if (o.cnt == 1) {
    float hi, lo;
    guardBand(1.0e-10f * (float)soft2, L, hi, lo);
    o.hi = fminf(o.hi, hi);
    o.lo = fminf(o.lo, lo);
  }
}

__device__ __forceinline__ void cell32(const TreeCell& cl, double thr, double soft2, const double* __restrict__ box,
                                       TreeCell32* __restrict__ out) {
  TreeCell32 o;
  splitDF(cl.x - box[0], o.xh, o.xl);
  splitDF(cl.y - box[1], o.yh, o.yl);
  splitDF(cl.z - box[2], o.zh, o.zl);
  o.M = (float)cl.M;
  o.skip = cl.skip;
  o.start = cl.start;
  o.cnt = (cl.lvl >> 8) ? cl.count : 0;
  setThresholds(o, __dadd_rn(thr, cl.r2cc), soft2, (float)box[3]);
  *out = o;
}

// Sums of m and m x of every cell, bottom-up in one launch: a thread per leaf
// sums its nodes and climbs; the last daughter to arrive at a cell sums its
// daughters in pre-order (so the sums do not depend on who arrives last).  Few
// lanes of a warp climb far, so only the additions are done here: with the
// divisions and opening distances it took 232 us at 222,119 cells, without them
// 67 us and cellFinalKernel 34 us.
__global__ void momentKernel(const TreeCell* __restrict__ cells, long long numCells,
                             const TreeNode* __restrict__ tpos, const int* __restrict__ parent,
                             int* __restrict__ pending, Sums4* __restrict__ sums) {
  const long long c0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c0 >= numCells) return;
  {
    const TreeCell& cl = cells[c0];
    if (!(cl.lvl >> 8)) return;
    double M = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
    for (int j = cl.start; j < cl.start + cl.count; ++j) {
      const TreeNode p = tpos[j];
      M += p.m; sx += p.m * p.x; sy += p.m * p.y; sz += p.m * p.z;
    }
    sums[c0] = Sums4{sx, sy, sz, M};
  }
  for (int c = parent[c0]; c >= 0; c = parent[c]) {
    __threadfence();
    if (atomicSub(&pending[c], 1) != 1) return;
    __threadfence();
    // the daughters' sums come from other threads: volatile reads pass L1
    const int end = cells[c].skip;
    double M = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
    for (int ch = c + 1; ch < end; ch = cells[ch].skip) {
      const volatile double* m = reinterpret_cast<const volatile double*>(sums + ch);
      sx += m[0]; sy += m[1]; sz += m[2]; M += m[3];
    }
    sums[c] = Sums4{sx, sy, sz, M};
  }
}

// Centres of mass, opening distances and the walks' copy.  A one-node leaf
// keeps the node's position exactly, as the reference's single-node cell does.
__global__ void cellFinalKernel(TreeCell* __restrict__ cells, long long numCells, const TreeNode* __restrict__ tpos,
                                const uint64_t* __restrict__ skey, const double* __restrict__ box,
                                const double* __restrict__ thrLevel, double soft2, const Sums4* __restrict__ sums,
                                TreeCell32* __restrict__ c32) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= numCells) return;
  TreeCell cl = cells[c];
  const int level = cl.lvl & 255;
  const Sums4 sm = sums[c];
  if ((cl.lvl >> 8) && cl.count == 1) {
    const TreeNode p = tpos[cl.start];
    cl.x = p.x; cl.y = p.y; cl.z = p.z; cl.M = p.m;
  } else {
    // correctly rounded: the centre decides which cells open
    cl.x = __ddiv_rn(sm.x, sm.w); cl.y = __ddiv_rn(sm.y, sm.w); cl.z = __ddiv_rn(sm.z, sm.w); cl.M = sm.w;
  }
  // Geometric centre: xmin + (ix + 0.5) * cellsize, cellsize = boxLength / 2^level.
  const uint64_t key = skey[cl.start];
  const int sh = kMaxLevel - level;
  const double cs = __dmul_rn(box[3], __hiloint2double((1023 - level) << 20, 0));
  const double cx = __dadd_rn(box[0], __dmul_rn((double)(compact3(key) >> sh) + 0.5, cs));
  const double cy = __dadd_rn(box[1], __dmul_rn((double)(compact3(key >> 1) >> sh) + 0.5, cs));
  const double cz = __dadd_rn(box[2], __dmul_rn((double)(compact3(key >> 2) >> sh) + 0.5, cs));
  const double dx = __dsub_rn(cl.x, cx), dy = __dsub_rn(cl.y, cy), dz = __dsub_rn(cl.z, cz);
  cl.r2cc = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  cells[c] = cl;
  cell32(cl, thrLevel[level], soft2, box, c32 + c);
}

//------------------------------------------------------------------------------
// Walk (TreeGravity::applyTreeForces, TreeGravity.cc:819-932).
//------------------------------------------------------------------------------
__device__ __forceinline__ void addMonopole(double M, double dx, double dy, double dz, double soft2, double& ax,
                                            double& ay, double& az, double& phi) {
  // nhat = unitVector(xji); rji2 += soft2; a += M/rji2 nhat; phi -= M/sqrt(rji2)
  const double r2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
  const double irs = dev::rsqrt64(r2 + soft2);
  const double m = M * irs;
  if (__double2hiint(r2) > 0x2b000000) {   // r > ~1e-50
    const double f = (m * irs) * dev::rsqrt64(r2);
    ax = __fma_rn(f, dx, ax); ay = __fma_rn(f, dy, ay); az = __fma_rn(f, dz, az);
  } else {
    ax = __fma_rn(m, irs, ax);   // the unit vector of a zero separation is (1, 0, 0)
  }
  phi -= m;
}

// A node in the walks' double-float form, negated so that separations are sums.
struct WalkNode {
  dev::f32x2 nxyh, nxyl, nz;
};
__device__ __forceinline__ WalkNode walkNode(double x, double y, double z) {
  float xh, yh, zh, xl, yl, zl;
  splitDF(x, xh, xl);
  splitDF(y, yh, yl);
  splitDF(z, zh, zl);
  return WalkNode{dev::pack2(-xh, -yh), dev::pack2(-xl, -yl), dev::pack2(-zh, -zl)};
}

struct WalkCell {
  ulonglong2 xy;   // (xh yh) (xl yl)
  ulonglong2 zt;   // (zh zl) (hi lo)
  int4 q;          // M skip start cnt
};
__device__ __forceinline__ WalkCell loadCell(const TreeCell32* __restrict__ c32, unsigned c) {
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(c32 + c);
  return WalkCell{__ldg(p), __ldg(p + 1), __ldg(reinterpret_cast<const int4*>(p + 2))};
}

// Separation (hi_c - hi_i) + (lo_c - lo_i) and its square.
__device__ __forceinline__ float separation(const WalkCell& q, const WalkNode& me, dev::f32x2& dxy, float& dz) {
  dxy = dev::add2(dev::add2(q.xy.x, me.nxyh), dev::add2(q.xy.y, me.nxyl));
  float zh, zl, dx, dy;
  dev::unpack2(dev::add2(q.zt.x, me.nz), zh, zl);
  dz = __fadd_rn(zh, zl);
  dev::unpack2(dxy, dx, dy);
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// The FP64 decision, the reference's expressions: does the cell's monopole
// apply (far, or a one-node leaf beyond the separation limit)?
__device__ __noinline__ bool applies64(const TreeCell* __restrict__ cells, unsigned c, double x, double y, double z,
                                       const double* thr, double soft2) {
  const TreeCell& cd = cells[c];
  const double ex = __dsub_rn(cd.x, x), ey = __dsub_rn(cd.y, y), ez = __dsub_rn(cd.z, z);
  const double q2 = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
  if (q2 > __dadd_rn(thr[cd.lvl & 255], cd.r2cc)) return true;
  return (cd.lvl >> 8) && cd.count == 1 && __ddiv_rn(q2, soft2) > 1.0e-10;
}

// FP64 walk.  GB300's FP64 unit takes a warp instruction every 16 cycles per
// SM, so what counts is the number of warp interactions of ~22 FP64 operations:
// the decisions take FP32 (TreeCell32), and a warp walks for 8 nodes, which
// queue the cells that apply in shared memory; all 32 lanes (4 per node) then
// work through the queues.  Of 32 nodes that walk in step only 12 apply a cell
// at a time; the queues bring that to 28.  They drain to half their length, so
// that short ones need not keep up.  30,011 nodes of the Evrard sphere: gravity
// 4764 -> 1881 us per step.
constexpr int kWalkLanes = 4, kWalkNodes = 32 / kWalkLanes, kQueue = 128;
__global__ void __launch_bounds__(128) treeWalkKernel(const TreeCell32* __restrict__ c32,
                                                     const TreeCell* __restrict__ cells, long long numCells,
                                                     const TreeNode* __restrict__ tpos, const int* __restrict__ vals,
                                                     long n, const double* __restrict__ thrLevel, double soft2,
                                                     double softening, double G, Fields F,
                                                     unsigned long long* __restrict__ dtBits,
                                                     double* __restrict__ energyPart,
                                                     const double* __restrict__ box) {
  __shared__ double thr[kMaxLevel + 1];
  __shared__ double esum[4];
  __shared__ double dmin[4];
  __shared__ unsigned queues[4][kWalkNodes][kQueue + kWalkLanes];   // the odd 4 spread the banks
  if (threadIdx.x <= kMaxLevel) thr[threadIdx.x] = thrLevel[threadIdx.x];
  __syncthreads();
  const long k = (blockIdx.x * (long)blockDim.x + threadIdx.x) / kWalkLanes;
  const int sub = threadIdx.x % kWalkLanes;
  const bool valid = k < n;
  double xi = 0, yi = 0, zi = 0, mi = 0;
  if (valid) {
    const TreeNode p = tpos[k];
    xi = p.x; yi = p.y; zi = p.z; mi = p.m;
  }
  const WalkNode me = walkNode(xi - box[0], yi - box[1], zi - box[2]);
  double ax = 0, ay = 0, az = 0, phi = 0;
  unsigned* queue = queues[threadIdx.x >> 5][(threadIdx.x & 31) / kWalkLanes];
  unsigned head = 0, tail = 0;
  auto drain = [&](unsigned keep) {
    __syncwarp();
    while (__any_sync(0xffffffffu, tail - head > keep)) {
      const unsigned e = head + sub;
      if (e < tail) {
        const double2* dp = reinterpret_cast<const double2*>(cells + queue[e % kQueue]);
        const double2 qa = __ldg(dp), qb = __ldg(dp + 1);
        addMonopole(qb.y, qa.x - xi, qa.y - yi, qb.x - zi, soft2, ax, ay, az, phi);
      }
      head = min(head + kWalkLanes, tail);
    }
    __syncwarp();
  };
  // until: this lane ignores cells below this pre-order index
  unsigned until = valid ? 0u : 0xFFFFFFFFu;
  unsigned c = 1;   // the walk starts at the root's daughters
  const unsigned nc = (unsigned)numCells;
  if (__all_sync(0xffffffffu, !valid)) c = nc;
  while (c < nc) {
    const WalkCell q = loadCell(c32, c);
    const unsigned skip = (unsigned)q.q.y;
    bool descend = false;
    if (c >= until) {
      dev::f32x2 dxy;
      float dz, hi, lo;
      const float r2 = separation(q, me, dxy, dz);
      dev::unpack2(q.zt.y, hi, lo);
      bool apply = r2 > hi;
      if (!apply && !(r2 < lo)) apply = applies64(cells, c, xi, yi, zi, thr, soft2);
      descend = !apply && q.q.w == 0;
      if (!descend) until = skip;
      if (apply) {
        if (sub == 0) queue[tail % kQueue] = c;
        ++tail;
      } else if (q.q.w > 1) {   // nodes that share a deepest cell
        const double lim = 1.0e-10 * soft2;
        for (int j = q.q.z + sub; j < q.q.z + q.q.w; j += kWalkLanes) {
          const TreeNode p = loadNode(tpos + j);
          const double ex = __dsub_rn(p.x, xi), ey = __dsub_rn(p.y, yi), ez = __dsub_rn(p.z, zi);
          // s2 / soft2 > 1e-10, the division only near the limit
          const double s2 = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
          bool use = s2 > lim * 1.001;
          if (!use && s2 >= lim * 0.999) use = __ddiv_rn(s2, soft2) > 1.0e-10;
          if (use) addMonopole(p.m, ex, ey, ez, soft2, ax, ay, az, phi);
        }
      }
    }
    if (__any_sync(0xffffffffu, tail - head == kQueue)) drain(kQueue / 2);
    // the lanes that passed over c left it by its skip, the others lie beyond
    c = __any_sync(0xffffffffu, descend) ? c + 1 : skip;
  }
  drain(0);
#pragma unroll
  for (int o = kWalkLanes / 2; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
    az += __shfl_xor_sync(0xffffffffu, az, o);
    phi += __shfl_xor_sync(0xffffffffu, phi, o);
  }
  // Outputs: a, phi times G; dt vote sqrt(softening / |a|) before G.
  double vote = DBL_MAX, e = 0.0;
  if (valid && sub == 0) {
    const int i = vals[k];
    F.f[F_GRAV_X][i] = G * ax;
    F.f[F_GRAV_Y][i] = G * ay;
    F.f[F_GRAV_Z][i] = G * az;
    const double pot = G * phi;
    F.f[F_POT][i] = pot;
    const double amag = sqrt(ax * ax + ay * ay + az * az);
    if (amag > 0.0) vote = sqrt(softening / amag);
    e = 0.5 * mi * pot;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vote = fmin(vote, __shfl_xor_sync(0xffffffffu, vote, o));
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if (lane == 0) { dmin[warp] = vote; esum[warp] = e; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = dmin[0], s = esum[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { v = fmin(v, dmin[w]); s += esum[w]; }
    energyPart[blockIdx.x] = s;
    atomicMin(dtBits, (unsigned long long)__double_as_longlong(v));   // positive doubles order as integers
  }
}

// Compensated (Kahan) FP32 sums of (a_x, a_y) and (a_z, phi): the sum and the
// negated compensation, y = x + nc, t = s + y, nc = y - (t - s).
struct Acc32 {
  dev::f32x2 xy, zp, nxy, nzp;
};
__device__ __forceinline__ void kahan2(dev::f32x2& s, dev::f32x2& nc, dev::f32x2 x) {
  const dev::f32x2 kMinus = 0xBF800000BF800000ull;   // (-1, -1)
  const dev::f32x2 y = dev::add2(x, nc), t = dev::add2(s, y);
  nc = dev::add2(y, dev::fma2(t, kMinus, s));
  s = t;
}
// 1 / sqrt of a normal number.
__device__ __forceinline__ float rsqrtNormal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Monopole term: a += M/(r^2+eps^2) rhat, phi -= M/sqrt(r^2+eps^2); r2 > 1e-30.
__device__ __forceinline__ void addMonopole32(float M, dev::f32x2 dxy, float dz, float r2, float soft2, Acc32& a) {
  const float irs = rsqrtNormal(r2 + soft2);
  const float m = M * irs;
  const float f = (m * irs) * rsqrtNormal(r2);
  kahan2(a.xy, a.nxy, dev::mul2(dxy, dev::pack2(f, f)));
  kahan2(a.zp, a.nzp, dev::pack2(f * dz, -m));
}
// The same for any r2: the unit vector of a zero separation is (1, 0, 0).
__device__ __forceinline__ void addMonopole32Any(float M, dev::f32x2 dxy, float dz, float r2, float soft2, Acc32& a) {
  float dx, dy;
  dev::unpack2(dxy, dx, dy);
  const float irs = rsqrtf(r2 + soft2);
  const float m = M * irs, f0 = m * irs;
  const bool apart = r2 > 1.0e-30f;
  const float f = apart ? f0 * rsqrtf(r2) : f0;
  kahan2(a.xy, a.nxy, dev::pack2(f * (apart ? dx : 1.0f), f * dy));
  kahan2(a.zp, a.nzp, dev::pack2(f * dz, -m));
}

// Mixed walk: 32 nodes in step.  Bound by issue slots (~1900 visits per warp at
// 150,001 nodes) and the latency of the next cell: the thresholds, the one-node
// leaves and the next cell's index come with the cell, the separations and
// compensated sums are packed pairs; ~50 instructions per visit.  150,001 nodes:
// 905 us.  Loading both cells that may come next ahead of the decision took 89
// registers and 1173 us.
__global__ void __launch_bounds__(128) treeWalkMixedKernel(
    const TreeCell32* __restrict__ c32, const TreeCell* __restrict__ cells, long long numCells,
    const TreeNode32* __restrict__ t32, const TreeNode* __restrict__ tpos, const int* __restrict__ vals, long n,
    const double* __restrict__ thrLevel, double soft2d, double softening, double G, Fields F,
    unsigned long long* __restrict__ dtBits, double* __restrict__ energyPart, const double* __restrict__ box) {
  __shared__ double thr[kMaxLevel + 1];
  __shared__ double esum[4];
  __shared__ double dmin[4];
  if (threadIdx.x <= kMaxLevel) thr[threadIdx.x] = thrLevel[threadIdx.x];
  __syncthreads();
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const bool valid = k < n;
  double xd = 0, yd = 0, zd = 0, mi = 0;
  if (valid) {
    const TreeNode p = tpos[k];
    xd = p.x; yd = p.y; zd = p.z; mi = p.m;
  }
  const WalkNode me = walkNode(xd - box[0], yd - box[1], zd - box[2]);
  const float soft2 = (float)soft2d, boxLength = (float)box[3];
  Acc32 acc{0ull, 0ull, 0ull, 0ull};
  unsigned until = valid ? 0u : 0xFFFFFFFFu;
  unsigned c = 1;
  const unsigned nc = (unsigned)numCells;
  if (__all_sync(0xffffffffu, !valid)) c = nc;
  while (c < nc) {
    const WalkCell q = loadCell(c32, c);
    const unsigned skip = (unsigned)q.q.y;
    bool descend = false;
    if (c >= until) {
      const float M = __int_as_float(q.q.x);
      dev::f32x2 dxy;
      float dz, hi, lo;
      const float r2 = separation(q, me, dxy, dz);
      dev::unpack2(q.zt.y, hi, lo);
      if (r2 > hi) {
        addMonopole32(M, dxy, dz, r2, soft2, acc);
        until = skip;
      } else if (!(r2 < lo) && applies64(cells, c, xd, yd, zd, thr, soft2d)) {
        addMonopole32Any(M, dxy, dz, r2, soft2, acc);
        until = skip;
      } else {
        descend = q.q.w == 0;
        if (!descend) until = skip;
        if (q.q.w > 1) {   // nodes that share a deepest cell
          float limHi, limLo;
          guardBand(1.0e-10f * soft2, boxLength, limHi, limLo);
          for (int j = q.q.z; j < q.q.z + q.q.w; ++j) {
            const TreeNode32 p = t32[j];
            WalkCell w;
            w.xy = make_ulonglong2(dev::pack2(p.xh, p.yh), dev::pack2(p.xl, p.yl));
            w.zt.x = dev::pack2(p.zh, p.zl);
            dev::f32x2 exy;
            float ez;
            const float q2 = separation(w, me, exy, ez);
            bool use;
            if (q2 > limHi) use = true;
            else if (q2 < limLo) use = false;
            else {   // the reference's r2 / soft2 > 1e-10 in FP64
              const TreeNode pd = tpos[j];
              const double fx = __dsub_rn(pd.x, xd), fy = __dsub_rn(pd.y, yd), fz = __dsub_rn(pd.z, zd);
              const double w2 = __dadd_rn(__dadd_rn(__dmul_rn(fx, fx), __dmul_rn(fy, fy)), __dmul_rn(fz, fz));
              use = __ddiv_rn(w2, soft2d) > 1.0e-10;
            }
            if (use) addMonopole32Any(p.m, exy, ez, q2, soft2, acc);
          }
        }
      }
    }
    // the lanes that passed over c left it by its skip, the others lie beyond
    c = __any_sync(0xffffffffu, descend) ? c + 1 : skip;
  }
  double vote = DBL_MAX, e = 0.0;
  if (valid) {
    float sx, sy, sz, sp, cx, cy, cz, cp;
    dev::unpack2(acc.xy, sx, sy);
    dev::unpack2(acc.zp, sz, sp);
    dev::unpack2(acc.nxy, cx, cy);
    dev::unpack2(acc.nzp, cz, cp);
    const double ax = (double)sx + (double)cx, ay = (double)sy + (double)cy;
    const double az = (double)sz + (double)cz, phi = (double)sp + (double)cp;
    const int i = vals[k];
    F.f[F_GRAV_X][i] = G * ax;
    F.f[F_GRAV_Y][i] = G * ay;
    F.f[F_GRAV_Z][i] = G * az;
    const double pot = G * phi;
    F.f[F_POT][i] = pot;
    const double amag = sqrt(ax * ax + ay * ay + az * az);
    if (amag > 0.0) vote = sqrt(softening / amag);
    e = 0.5 * mi * pot;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vote = fmin(vote, __shfl_xor_sync(0xffffffffu, vote, o));
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if (lane == 0) { dmin[warp] = vote; esum[warp] = e; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = dmin[0], sm = esum[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { v = fmin(v, dmin[w]); sm += esum[w]; }
    energyPart[blockIdx.x] = sm;
    atomicMin(dtBits, (unsigned long long)__double_as_longlong(v));
  }
}

__global__ void walkFinalKernel(const double* __restrict__ energyPart, int nb, const unsigned long long* dtBits,
                                double G, double* __restrict__ out) {
  __shared__ double sm[32];
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += energyPart[b];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sm[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm[w];
    out[0] = __longlong_as_double((long long)*dtBits) / sqrt(G);   // dtMinAcc
    out[1] = t;                                                      // extraEnergy
  }
}

__global__ void zeroGravityKernel(Fields F, long n, double G, double* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i == 0) { out[0] = DBL_MAX / sqrt(G); out[1] = 0.0; }
  if (i >= n) return;
  F.f[F_GRAV_X][i] = F.f[F_GRAV_Y][i] = F.f[F_GRAV_Z][i] = 0.0;
  F.f[F_POT][i] = 0.0;
}

}  // namespace

struct GravityWork {
  GBuf part, box, thr, dtBits, key64, timeout, vals, vals2, sortWs, skey, tpos, nc, off, scanWs, total, cells, mx,
      energy, tpos32, cells32, parent, pending;
  long long* hTotal = nullptr;
};

GravityWork* gravityCreate() {
  GravityWork* w = new GravityWork();
  if (cudaMallocHost(&w->hTotal, 2 * sizeof(long long)) != cudaSuccess) w->hTotal = nullptr;
  return w;
}

void gravityDestroy(GravityWork* w) {
  if (!w) return;
  GBuf* all[] = {&w->part, &w->box, &w->thr, &w->dtBits, &w->key64, &w->timeout, &w->vals, &w->vals2,
                 &w->sortWs, &w->skey, &w->tpos, &w->nc, &w->off, &w->scanWs, &w->total, &w->cells, &w->mx,
                 &w->energy, &w->tpos32, &w->cells32, &w->parent, &w->pending};
  for (GBuf* b : all) b->release();
  if (w->hTotal) cudaFreeHost(w->hTotal);
  delete w;
}

int gravityEvaluate(GravityWork* w, Fields F, long n, double G, double softening, double opening, bool mixed,
                    double* dOut, cudaStream_t s, LaunchCounter* lc, char* err, int errlen) {
#define GCHK(expr)                                                                     \
  do {                                                                                 \
    const cudaError_t e_ = (expr);                                                     \
    if (e_ != cudaSuccess) {                                                           \
      std::snprintf(err, errlen, "%s: %s", #expr, cudaGetErrorString(e_));             \
      return SPHGPU_E_CUDA;                                                            \
    }                                                                                  \
  } while (0)
  if (!w || !w->hTotal) { std::snprintf(err, errlen, "gravity work space missing"); return SPHGPU_E_STATE; }
  if (!(softening > 0.0) || !(opening > 0.0) || !(G > 0.0)) {
    std::snprintf(err, errlen, "TreeGravity needs G, softening and opening > 0");
    return SPHGPU_E_ARG;
  }
  if (n <= 1) {
    zeroGravityKernel<<<blocksFor(n > 0 ? n : 1, kThreads), kThreads, 0, s>>>(F, n, G, dOut);
    lc->add(1);
    GCHK(cudaGetLastError());
    return SPHGPU_OK;
  }
  const int nbBox = 304;
  GCHK(w->part.ensure(nbBox * 6 * sizeof(double)));
  GCHK(w->box.ensure(8 * sizeof(double)));
  GCHK(w->thr.ensure(32 * sizeof(double)));
  GCHK(w->dtBits.ensure(sizeof(unsigned long long)));
  GCHK(w->key64.ensure(n * sizeof(uint64_t)));
  GCHK(w->skey.ensure(n * sizeof(uint64_t)));
  GCHK(w->timeout.ensure(sizeof(int)));
  GCHK(w->vals.ensure(n * sizeof(int)));
  GCHK(w->vals2.ensure(n * sizeof(int)));
  GCHK(w->sortWs.ensure(radixSortWorkspaceBytes(n)));
  GCHK(w->tpos.ensure(n * sizeof(TreeNode)));
  if (mixed) GCHK(w->tpos32.ensure(n * sizeof(TreeNode32)));
  GCHK(w->nc.ensure(n * sizeof(int)));
  GCHK(w->off.ensure((n + 1) * sizeof(long long)));
  GCHK(w->scanWs.ensure(scanWorkspaceBytes(n)));
  GCHK(w->total.ensure(sizeof(long long)));
  const int nbWalk = blocksFor(mixed ? n : kWalkLanes * n, 128);
  GCHK(w->energy.ensure(nbWalk * sizeof(double)));

  boxPartialKernel<<<nbBox, kThreads, 0, s>>>(F, n, w->part.as<double>());
  boxFinalKernel<<<1, 192, 0, s>>>(w->part.as<double>(), nbBox, opening, w->box.as<double>(), w->thr.as<double>(),
                                 w->dtBits.as<unsigned long long>());
  treeKeyKernel<<<blocksFor(n, kThreads), kThreads, 0, s>>>(F, n, w->box.as<double>(), w->key64.as<uint64_t>(),
                                                           w->vals.as<int>());
  lc->add(3);
  uint64_t* skey = w->key64.as<uint64_t>();
  uint64_t* skeyAlt = w->skey.as<uint64_t>();
  int* vals = w->vals.as<int>();
  int* valsAlt = w->vals2.as<int>();
  GCHK(cudaMemsetAsync(w->timeout.p, 0, sizeof(int), s));
  radixSortPairs(skey, vals, skeyAlt, valsAlt, n, 3 * kMaxLevel, w->sortWs.p, w->timeout.as<int>(), false, s, lc);
  treeNodesKernel<<<blocksFor(n, kThreads), kThreads, 0, s>>>(F, vals, n, w->box.as<double>(), w->tpos.as<TreeNode>(),
                                                             mixed ? w->tpos32.as<TreeNode32>() : nullptr);
  chainCountKernel<<<blocksFor(n, kThreads), kThreads, 0, s>>>(skey, n, w->nc.as<int>());
  lc->add(2);
  scanExclusive<int>(w->nc.as<int>(), w->off.as<long long>(), n, w->scanWs.p, w->total.as<long long>(), s, lc);
  GCHK(cudaMemcpyAsync(w->hTotal, w->total.p, sizeof(long long), cudaMemcpyDeviceToHost, s));
  GCHK(cudaMemcpyAsync(w->hTotal + 1, w->timeout.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  GCHK(cudaStreamSynchronize(s));
  const long long numCells = *w->hTotal;
  if (*reinterpret_cast<const int*>(w->hTotal + 1)) {
    std::snprintf(err, errlen, "a wait inside the octree sort ran out");
    return SPHGPU_E_TIMEOUT;
  }
  if (numCells <= 0 || numCells > 0x7FFFFFFFll) {
    std::snprintf(err, errlen, "octree cell count %lld out of range", numCells);
    return SPHGPU_E_OVERFLOW;
  }
  GCHK(w->cells.ensure(numCells * sizeof(TreeCell)));
  GCHK(w->mx.ensure(numCells * sizeof(Sums4)));
  TreeCell* cells = w->cells.as<TreeCell>();
  cellBuildKernel<<<blocksFor(n, kThreads), kThreads, 0, s>>>(skey, n, w->off.as<long long>(),
                                                             numCells, cells);
  lc->add(1);
  const int nbCells = (int)((numCells + kThreads - 1) / kThreads);
  GCHK(w->cells32.ensure(numCells * sizeof(TreeCell32)));
  GCHK(w->parent.ensure(numCells * sizeof(int)));
  GCHK(w->pending.ensure(numCells * sizeof(int)));
  linkKernel<<<nbCells, kThreads, 0, s>>>(cells, numCells, w->parent.as<int>(), w->pending.as<int>());
  momentKernel<<<nbCells, kThreads, 0, s>>>(cells, numCells, w->tpos.as<TreeNode>(), w->parent.as<int>(),
                                            w->pending.as<int>(), w->mx.as<Sums4>());
  cellFinalKernel<<<nbCells, kThreads, 0, s>>>(cells, numCells, w->tpos.as<TreeNode>(), skey, w->box.as<double>(),
                                               w->thr.as<double>(), softening * softening, w->mx.as<Sums4>(),
                                               w->cells32.as<TreeCell32>());
  lc->add(3);
  if (mixed)
    treeWalkMixedKernel<<<nbWalk, 128, 0, s>>>(w->cells32.as<TreeCell32>(), cells, numCells,
                                               w->tpos32.as<TreeNode32>(), w->tpos.as<TreeNode>(), vals, n,
                                               w->thr.as<double>(), softening * softening, softening, G, F,
                                               w->dtBits.as<unsigned long long>(), w->energy.as<double>(),
                                               w->box.as<double>());
  else
    treeWalkKernel<<<nbWalk, 128, 0, s>>>(w->cells32.as<TreeCell32>(), cells, numCells, w->tpos.as<TreeNode>(), vals,
                                          n, w->thr.as<double>(), softening * softening, softening, G, F,
                                          w->dtBits.as<unsigned long long>(), w->energy.as<double>(),
                                          w->box.as<double>());
  walkFinalKernel<<<1, 256, 0, s>>>(w->energy.as<double>(), nbWalk, w->dtBits.as<unsigned long long>(), G, dOut);
  lc->add(2);
  GCHK(cudaGetLastError());
  return SPHGPU_OK;
#undef GCHK
}

}  // namespace sph
