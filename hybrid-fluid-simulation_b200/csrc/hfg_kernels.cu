// hfg_kernels.cu -- sm_100a kernels of the grid half of the hybrid fluid step.
//
// Every kernel restates one stage of the reference engine's CUDA code
// (junwei-jiang/Hybrid-Fluid-Simulation, MPhysics/) in a B200-first shape:
// grid-stride launches sized to the SM count, fused stages, uint8 cell
// markers, FP64 deterministic reductions and device-resident solver scalars.
// The reference line each kernel follows is cited beside it.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <map>
#include <mutex>

#include "hfg_kernels.h"

namespace hfg {

namespace {
int g_numSMs = 0;
constexpr int kThreads = 256;

inline int gridFor(long long n, int threads = kThreads, int perSM = 16) {
  long long b = (n + threads - 1) / threads;
  long long cap = (long long)numSMs() * perSM;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// Grid-stride loop over [0, n).
#define HFG_FOR(i, n) \
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

// The same loop with a 32-bit index that does not step past n: n may lie within
// a step of 2^32.
#define HFG_FOR_U(i, n)                                                                                       \
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x, i##Step = gridDim.x * blockDim.x, i##On = i < (n); \
       i##On; i##On = (n)-i > i##Step, i += i##Step)

// The same loop with an index of type I.  The particle kernels take I = int
// when 3 n and n + the grid's thread count stay below 2^31, which saves the
// 64-bit index and address arithmetic of every iteration.
#define HFG_FOR_T(I, i, n) \
  for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < (I)(n); i += (I)gridDim.x * blockDim.x)


// True when a particle kernel over n particles may index in 32 bits.
inline bool index32(long long n) { return 3 * n + (long long)numSMs() * 16 * kThreads < (1ll << 31); }

__device__ inline void cellCoord(long long c, const Dim3i& r, int& x, int& y, int& z) {
  x = (int)(c % r.x);
  long long t = c / r.x;
  y = (int)(t % r.y);
  z = (int)(t / r.y);
}

}  // namespace

cudaError_t clusterSize(const void* kernel, int threads, size_t smem, int* size) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> known;  // by kernel and device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find({kernel, dev});
  if (it != known.end()) {
    *size = it->second;
    return cudaSuccess;
  }
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess && smem > 0)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  *size = 0;
  for (int n : {16, 8}) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = n;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) {
      *size = n;
      break;
    }
    cudaGetLastError();
  }
  known[{kernel, dev}] = *size;
  return cudaSuccess;
}

int numSMs() {
  if (g_numSMs == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&g_numSMs, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || g_numSMs <= 0)
      g_numSMs = 148;
  }
  return g_numSMs;
}


// ===========================================================================
// Boundaries and classification
// ===========================================================================

// Boundary.cpp:129-146 + BoundaryTool.cu:3-26,85-113: re-sample every solid
// SDF at (cell centre + translation) and keep the first solid that contains
// the cell.  solidIdx = 0 outside every solid, i+1 inside solid i.
__global__ void kSolidClassify(Geom g, BoundarySet b, uint8_t* __restrict__ solidIdx, float* const* curSDF) {
  long long n = g.r.size();
  HFG_FOR(c, n) {
    int x, y, z;
    cellCoord(c, g.r, x, y, z);
    float cx = __fadd_rn(__fadd_rn(g.ox, 0.5f * g.hx), __fmul_rn(g.hx, (float)x));
    float cy = __fadd_rn(__fadd_rn(g.oy, 0.5f * g.hy), __fmul_rn(g.hy, (float)y));
    float cz = __fadd_rn(__fadd_rn(g.oz, 0.5f * g.hz), __fmul_rn(g.hz, (float)z));
    uint8_t idx = 0;
    for (int i = 0; i < b.n; ++i) {
      float v = trilerp(b.sdf[i], g, __fadd_rn(cx, b.tx[i]), __fadd_rn(cy, b.ty[i]), __fadd_rn(cz, b.tz[i]));
      if (curSDF && curSDF[i]) curSDF[i][c] = v;
      if (idx == 0 && v < 0.f) idx = (uint8_t)(i + 1);
    }
    solidIdx[c] = idx;
  }
}

cudaError_t launchSolidClassify(const Geom& g, const BoundarySet& b, uint8_t* solidIdx, float* const* curSDF,
                                cudaStream_t s) {
  kSolidClassify<<<gridFor(g.r.size()), kThreads, 0, s>>>(g, b, solidIdx, curSDF);
  return cudaGetLastError();
}

__global__ void kSolidFromSDF(long long n, const float* __restrict__ sdf, uint8_t* __restrict__ idx) {
  HFG_FOR(c, n) idx[c] = sdf[c] < 0.f ? 1 : 0;
}
__global__ void kAnalyticSdf(Geom g, int type, double p0, double p1, double p2, double p3, double p4, double p5,
                             float* __restrict__ sdf) {
  const Dim3i R = g.r;
  HFG_FOR(c, R.size()) {
    int x, y, z;
    cellCoord(c, R, x, y, z);
    const double P[3] = {(double)g.ox + (x + 0.5) * (double)g.hx, (double)g.oy + (y + 0.5) * (double)g.hy,
                         (double)g.oz + (z + 0.5) * (double)g.hz};
    double d;
    if (type == 0) {
      const double lo[3] = {(double)g.ox + g.hx, (double)g.oy + g.hy, (double)g.oz + g.hz};
      const double hi[3] = {(double)g.ox + (R.x - 1) * (double)g.hx, (double)g.oy + (R.y - 1) * (double)g.hy,
                            (double)g.oz + (R.z - 1) * (double)g.hz};
      double in = 1e300, outsq = 0.0;
      for (int a = 0; a < 3; ++a) {
        double da = fmin(P[a] - lo[a], hi[a] - P[a]);
        in = fmin(in, da);
        if (da < 0.0) outsq += da * da;
      }
      d = in >= 0.0 ? in : -sqrt(outsq);
    } else if (type == 1) {
      const double dx = P[0] - p0, dy = P[1] - p1, dz = P[2] - p2;
      d = sqrt(dx * dx + dy * dy + dz * dz) - p3;
    } else {
      const double c3[3] = {p0, p1, p2}, s3[3] = {p3, p4, p5};
      double outsq = 0.0, mx = -1e300;
      for (int a = 0; a < 3; ++a) {
        double q = fabs(P[a] - c3[a]) - 0.5 * s3[a];
        if (q > 0.0) outsq += q * q;
        mx = fmax(mx, q);
      }
      d = sqrt(outsq) + fmin(mx, 0.0);
    }
    sdf[c] = (float)d;
  }
}
cudaError_t launchAnalyticSdf(const Geom& g, int type, const double* p, float* sdf, cudaStream_t s) {
  kAnalyticSdf<<<gridFor(g.r.size()), kThreads, 0, s>>>(g, type, p[0], p[1], p[2], p[3], p[4], p[5], sdf);
  return cudaGetLastError();
}

cudaError_t launchSolidFromSDF(long long n, const float* solidSDF, uint8_t* solidIdx, cudaStream_t s) {
  kSolidFromSDF<<<gridFor(n), kThreads, 0, s>>>(n, solidSDF, solidIdx);
  return cudaGetLastError();
}

// The reference's "total boundary SDF" (BoundaryTool.cu:3-26): 0 everywhere
// with no solid, else -(first solid index) inside and UNKNOWN outside.
__global__ void kTotalSolidSDF(long long n, int nb, const uint8_t* __restrict__ idx, float* __restrict__ out) {
  HFG_FOR(c, n) {
    uint8_t i = idx[c];
    out[c] = nb == 0 ? 0.f : (i ? -(float)i : kUnknown);
  }
}
cudaError_t launchTotalSolidSDF(long long n, int nb, const uint8_t* solidIdx, float* out, cudaStream_t s) {
  kTotalSolidSDF<<<gridFor(n), kThreads, 0, s>>>(n, nb, solidIdx, out);
  return cudaGetLastError();
}

__global__ void kSolidVelField(Geom g, SolidVelTable t, FaceField out) {
  for (int a = 0; a < 3; ++a) {
    Dim3i fr = g.r;
    if (a == 0) fr.x += 1;
    if (a == 1) fr.y += 1;
    if (a == 2) fr.z += 1;
    long long n = fr.size();
    HFG_FOR(f, n) {
      int x, y, z;
      cellCoord(f, fr, x, y, z);
      int hx = x, hy = y, hz = z, lx = x, ly = y, lz = z;
      if (a == 0) lx = x - 1;
      if (a == 1) ly = y - 1;
      if (a == 2) lz = z - 1;
      bool hiIn = (a == 0 ? hx < g.r.x : (a == 1 ? hy < g.r.y : hz < g.r.z));
      bool loIn = (a == 0 ? lx >= 0 : (a == 1 ? ly >= 0 : lz >= 0));
      uint8_t hi = hiIn ? t.solidIdx[((long long)hz * g.r.y + hy) * g.r.x + hx] : 0;
      uint8_t lo = loIn ? t.solidIdx[((long long)lz * g.r.y + ly) * g.r.x + lx] : 0;
      out.c[a][f] = solidFaceVel(t, lo, hi, a);
    }
  }
}
cudaError_t launchSolidVelField(const Geom& g, const SolidVelTable& t, FaceField out, cudaStream_t s) {
  kSolidVelField<<<gridFor(g.r.size()), kThreads, 0, s>>>(g, t, out);
  return cudaGetLastError();
}

__global__ void kMarkersInit(long long n, const uint8_t* __restrict__ idx, uint8_t* __restrict__ mk) {
  HFG_FOR(c, n) mk[c] = idx[c] ? kSolid : kAir;
}
cudaError_t launchMarkersInit(long long n, const uint8_t* solidIdx, uint8_t* markers, cudaStream_t s) {
  kMarkersInit<<<gridFor(n), kThreads, 0, s>>>(n, solidIdx, markers);
  return cudaGetLastError();
}

// EulerParticlesTool.cu:27-77: a non-solid cell holding at least one particle
// (truncating binning) is fluid.  Only "count > 0" matters, so the count is
// replaced by an idempotent store; cells stay bit-exact.
__global__ void kMarkersFromParticles(Geom g, const float* __restrict__ pos, long long P, uint8_t* __restrict__ mk) {
  HFG_FOR(p, P) {
    long long c = binCell(g, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2]);
    if (mk[c] == kAir) mk[c] = kFluid;
  }
}
cudaError_t launchMarkersFromParticles(const Geom& g, const float* pos, long long P, uint8_t* markers, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  kMarkersFromParticles<<<gridFor(P), kThreads, 0, s>>>(g, pos, P, markers);
  return cudaGetLastError();
}

// statisticalFluidDensity (EulerParticlesTool.cu:27-46) with warp-aggregated
// integer atomics: lanes that hit the same cell add once.
__global__ void kBinCounts(Geom g, const float* __restrict__ pos, long long P, unsigned int* __restrict__ counts) {
  for (long long base = (long long)blockIdx.x * blockDim.x; base < P; base += (long long)gridDim.x * blockDim.x) {
    long long p = base + threadIdx.x;
    bool valid = p < P;
    unsigned int active = __ballot_sync(0xffffffffu, valid);
    if (!valid) continue;
    long long c = binCell(g, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2]);
    unsigned int peers = __match_any_sync(active, c);
    int leader = __ffs(peers) - 1;
    if ((int)(threadIdx.x & 31) == leader) atomicAdd(counts + c, (unsigned int)__popc(peers));
  }
}
cudaError_t launchBinCounts(const Geom& g, const float* pos, long long P, unsigned int* counts, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  kBinCounts<<<gridFor(P), kThreads, 0, s>>>(g, pos, P, counts);
  return cudaGetLastError();
}

// EulerSolverTool.cu:30-56 buildFluidMarkers (SDF form)
__global__ void kMarkersFromSDF(long long n, const uint8_t* __restrict__ idx, const float* __restrict__ fsdf,
                                uint8_t* __restrict__ mk) {
  HFG_FOR(c, n) mk[c] = idx[c] ? kSolid : (fsdf[c] < 0.f ? kFluid : kAir);
}
cudaError_t launchMarkersFromSDF(long long n, const uint8_t* solidIdx, const float* fluidSDF, uint8_t* markers,
                                 cudaStream_t s) {
  kMarkersFromSDF<<<gridFor(n), kThreads, 0, s>>>(n, solidIdx, fluidSDF, markers);
  return cudaGetLastError();
}

// EulerSolverTool.cu:581-608 generateFluidDomainFromBBox (strict inequalities,
// every cell rewritten).
__global__ void kFluidDomainFromBBox(Geom g, float mnx, float mny, float mnz, float mxx, float mxy, float mxz,
                                     float* __restrict__ out) {
  HFG_FOR(c, g.r.size()) {
    int x, y, z;
    cellCoord(c, g.r, x, y, z);
    float cx = __fadd_rn(__fadd_rn(g.ox, 0.5f * g.hx), __fmul_rn(g.hx, (float)x));
    float cy = __fadd_rn(__fadd_rn(g.oy, 0.5f * g.hy), __fmul_rn(g.hy, (float)y));
    float cz = __fadd_rn(__fadd_rn(g.oz, 0.5f * g.hz), __fmul_rn(g.hz, (float)z));
    bool in = cx > mnx && cy > mny && cz > mnz && cx < mxx && cy < mxy && cz < mxz;
    out[c] = in ? -500.f : 500.f;  // FluidDomainValue (Common.h:245)
  }
}
cudaError_t launchFluidDomainFromBBox(const Geom& g, const float mn[3], const float mx[3], float* out, cudaStream_t s) {
  kFluidDomainFromBBox<<<gridFor(g.r.size()), kThreads, 0, s>>>(g, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], out);
  return cudaGetLastError();
}

// EulerSolverTool.cu:229-322 applyPressureGradient: faces with a fluid side
// and a solid side take the solid velocity, fluid-fluid/fluid-air faces get
// -dt/(rho h) * dp, all others and the far boundary faces become UNKNOWN.
template <class TP>
__global__ void kGradient(Geom g, float gx, float gy, float gz, const uint8_t* __restrict__ mk,
                          const TP* __restrict__ p, FaceField v, ConstFaceField svArr, SolidVelTable svTab) {
  const Dim3i R = g.r;
  const Dim3i rx{R.x + 1, R.y, R.z}, ry{R.x, R.y + 1, R.z}, rz{R.x, R.y, R.z + 1};
  HFG_FOR(c, R.size()) {
    int x, y, z;
    cellCoord(c, R, x, y, z);
    long long sy = R.x, sz = (long long)R.x * R.y;
    long long cl = x > 0 ? c - 1 : c, cd = y > 0 ? c - sy : c, cb = z > 0 ? c - sz : c;
    const long long px = cgPitch(R.x);
    const long long pc = ((long long)z * R.y + y) * px + x;  // pressure is pitched
    const long long po[3] = {x > 0 ? pc - 1 : pc, y > 0 ? pc - px : pc, z > 0 ? pc - px * R.y : pc};
    uint8_t mc = mk[c];
    long long fx = ((long long)z * rx.y + y) * rx.x + x;
    long long fy = ((long long)z * ry.y + y) * ry.x + x;
    long long fz = ((long long)z * rz.y + y) * rz.x + x;
    const long long fo[3] = {fx, fy, fz};
    const long long co[3] = {cl, cd, cb};
    const float gs[3] = {gx, gy, gz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      uint8_t ml = mk[co[a]];
      float* vv = v.c[a];
      if (ml == kFluid || mc == kFluid) {
        if (ml == kSolid || mc == kSolid) {
          float s;
          if (svArr.c[0]) s = svArr.c[a][fo[a]];
          else s = solidFaceVel(svTab, co[a] == c ? 0 : svTab.solidIdx[co[a]], svTab.solidIdx[c], a);
          vv[fo[a]] = s;
        } else {
          const float dp = sizeof(TP) == 8 ? __double2float_rn(__dsub_rn((double)p[pc], (double)p[po[a]]))
                                           : __fsub_rn((float)p[pc], (float)p[po[a]]);
          vv[fo[a]] = __fsub_rn(vv[fo[a]], __fmul_rn(gs[a], dp));
        }
      } else {
        vv[fo[a]] = kUnknown;
      }
    }
    if (x == R.x - 1) v.c[0][fx + 1] = kUnknown;
    if (y == R.y - 1) v.c[1][fy + ry.x] = kUnknown;
    if (z == R.z - 1) v.c[2][fz + (long long)rz.x * rz.y] = kUnknown;
  }
}
cudaError_t launchGradient(const Geom& g, float gx, float gy, float gz, const uint8_t* markers, const void* p,
                           bool pDouble, FaceField v, ConstFaceField svArr, const SolidVelTable& svTab,
                           cudaStream_t s) {
  if (pDouble)
    kGradient<double><<<gridFor(g.r.size()), kThreads, 0, s>>>(g, gx, gy, gz, markers, (const double*)p, v, svArr,
                                                               svTab);
  else
    kGradient<float><<<gridFor(g.r.size()), kThreads, 0, s>>>(g, gx, gy, gz, markers, (const float*)p, v, svArr,
                                                              svTab);
  return cudaGetLastError();
}

// ===========================================================================
// Extrapolation (EulerSolverTool.cu:450-557, :904-969)
// ===========================================================================
//
// The reference grows UNKNOWN entries layer by layer from the known ones with
// 6-neighbour clamp-to-edge steps, 999 layers at most, then sets every layer-d
// entry to the mean of its neighbours of smaller layer.  Without obstacles the
// layer of an entry equals its L1 distance to the nearest known entry, so the
// layers come from a separable exact L1 distance transform (three 1-D min-plus
// passes); entries are then bucketed by layer and each layer is one launch.

constexpr uint16_t kFar = 0xFFFF;

__device__ inline uint16_t satInc(uint16_t a) { return a >= kFar - 1 ? kFar : (uint16_t)(a + 1); }

// The grids of one extrapolation: up to three (one per blockIdx.y), an unused
// one with no entries.
struct ExtrapGrids {
  Dim3i r[3];
  float* v[3];
  unsigned off[3];  // first entry of each grid in the joint numbering
};

// First distances and the 1-D pass along x: one warp per row, 32 entries at a
// time.  The forward sweep f[i] = min(d[i], f[i-1] + 1), d = 0 at known
// entries, is a warp prefix-min of d[j] - j plus the carry from the previous
// chunk; the backward sweep mirrors it.
__global__ void kDistRows(const __grid_constant__ ExtrapGrids g, uint16_t* __restrict__ dist) {
  constexpr int BIG = 1 << 20;
  const Dim3i r = g.r[blockIdx.y];
  const float* __restrict__ val = g.v[blockIdx.y];
  uint16_t* __restrict__ d = dist + g.off[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)r.y * r.z, nw = (gridDim.x * blockDim.x) >> 5;
  for (long long row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += nw) {
    uint16_t* q = d + (size_t)row * r.x;
    const float* p = val + (size_t)row * r.x;
    int carry = BIG;
    for (int s0 = 0; s0 < r.x; s0 += 32) {
      int i = s0 + lane;
      int v = i < r.x && p[i] != kUnknown ? 0 : BIG;
      int a = v - lane;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, a, o);
        if (lane >= o) a = min(a, t);
      }
      int f = min(a + lane, carry + lane + 1);
      if (i < r.x) q[i] = (uint16_t)min(f, (int)kFar);
      carry = __shfl_sync(0xffffffffu, f, 31);
    }
    carry = BIG;
    int last = ((r.x - 1) / 32) * 32;
    for (int s0 = last; s0 >= 0; s0 -= 32) {
      int i = s0 + lane;
      int v = i < r.x ? (q[i] == kFar ? BIG : (int)q[i]) : BIG;
      int b = v + lane;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_down_sync(0xffffffffu, b, o);
        if (lane + o < 32) b = min(b, t);
      }
      int gm = min(b - lane, carry + (32 - lane));
      if (i < r.x) q[i] = (uint16_t)min(gm, (int)kFar);
      carry = __shfl_sync(0xffffffffu, gm, 0);
    }
  }
}

// 1-D pass along y or z: threads walk columns, coalesced across x.  Columns
// in batches of B: the B loads of a batch are in flight together, then the
// batch is relaxed in order.  Both axes of three
// 256^3 grids, with batches of 16 and one launch per axis: 283 -> 179 us.
__global__ void kDistCols(const __grid_constant__ ExtrapGrids g, int axis, uint16_t* __restrict__ dist) {
  const Dim3i r = g.r[blockIdx.y];
  uint16_t* __restrict__ d = dist + g.off[blockIdx.y];
  const unsigned nx = (unsigned)r.x, plane = nx * (unsigned)r.y;
  const unsigned stride = axis == 1 ? nx : plane;
  const int len = axis == 1 ? r.y : r.z;
  const unsigned lines = axis == 1 ? nx * (unsigned)r.z : plane;
  HFG_FOR_U(l, lines) {
    unsigned base = l;
    if (axis == 1) {
      const unsigned z = l / nx;
      base = z * plane + (l - z * nx);
    }
    constexpr int B = 16;
    uint16_t* col = d + base;
    uint16_t prev = kFar;
    for (int i0 = 0; i0 < len; i0 += B) {
      uint16_t v[B];
#pragma unroll
      for (int k = 0; k < B; ++k) v[k] = i0 + k < len ? col[(unsigned)(i0 + k) * stride] : kFar;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        if (i0 + k < len) {
          const uint16_t cand = satInc(prev);
          if (cand < v[k]) {
            v[k] = cand;
            col[(unsigned)(i0 + k) * stride] = cand;
          }
          prev = v[k];
        }
      }
    }
    prev = kFar;
    for (int i0 = len - 1; i0 >= 0; i0 -= B) {
      uint16_t v[B];
#pragma unroll
      for (int k = 0; k < B; ++k) v[k] = i0 - k >= 0 ? col[(unsigned)(i0 - k) * stride] : kFar;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        if (i0 - k >= 0) {
          const uint16_t cand = satInc(prev);
          if (cand < v[k]) {
            v[k] = cand;
            col[(unsigned)(i0 - k) * stride] = cand;
          }
          prev = v[k];
        }
      }
    }
  }
}

// Histogram of layers 1..nums-1 (layers >= nums stay UNKNOWN).
__global__ void kDistHist(long long n, const uint16_t* __restrict__ d, int nums, unsigned int* __restrict__ hist) {
  __shared__ unsigned int sh[kMaxLayers + 1];
  for (int i = threadIdx.x; i <= kMaxLayers; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  HFG_FOR(i, n) {
    const unsigned v = d[i];
    if (v >= 1 && (int)v < nums) atomicAdd(&sh[v], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= kMaxLayers; i += blockDim.x)
    if (sh[i]) atomicAdd(hist + i, sh[i]);
}

// Exclusive scan of at most 1024 counts by one block.
__global__ void __launch_bounds__(1024) kExclusiveScanSmall(const unsigned int* __restrict__ hist,
                                                            unsigned int* __restrict__ off,
                                                            unsigned int* __restrict__ cursor, int n) {
  __shared__ unsigned int tot[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned mine = t < n ? hist[t] : 0u;
  unsigned inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) tot[w] = inc;
  __syncthreads();
  if (w == 0) {
    unsigned v = tot[lane], vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += u;
    }
    tot[lane] = vi - v;
  }
  __syncthreads();
  const unsigned ex = tot[w] + inc - mine;
  if (t < n) {
    off[t] = ex;
    cursor[t] = ex;
    if (t == n - 1) off[n] = ex + mine;
  }
}

// Neighbours of entry i of grid r in the order left, right, down, up, back,
// front, clamped to the grid (an edge entry is its own neighbour there).
__device__ __forceinline__ void extrapNeighbours(const Dim3i& r, unsigned i, unsigned nb[6]) {
  const unsigned nx = (unsigned)r.x, ny = (unsigned)r.y, t = i / nx;
  const int x = (int)(i - t * nx), y = (int)(t % ny), z = (int)(t / ny);
  const unsigned plane = nx * ny;
  nb[0] = x > 0 ? i - 1 : i;
  nb[1] = x + 1 < r.x ? i + 1 : i;
  nb[2] = y > 0 ? i - nx : i;
  nb[3] = y + 1 < r.y ? i + nx : i;
  nb[4] = z > 0 ? i - plane : i;
  nb[5] = z + 1 < r.z ? i + plane : i;
}

// Bucket the entries by layer: a block counts its chunk per layer in shared
// memory (the count before an entry is its rank), reserves one global range
// per (block, layer) and writes the entries to their slots.  Only the bins
// between the chunk's lowest and highest layer are touched: neighbouring
// entries have neighbouring layers.  Each entry also gets the mask of its
// neighbours in earlier layers, so that the layer pass reads no distances
// (reading them there instead cost a layer 1.5 us: three loads deep).
// Against clearing and reserving all 1001 bins with a second shared atomic
// per entry: 555 -> 489 us (256^3, three grids).
constexpr int kScatterThreads = 512, kScatterPer = 8, kScatterChunk = kScatterThreads * kScatterPer;
__global__ void __launch_bounds__(kScatterThreads)
    kDistScatter(const __grid_constant__ ExtrapGrids g, const uint16_t* __restrict__ dist, int nums, unsigned int* __restrict__ cursor,
                 unsigned int* __restrict__ list, uint8_t* __restrict__ mask) {
  const Dim3i r = g.r[blockIdx.y];
  const unsigned base = g.off[blockIdx.y], n = (unsigned)r.size();
  const uint16_t* __restrict__ d = dist + base;
  __shared__ unsigned int cnt[kMaxLayers + 1], start[kMaxLayers + 1];
  __shared__ int lo, hi;
  for (unsigned long long at = blockIdx.x * kScatterChunk; at < n; at += gridDim.x * kScatterChunk) {
    const unsigned c0 = (unsigned)at;
    if (threadIdx.x == 0) {
      lo = kMaxLayers + 1;
      hi = 0;
    }
    unsigned v[kScatterPer], rank[kScatterPer];
    unsigned mn = kMaxLayers + 1, mx = 0;
#pragma unroll
    for (int k = 0; k < kScatterPer; ++k) {
      const unsigned o = k * kScatterThreads + threadIdx.x;
      const unsigned dv = o < n - c0 ? d[c0 + o] : 0u;
      v[k] = dv >= 1 && (int)dv < nums ? dv : 0u;
      if (v[k]) {
        mn = min(mn, dv);
        mx = max(mx, dv);
      }
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && mx > 0) {
      atomicMin(&lo, (int)mn);
      atomicMax(&hi, (int)mx);
    }
    __syncthreads();
    const int l0 = lo, l1 = hi;
    for (int i = l0 + threadIdx.x; i <= l1; i += kScatterThreads) cnt[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kScatterPer; ++k)
      if (v[k]) rank[k] = atomicAdd(&cnt[v[k]], 1u);
    __syncthreads();
    for (int i = l0 + threadIdx.x; i <= l1; i += kScatterThreads) start[i] = cnt[i] ? atomicAdd(cursor + i, cnt[i]) : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kScatterPer; ++k) {
      if (v[k]) {
        const unsigned i = c0 + k * kScatterThreads + threadIdx.x;
        unsigned nb[6];
        extrapNeighbours(r, i, nb);
        unsigned m = 0;
#pragma unroll
        for (int q = 0; q < 6; ++q) m |= (unsigned)(d[nb[q]] < v[k]) << q;
        const unsigned slot = start[v[k]] + rank[k];
        list[slot] = base + i;
        mask[slot] = (uint8_t)m;
      }
    }
  }
}

namespace {
ExtrapGrids extrapGrids(const Dim3i rc[3], float* const vals[3], const long long off[3]) {
  ExtrapGrids g;
  for (int a = 0; a < 3; ++a) {
    g.r[a] = rc[a];
    g.v[a] = vals[a];
    g.off[a] = (unsigned)off[a];
  }
  return g;
}
}  // namespace

cudaError_t launchExtrapDistance(const Dim3i rc[3], float* const vals[3], long long off[3], int nums,
                                 ExtrapScratch sc, cudaStream_t s) {
  if (nums > kMaxLayers) nums = kMaxLayers;
  const ExtrapGrids g = extrapGrids(rc, vals, off);
  long long rows = 1, colsY = 1, colsZ = 1, most = 1, total = 0;
  int grids = 0;
  for (int a = 0; a < 3; ++a) {
    if (rc[a].size() > 0) grids = a + 1;
    rows = std::max(rows, (long long)rc[a].y * rc[a].z * 32);
    colsY = std::max(colsY, (long long)rc[a].x * rc[a].z);
    colsZ = std::max(colsZ, (long long)rc[a].x * rc[a].y);
    most = std::max(most, rc[a].size());
    total += rc[a].size();
  }
  kDistRows<<<dim3(gridFor(rows), grids), kThreads, 0, s>>>(g, sc.dist);
  kDistCols<<<dim3(gridFor(colsY, 128), grids), 128, 0, s>>>(g, 1, sc.dist);
  kDistCols<<<dim3(gridFor(colsZ, 128), grids), 128, 0, s>>>(g, 2, sc.dist);
  cudaError_t e = cudaMemsetAsync(sc.hist, 0, sizeof(unsigned int) * kExtrapHistWords, s);
  if (e != cudaSuccess) return e;
  // every block adds its bins to the global ones: few blocks on small grids.  Four
  // an SM / sixteen, us a call of four layers: 48^3 92 / 98, 64^3 102 / 104, alike
  // from 80^3 to 160^3, 256^3 (51 M faces) 696 / 674
  kDistHist<<<gridFor(total, kThreads, total > 8000000 ? 16 : 4), kThreads, 0, s>>>(total, sc.dist, nums, sc.hist);
  kExclusiveScanSmall<<<1, 1024, 0, s>>>(sc.hist, sc.offsets, sc.cursor, kMaxLayers + 1);
  const int blocks =
      (int)std::min<long long>((most + kScatterChunk - 1) / kScatterChunk, (long long)numSMs() * 8);
  kDistScatter<<<dim3(blocks, grids), kScatterThreads, 0, s>>>(g, sc.dist, nums, sc.cursor, sc.list, sc.mask);
  return cudaGetLastError();
}

// One entry of layer d: mean of the neighbours with a smaller layer (mask m),
// summed in the fixed order left, right, down, up, back, front
// (extrapolatingData).
// The values of earlier layers were written by other blocks of the same
// launch, so they are read from L2 (ld.cg), never from a stale L1 line.
// 32-bit index arithmetic: every face grid holds fewer than 2^31 entries.
struct ExtrapEntry {
  float* v = nullptr;  // null: no entry
  unsigned i, nb[6], m;
};
__device__ __forceinline__ ExtrapEntry extrapFetch(const ExtrapGrids& g, const unsigned* __restrict__ list,
                                                   const uint8_t* __restrict__ mask, unsigned k, unsigned end) {
  ExtrapEntry e;
  if (k < end) {
    const unsigned id = __ldg(list + k);
    e.m = __ldg(mask + k);
    const int a = id >= g.off[2] ? 2 : (id >= g.off[1] ? 1 : 0);
    const Dim3i r = a == 2 ? g.r[2] : (a == 1 ? g.r[1] : g.r[0]);
    e.v = a == 2 ? g.v[2] : (a == 1 ? g.v[1] : g.v[0]);
    e.i = id - (a == 2 ? g.off[2] : (a == 1 ? g.off[1] : 0u));
    extrapNeighbours(r, e.i, e.nb);
  }
  return e;
}
__device__ __forceinline__ void extrapFill(const ExtrapEntry& e) {
  if (!e.v) return;
  float w[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) w[q] = (e.m >> q) & 1u ? __ldcg(e.v + e.nb[q]) : 0.f;
  float acc = 0.f, cnt = 0.f;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if ((e.m >> q) & 1u) {
      acc = __fadd_rn(acc, w[q]);
      cnt = __fadd_rn(cnt, 1.f);
    }
  }
  if (cnt != 0.f) acc = __fdiv_rn(acc, cnt);
  __stcg(e.v + e.i, acc);
}

// Block shape of the layer pass: 1024 threads, at most one block per SM, as few
// arrivals as possible at the barriers.
constexpr int kExtrapThreads = 1024;

// Layers 1 .. nums-1, persistent: a layer of some size is spread over the
// blocks; a run of smaller consecutive layers is filled by block 0 alone with
// block barriers between them.  Every block walks the same layer bounds
// (sc.offsets), so all meet at the same barriers.  A layer is bound by latency:
// its faces are one or a few to a thread, and each step is neighbour loads, a
// store and a barrier.  So a thread's first face of the next phase is fetched
// and decoded while the barrier is on its way, and the loads of the neighbours
// that count are in flight together.
// CLUSTER: the blocks are one thread block cluster and meet at its hardware
// barrier; otherwise they are a cooperative grid and meet through mailboxes.
// barWords: kExtrapError, kExtrapDepth, then the mailboxes.
template <bool CLUSTER>
__global__ void __launch_bounds__(kExtrapThreads, 1)
    kExtrapLayers(const __grid_constant__ ExtrapGrids g, const uint8_t* __restrict__ mask,
                  const unsigned int* __restrict__ list, const unsigned int* __restrict__ offsets, int nums,
                  unsigned* barWords) {
  // a layer of at most this many faces is filled by block 0
  constexpr unsigned kSmall = CLUSTER ? kExtrapThreads : kExtrapSmallLayer;
  __shared__ unsigned offS[kMaxLayers + 2];
  for (int i = threadIdx.x; i < kMaxLayers + 2; i += kExtrapThreads) offS[i] = __ldg(offsets + i);
  __syncthreads();
  unsigned* mail = barWords + kExtrapSlots;
  const unsigned nblk = gridDim.x, stride = nblk * kExtrapThreads;
  const unsigned gtid = blockIdx.x * kExtrapThreads + threadIdx.x;
  auto size = [&](int d) -> unsigned {  // faces of layer d, 0 past the last layer
    return d < nums && d <= kMaxLayers ? offS[d + 1] - offS[d] : 0u;
  };
  auto fetch = [&](int d, unsigned k) -> ExtrapEntry {  // k-th face of layer d
    return extrapFetch(g, list, mask, offS[d] + k, offS[d] + size(d));
  };
  // this thread's first face of a phase that starts at layer d
  auto firstOf = [&](int d) -> ExtrapEntry {
    if (size(d) == 0) return ExtrapEntry{};
    return fetch(d, size(d) > kSmall ? gtid : (blockIdx.x == 0 ? threadIdx.x : size(d)));
  };
  unsigned epoch = 0;
  int d = 1;
  ExtrapEntry e = firstOf(d);
  while (size(d) > 0) {
    if (size(d) > kSmall) {
      extrapFill(e);
      for (unsigned k = gtid + stride; k < size(d); k += stride) extrapFill(fetch(d, k));
      ++d;
    } else {
      int last = d;
      while (size(last + 1) > 0 && size(last + 1) <= kSmall) ++last;
      if (blockIdx.x == 0) {
        for (int l = d; l <= last; ++l) {
          extrapFill(e);
          for (unsigned k = threadIdx.x + kExtrapThreads; k < size(l); k += kExtrapThreads) extrapFill(fetch(l, k));
          if (l < last) e = fetch(l + 1, threadIdx.x);
          __syncthreads();
        }
      }
      d = last + 1;
    }
    if (size(d) == 0) break;
    if (CLUSTER) clusterArrive();
    else if (nblk > 1) gridArrive(mail, ++epoch, nblk);
    else __syncthreads();
    e = firstOf(d);
    if (CLUSTER) clusterWait();
    else if (nblk > 1 && !gridWait(mail, epoch, barWords + kExtrapError, nblk)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) barWords[kExtrapDepth] = (unsigned)(d - 1);
}

namespace {
std::atomic<int> g_extrapUsers{0};
}
void extrapUsers(int delta) { g_extrapUsers.fetch_add(delta); }

namespace {
std::mutex g_coopMu;
std::condition_variable g_coopFree;
struct Coop {
  int shared = 0;  // holders of the shared lease, and their blocks
  int blocks = 0;
  bool exclusive = false;
};
std::map<int, Coop> g_coop;  // by device
}  // namespace

CoopLease::CoopLease() : exclusive_(true) {
  cudaGetDevice(&dev_);
  std::lock_guard<std::mutex> lk(g_coopMu);
  Coop& c = g_coop[dev_];
  held_ = !c.exclusive && c.shared == 0;
  if (held_) c.exclusive = true;
}
// Up to twice the fair share where that many are free: the users are seldom all
// here at once.  A call on 256^3 (2.6 ms on the whole GPU) beside 31 idle scenes
// takes 9.2 ms, on the fair share alone 16.4; 32 threads that extrapolate 112^3
// at once 6.7 ms for all, on fair shares 8.8.
CoopLease::CoopLease(int want, int slots) : exclusive_(false), held_(true) {
  cudaGetDevice(&dev_);
  std::unique_lock<std::mutex> lk(g_coopMu);
  Coop& c = g_coop[dev_];
  int fair = 0;
  g_coopFree.wait(lk, [&] {
    fair = std::min(want, std::max(1, slots / std::max(1, g_extrapUsers.load())));
    return !c.exclusive && slots - c.blocks >= fair;
  });
  blocks_ = std::min({want, 2 * fair, slots - c.blocks});
  ++c.shared;
  c.blocks += blocks_;
}
CoopLease::~CoopLease() {
  if (!held_) return;
  {
    std::lock_guard<std::mutex> lk(g_coopMu);
    Coop& c = g_coop[dev_];
    if (exclusive_) {
      c.exclusive = false;
    } else {
      --c.shared;
      c.blocks -= blocks_;
    }
  }
  g_coopFree.notify_all();
}

// The layers' launch.  Grids of at most kExtrapClusterFaces faces: one cluster
// of 16 blocks (8 where the device has no 16), whose barrier and values stay
// within one GPC: a layer of 64^3 takes 3.0 us instead of 4.7; the L2 bandwidth
// of 16 SMs is what limits it on larger grids.  Those take a cooperative grid: about one
// block per 4096 faces, at most one per SM, and at most what its lease grants,
// so that the grids of concurrent scenes always fit on the GPU together.
// Whole calls in us, cluster / cooperative grid: 64^3 294 / 400, 96^3 (2.7 M
// faces) 553 / 581, 128^3 (6.3 M) 927 / 806, 256^3 5333 / 2612; hence the line.
constexpr long long kExtrapClusterFaces = 3000000;
cudaError_t extrapForm(const Dim3i rc[3], ExtrapForm* form) {
  const long long faces = rc[0].size() + rc[1].size() + rc[2].size();
  if (faces <= kExtrapClusterFaces) {
    int size = 0;
    const cudaError_t e = clusterSize((const void*)kExtrapLayers<true>, kExtrapThreads, 0, &size);
    if (e != cudaSuccess) return e;
    // small grids need fewer blocks than the cluster could have
    while (size > 1 && (long long)(size / 2) * kExtrapThreads * 16 >= faces) size /= 2;
    if (size > 0) {
      form->cluster = true;
      form->blocks = size;
      return cudaSuccess;
    }
  }
  static std::atomic<int> perSM{0};
  if (perSM.load() == 0) {
    int v = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kExtrapLayers<false>, kExtrapThreads, 0);
    if (e != cudaSuccess) return e;
    perSM.store(std::max(1, v));
  }
  form->cluster = false;
  form->slots = numSMs() * perSM.load();
  form->blocks =
      (int)std::max(1LL, std::min({(faces + 4095) / 4096, (long long)numSMs(), (long long)kExtrapMaxBlocks}));
  return cudaSuccess;
}
cudaError_t launchExtrapLayers(const Dim3i rc[3], float* const vals[3], const long long off[3], ExtrapScratch sc,
                               int nums, bool cluster, int blocks, cudaStream_t s, long long* launches) {
  if (nums <= 1) return cudaSuccess;
  ExtrapGrids g = extrapGrids(rc, vals, off);
  const uint8_t* mask = sc.mask;
  const unsigned int* list = sc.list;
  const unsigned int* offs = sc.offsets;
  unsigned* bar = extrapBarWords(sc);
  cudaError_t e;
  if (cluster) {
    e = launchCluster(kExtrapLayers<true>, blocks, kExtrapThreads, 0, s, g, mask, list, offs, nums, bar);
  } else {
    void* args[] = {&g, &mask, &list, &offs, &nums, &bar};
    e = cudaLaunchCooperativeKernel((const void*)kExtrapLayers<false>, dim3(blocks), dim3(kExtrapThreads), args, 0, s);
  }
  if (e == cudaSuccess && launches) ++*launches;
  return e;
}

// One warp copies `words` 32-bit words (small state read-backs into mapped
// host memory).
__global__ void kCopyWords(const unsigned* __restrict__ src, unsigned* __restrict__ dst, int words) {
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}
cudaError_t launchCopyWords(const unsigned* src, unsigned* dst, int words, cudaStream_t s) {
  kCopyWords<<<1, 32, 0, s>>>(src, dst, words);
  return cudaGetLastError();
}

// ===========================================================================
// Distance fields in cells (buildFluidSDF and the hybrid coupler's inside /
// outside fields below): the number of 6-neighbour steps from a set of seed
// cells, some cells closed to the walk.  The reference grows the field one
// step per sweep of the whole grid, up to 1000 of them.  Here the distances
// relax along whole lines: one pass each along x, y and z (a forward and a
// backward min(d, d_before + 1) sweep, stopping at closed cells) is a round.
// With no closed cell one round gives every distance (the separable L1
// transform); otherwise a cell at distance d is right after as many rounds as
// its shortest walk has straight pieces at most, and a round that changes
// nothing ends it: the passes are exact at their fixed point.  A few rounds
// replace a launch and a host read per distance step: density, the three
// distance fields and a field mix on 96^3 7.0 -> 0.36 ms.
// ===========================================================================
namespace {
constexpr double kSurf = 0.2;  // FluidSurfaceDensity (Common.h:244)
__device__ __forceinline__ float outsideValue(int d) { return (float)((double)d + (1.5 - kSurf)); }
__device__ __forceinline__ float insideValue(int d) { return d == 0 ? (float)(0.5 - kSurf) : (float)(-((double)d - (0.5 - kSurf))); }
constexpr int kStepsFar = 0x7fffff00, kStepsClosed = -1;
}  // namespace

// A pass of round `round` does nothing once an earlier round changed nothing.
__device__ __forceinline__ bool stepsDone(const unsigned* changed, int round) {
  return round > 0 && *(volatile const unsigned*)(changed + round - 1) == 0u;
}

// Records that a pass changed something: one store per block at most, since the
// stores of many threads to the one word queue up in L2: 128^3, a tenth of
// the cells closed at random, 1.85 -> 0.41 ms a call
__device__ __forceinline__ void markChanged(bool any, unsigned* flag) {
  if (__syncthreads_or(any) && flatTid() == 0 && *(volatile unsigned*)flag == 0u) *(volatile unsigned*)flag = 1u;
}

// Along x: one warp per row, 32 cells at a time; a sweep is a warp prefix-min
// of d - lane between closed cells, plus the carry of the chunk before.
__global__ void kStepsRows(Dim3i r, int* __restrict__ d, unsigned* changed, int round) {
  if (stepsDone(changed, round)) return;
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)r.y * r.z, nw = (gridDim.x * blockDim.x) >> 5;
  bool any = false;
  for (long long row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += nw) {
    int* q = d + (size_t)row * r.x;
#pragma unroll
    for (int back = 0; back < 2; ++back) {
      int carry = kStepsFar;
      for (int s0 = 0; s0 < r.x; s0 += 32) {
        const int j = s0 + lane, i = back ? r.x - 1 - j : j;
        const int v = j < r.x ? q[i] : kStepsClosed;
        const unsigned closed = __ballot_sync(0xffffffffu, v < 0);
        // the last closed lane up to this one (-1: none)
        const int wall = 31 - __clz((int)(closed & (0xffffffffu >> (31 - lane))));
        int a = v < 0 ? kStepsFar : v - lane;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, a, o);
          if (lane - o > wall) a = min(a, t);
        }
        int f = v < 0 ? kStepsFar : min(a + lane, kStepsFar);
        if (wall < 0) f = min(f, carry + lane + 1);
        if (v >= 0 && f < v) {
          q[i] = f;
          any = true;
        }
        carry = __shfl_sync(0xffffffffu, f, 31);
      }
      __syncwarp();
    }
  }
  markChanged(any, changed + round);
}

// Along y (axis 1) or z: one thread per line, coalesced across x, the loads of
// B cells in flight together.
__global__ void kStepsCols(Dim3i r, int axis, int* __restrict__ d, unsigned* changed, int round) {
  if (stepsDone(changed, round)) return;
  const size_t nx = (size_t)r.x, plane = nx * r.y, stride = axis == 1 ? nx : plane;
  const int len = axis == 1 ? r.y : r.z;
  const size_t lines = axis == 1 ? nx * r.z : plane;
  bool any = false;
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < lines; l += (size_t)gridDim.x * blockDim.x) {
    int* col = d + (axis == 1 ? (l / nx) * plane + l % nx : l);
    constexpr int B = 16;
#pragma unroll
    for (int back = 0; back < 2; ++back) {
      int prev = kStepsFar;
      for (int s0 = 0; s0 < len; s0 += B) {
        int v[B];
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int j = s0 + k;
          v[k] = j < len ? col[(size_t)(back ? len - 1 - j : j) * stride] : kStepsClosed;
        }
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int j = s0 + k;
          if (v[k] >= 0 && prev + 1 < v[k]) {
            v[k] = prev + 1;
            col[(size_t)(back ? len - 1 - j : j) * stride] = v[k];
            any = true;
          }
          prev = v[k] < 0 ? kStepsFar : v[k];
        }
      }
    }
  }
  markChanged(any, changed + round);
}

// The same distances level by level, on bits: a row of cells is ceil(nx / 32)
// words, with one bit a cell in the masks of the cells not yet reached and of
// the last level.  A level is then a dilation of an eighth of a byte a cell,
// 7-8 us at 256^3 where a pass
// over ints took 50.
struct StepBits {
  unsigned *open, *front[2];
  int words;  // of a row
};
namespace {
size_t stepBitsWords(const Dim3i& r) { return (size_t)((r.x + 31) / 32) * r.y * r.z; }
StepBits stepBits(const Dim3i& r, int* steps) {
  unsigned* p = reinterpret_cast<unsigned*>(steps + r.size());
  const size_t n = stepBitsWords(r);
  return StepBits{p, {p + n, p + 2 * n}, (r.x + 31) / 32};
}
}  // namespace
size_t sideSdfInts(const Dim3i& r) { return (size_t)r.size() + 3 * stepBitsWords(r); }

// seeds (distance 0) into front[0], the other cells that are not closed into open
__global__ void kStepsToBits(Dim3i r, const int* __restrict__ d, StepBits b) {
  const int lane = threadIdx.x & 31;
  const size_t n = (size_t)b.words * r.y * r.z, nw = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t w = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5; w < n; w += nw) {
    const size_t row = w / b.words;
    const int x = (int)(w - row * b.words) * 32 + lane;
    const int v = x < r.x ? d[row * r.x + x] : kStepsClosed;
    const unsigned seed = __ballot_sync(0xffffffffu, v == 0), open = __ballot_sync(0xffffffffu, v > 0);
    if (lane == 0) {
      b.front[0][w] = seed;
      b.open[w] = open;
    }
  }
}
// level k, from the bits of front[(k - 1) & 1] to front[k & 1]; a level without
// cells is the last, and the passes after it do nothing
__global__ void kStepsLevel(Dim3i r, int* __restrict__ d, StepBits b, unsigned* changed, int k, int slot) {
  if (stepsDone(changed, slot)) return;
  const unsigned* __restrict__ from = k & 1 ? b.front[0] : b.front[1];
  unsigned* __restrict__ to = k & 1 ? b.front[1] : b.front[0];
  const size_t plane = (size_t)b.words * r.y, n = plane * r.z;
  bool any = false;
  for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < n; w += (size_t)gridDim.x * blockDim.x) {
    const unsigned open = b.open[w];
    unsigned now = 0u;
    if (open) {
      const size_t row = w / b.words;
      const int i = (int)(w - row * b.words), z = (int)(row / r.y), y = (int)(row - (size_t)z * r.y);
      const unsigned c = from[w];
      const unsigned l = i > 0 ? from[w - 1] >> 31 : 0u, rt = i + 1 < b.words ? from[w + 1] << 31 : 0u;
      const unsigned dn = y > 0 ? from[w - b.words] : 0u, up = y + 1 < r.y ? from[w + b.words] : 0u;
      const unsigned be = z > 0 ? from[w - plane] : 0u, ab = z + 1 < r.z ? from[w + plane] : 0u;
      now = (c << 1 | l | c >> 1 | rt | dn | up | be | ab) & open;
      if (now) {
        b.open[w] = open & ~now;
        any = true;
        int* q = d + row * r.x + 32 * (size_t)i;
        for (unsigned m = now; m; m &= m - 1) q[__ffs((int)m) - 1] = k;
      }
    }
    to[w] = now;
  }
  markChanged(any, changed + slot);
}

namespace {
// The passes of rounds [0, rounds).
cudaError_t launchStepRounds(const Dim3i& r, int* d, unsigned* changed, int rounds, cudaStream_t s) {
  for (int k = 0; k < rounds; ++k) {
    kStepsRows<<<gridFor((long long)r.y * r.z * 32), kThreads, 0, s>>>(r, d, changed, k);
    kStepsCols<<<gridFor((long long)r.x * r.z, 64), 64, 0, s>>>(r, 1, d, changed, k);
    kStepsCols<<<gridFor((long long)r.x * r.y, 64), 64, 0, s>>>(r, 2, d, changed, k);
  }
  return cudaGetLastError();
}
// Levels [first, first + n), from the bits.
cudaError_t launchStepLevels(const Dim3i& r, int* d, const StepBits& b, unsigned* changed, int first, int n,
                             cudaStream_t s) {
  const int grid = gridFor((long long)stepBitsWords(r));
  for (int k = 0; k < n; ++k) kStepsLevel<<<grid, kThreads, 0, s>>>(r, d, b, changed, first + k, k);
  return cudaGetLastError();
}
}  // namespace

// Fluid SDF of the fluid-domain field (EulerSolverTool.cu:324-406, :760-785;
// GridFluidSolver.cpp:571-591).  The cells on both sides of the fluid surface
// are the seeds (0.5 - 0.2 inside, 1.5 - 0.2 outside); the field grows from
// them on its own side only, which needs no closed cells: the surface cell
// nearest to a cell lies on the cell's own side, and so does every shortest
// walk to it.
__global__ void kFluidSdfSeed(Dim3i r, const float* __restrict__ dom, int* __restrict__ d) {
  HFG_FOR(c, r.size()) {
    int x, y, z;
    cellCoord(c, r, x, y, z);
    const bool in = dom[c] < 0.f;
    bool mixed = false;
    const int dx[6] = {-1, 1, 0, 0, 0, 0}, dy[6] = {0, 0, -1, 1, 0, 0}, dz[6] = {0, 0, 0, 0, -1, 1};
#pragma unroll
    for (int k = 0; k < 6; ++k) mixed |= ((dom[linc(x + dx[k], y + dy[k], z + dz[k], r)] < 0.f) != in);
    d[c] = mixed ? 0 : kStepsFar;
  }
}
__global__ void kFluidSdfValue(long long n, const float* __restrict__ dom, const int* __restrict__ d, int layers,
                               float* __restrict__ sdf) {
  HFG_FOR(c, n) {
    const bool in = dom[c] < 0.f;
    const int k = d[c];
    const bool reached = k == 0 || k < layers;
    sdf[c] = in ? (reached ? insideValue(k) : -kUnknown) : (reached ? outsideValue(k) : kUnknown);
  }
}

// buildFluidDensity (EulerSolverTool.cu:408-448): 1 inside the fluid, the
// surface density 0.2 where a 6-neighbour (clamp-to-edge) is air, 0 outside
// the fluid or inside a solid.  A cell is air when neither the fluid domain
// nor the solid is negative there (isInsideAir, EulerMathTool.cu:344-348).
__global__ void kFluidDensity(Dim3i r, const float* __restrict__ dom, const float* __restrict__ solidSdf,
                              const uint8_t* __restrict__ solidIdx, float* __restrict__ out) {
  HFG_FOR(c, r.size()) {
    int x, y, z;
    cellCoord(c, r, x, y, z);
    auto solidAt = [&](long long i) { return solidSdf ? solidSdf[i] < 0.f : solidIdx[i] != 0; };
    float v = 0.f;
    if (dom[c] < 0.f && !solidAt(c)) {
      const int dx[6] = {-1, 1, 0, 0, 0, 0}, dy[6] = {0, 0, -1, 1, 0, 0}, dz[6] = {0, 0, 0, 0, -1, 1};
      bool air = false;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        long long nb = linc(x + dx[k], y + dy[k], z + dz[k], r);
        air |= dom[nb] >= 0.f && !solidAt(nb);
      }
      v = air ? (float)0.2 : 1.f;  // FluidSurfaceDensity (Common.h:244)
    }
    out[c] = v;
  }
}
cudaError_t launchFluidDensity(const Dim3i& r, const float* dom, const float* solidSdf, const uint8_t* solidIdx,
                               float* out, cudaStream_t s) {
  kFluidDensity<<<gridFor(r.size()), kThreads, 0, s>>>(r, dom, solidSdf, solidIdx, out);
  return cudaGetLastError();
}

// Grid <-> particle mixing of the hybrid coupler.
// HybridSimulatorMixFieldWithDensity.cu:6-265: B := (wA A + wB B) / (wA + wB)
// where wA + wB > FLT_EPSILON; on a face grid the weights are the means of the
// two adjacent cells (clamp to edge), scaled by the reference's double 0.5.
__device__ __forceinline__ void mixOne(float a, float& b, float wa, float wb) {
  float s = __fadd_rn(wa, wb);
  if (s > FLT_EPSILON) b = __fdiv_rn(__fadd_rn(__fmul_rn(wa, a), __fmul_rn(wb, b)), s);
}
__global__ void kMixCell(long long n, const float* __restrict__ a, float* __restrict__ b, const float* __restrict__ wa,
                         const float* __restrict__ wb) {
  HFG_FOR(i, n) {
    float v = b[i];
    mixOne(a[i], v, wa[i], wb[i]);
    b[i] = v;
  }
}
__global__ void kMixFace(Dim3i r, int axis, const float* __restrict__ a, float* __restrict__ b,
                         const float* __restrict__ wa, const float* __restrict__ wb) {
  const Dim3i f{r.x + (axis == 0), r.y + (axis == 1), r.z + (axis == 2)};
  HFG_FOR(c, f.size()) {
    int x, y, z;
    cellCoord(c, f, x, y, z);
    long long lo = linc(x - (axis == 0), y - (axis == 1), z - (axis == 2), r), hi = linc(x, y, z, r);
    float wA = __double2float_rn(__dmul_rn((double)__fadd_rn(wa[lo], wa[hi]), 0.5));
    float wB = __double2float_rn(__dmul_rn((double)__fadd_rn(wb[lo], wb[hi]), 0.5));
    float v = b[c];
    mixOne(a[c], v, wA, wB);
    b[c] = v;
  }
}
cudaError_t launchMixFieldWithDensity(const Dim3i& r, int face, const float* const a[3], float* const b[3],
                                      const float* wa, const float* wb, cudaStream_t s) {
  if (!face) {
    kMixCell<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), a[0], b[0], wa, wb);
    return cudaGetLastError();
  }
  for (int axis = 0; axis < 3; ++axis) {
    kMixFace<<<gridFor(r.size()), kThreads, 0, s>>>(r, axis, a[axis], b[axis], wa, wb);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
// HybridSimulatorMixParitcleVelWithPICAndFLIP.cu:5-57: by the particle's
// distance d: PIC up to g cells, PIC -> predicted up to gf, FLIP up to f,
// FLIP -> predicted up to p, predicted beyond (lerp(a, b, t) = a + t (b - a)).
__global__ void kMixParticleVel(const float* __restrict__ pic, const float* __restrict__ flip,
                                const float* __restrict__ dist, long long n, float cell, float g, float gf, float fr,
                                float pr, float* __restrict__ predict) {
  const float dg = __fmul_rn(g, cell), dgf = __fmul_rn(gf, cell), df = __fmul_rn(fr, cell), dp = __fmul_rn(pr, cell);
  HFG_FOR(i, n) {
    const float d = dist[i];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float P = pic[3 * i + a], F = flip[3 * i + a], Q = predict[3 * i + a];
      float m;
      if (d <= dg) m = P;
      else if (d <= dgf) m = __fadd_rn(P, __fmul_rn(__fdiv_rn(__fsub_rn(d, dg), __fsub_rn(dgf, dg)), __fsub_rn(Q, P)));
      else if (d <= df) m = F;
      else if (d <= dp) m = __fadd_rn(F, __fmul_rn(__fdiv_rn(__fsub_rn(d, df), __fsub_rn(dp, df)), __fsub_rn(Q, F)));
      else m = Q;
      predict[3 * i + a] = m;
    }
  }
}
cudaError_t launchMixParticleVel(const float* pic, const float* flip, const float* dist, long long n, float cell,
                                 float g, float gf, float f, float p, float* predict, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  kMixParticleVel<<<gridFor(n), kThreads, 0, s>>>(pic, flip, dist, n, cell, g, gf, f, p, predict);
  return cudaGetLastError();
}

cudaError_t launchFluidSdf(const Dim3i& r, const float* dom, float* sdf, int layers, int* steps, unsigned int* changed,
                           cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(changed, 0, sizeof(unsigned int) * kStepFlags, s);
  if (e != cudaSuccess) return e;
  kFluidSdfSeed<<<gridFor(r.size()), kThreads, 0, s>>>(r, dom, steps);
  if ((e = launchStepRounds(r, steps, changed, 1, s)) != cudaSuccess) return e;
  kFluidSdfValue<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), dom, steps, layers, sdf);
  return cudaGetLastError();
}

// ===========================================================================
// Inside / outside distance fields of the fluid density (the hybrid
// coupler's buildFluidInsideSDF / buildFluidOutsideSDF,
// HybridSimulatorBuildSDF.cu:4-146,177-238).  Sweep 0 gives solids 0,
// surface cells (density 0.2) the seed value s (0.2 - 0.5 inside, 0.5 - 0.2
// outside), cells of density 0 (inside) or 1 (outside) 0 and the rest
// UNKNOWN; sweep d then gives every UNKNOWN 6-neighbour of a cell holding
// d - 1 + s the value d + s, and negative values end as 0.  So the surface
// cells are the seeds and the cells that sweep 0 sets to 0 are closed.
// ===========================================================================
namespace {
__device__ __forceinline__ bool realEq(float a, float b) { return fabsf(__fsub_rn(a, b)) < FLT_MIN; }  // isRealEQ
}  // namespace

__global__ void kSideSdfSeed(long long n, const float* __restrict__ density, const float* __restrict__ solid,
                             float zero, int* __restrict__ d) {
  HFG_FOR(c, n) {
    const float rho = density[c];
    int v = kStepsFar;
    if (solid[c] < 0.f) v = kStepsClosed;
    else if (realEq(rho, (float)kSurf)) v = 0;
    else if (realEq(rho, zero)) v = kStepsClosed;
    d[c] = v;
  }
}
// the value of every cell, buildFluidSDFPostProcess (HybridSimulatorBuildSDF.cu:122-137) included
__global__ void kSideSdfValue(long long n, const int* __restrict__ d, double seed, int sweeps,
                              float* __restrict__ out) {
  HFG_FOR(c, n) {
    const int k = d[c];
    float v = kUnknown;
    if (k < 0) v = 0.f;
    else if (k < sweeps) v = fmaxf((float)((double)k + seed), 0.f);
    out[c] = v;
  }
}
__global__ void kNegativeToZero(long long n, float* __restrict__ out) {
  HFG_FOR(i, n) {
    if (out[i] < 0.f) out[i] = 0.f;
  }
}

cudaError_t launchFluidSideSdf(const Dim3i& r, const float* density, const float* solid, bool outside, int distance,
                               float* out, int* steps, unsigned int* changed, unsigned int* hostFlags,
                               cudaStream_t s) {
  if (distance <= 0) {
    kNegativeToZero<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), out);
    return cudaGetLastError();
  }
  // the reference's UInt + double expressions, rounded to Real once; sweep d
  // looks for (d + s) - 1, and where that is not the value sweep d - 1 wrote,
  // the reference's shell stops growing
  const double seed = outside ? 0.5 - kSurf : kSurf - 0.5;
  int sweeps = 1;
  while (sweeps < distance && (float)((double)sweeps + seed - 1) == (float)((double)(sweeps - 1) + seed)) ++sweeps;
  kSideSdfSeed<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), density, solid, outside ? 1.f : 0.f, steps);
  // Three rounds see most scenes through (walks around a convex solid have two
  // or three pieces); then twice as many each time.  Walks that wind among
  // scattered closed cells have a piece to every step or two: what is left after
  // a share of the rounds that the levels would pay for (a round costs 3 levels
  // on 33^3, 4 on 96^3, 14 on 256^3) is taken level by level, and so is all of it
  // when only a few levels are asked for.  Calls in us, rounds alone / this / one
  // launch and host read per level, three cells in ten closed at random: 96^3,
  // 1000 levels 1230 / 690 / 3400, 30 levels 1180 / 490 / 1010; 256^3 9100 / 5760
  // / 9000 and 9100 / 1750 / 1870; one corridor of 32 turns on 64^3 920 / 930 /
  // 22000.
  const int levels = sweeps - 1;
  const bool large = r.size() > (1 << 21);
  bool settled = levels == 0;
  auto pass = [&](int slots, auto&& launch) -> cudaError_t {  // and whether its last slot changed nothing
    cudaError_t e = cudaMemsetAsync(changed, 0, sizeof(unsigned int) * kStepFlags, s);
    if (e == cudaSuccess) e = launch();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(hostFlags, changed, sizeof(unsigned int) * slots, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    settled = hostFlags[slots - 1] == 0u;
    return e;
  };
  cudaError_t e = cudaSuccess;
  if (levels > (large ? 24 : 8))
    for (int n = 3, left = std::max(9, levels / (large ? 64 : 12)); !settled && left > 0 && e == cudaSuccess;
         n = std::min(2 * n, kStepFlags)) {
      const int rounds = std::min(n, left);
      e = pass(rounds, [&] { return launchStepRounds(r, steps, changed, rounds, s); });
      left -= rounds;
    }
  if (e == cudaSuccess && !settled) {
    const StepBits bits = stepBits(r, steps);
    kStepsToBits<<<gridFor((long long)stepBitsWords(r) * 32), kThreads, 0, s>>>(r, steps, bits);
    for (int k = 1; !settled && k <= levels && e == cudaSuccess; k += kStepFlags) {
      const int n = std::min(kStepFlags, levels - k + 1);
      if (k + n > levels) {  // the last ones: nobody asks whether there are more
        e = cudaMemsetAsync(changed, 0, sizeof(unsigned int) * kStepFlags, s);
        if (e == cudaSuccess) e = launchStepLevels(r, steps, bits, changed, k, n, s);
      } else {
        e = pass(n, [&] { return launchStepLevels(r, steps, bits, changed, k, n, s); });
      }
    }
  }
  if (e != cudaSuccess) return e;
  kSideSdfValue<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), steps, seed, sweeps, out);
  return cudaGetLastError();
}

// buildMixedFluidOutsideSDF (HybridSimulatorBuildSDF.cu:139-175): at a cell of
// grid density 0.2, 0.5 minus the mixed density (negative -> 0); elsewhere
// the grid fluid's outside distance.
__global__ void kMixedOutsideSdf(long long n, const float* __restrict__ gridDensity,
                                 const float* __restrict__ mixedDensity, const float* __restrict__ gridOutside,
                                 float* __restrict__ out) {
  HFG_FOR(c, n) {
    float v;
    if (realEq(gridDensity[c], (float)kSurf)) {
      v = __double2float_rn(0.5 - (double)mixedDensity[c]);
      if (v < 0.f) v = 0.f;
    } else {
      v = gridOutside[c];
    }
    out[c] = v;
  }
}
cudaError_t launchMixedOutsideSdf(const Dim3i& r, const float* gridDensity, const float* mixedDensity,
                                  const float* gridOutside, float* out, cudaStream_t s) {
  kMixedOutsideSdf<<<gridFor(r.size()), kThreads, 0, s>>>(r.size(), gridDensity, mixedDensity, gridOutside, out);
  return cudaGetLastError();
}

// ===========================================================================
// Particles
// ===========================================================================

// Philox4x32-10 (Salmon et al., SC'11): counter-based stream shared with the
// host so the seeding is reproducible anywhere.
__host__ __device__ inline void philox10(uint32_t c[4], uint32_t k0, uint32_t k1) {
  for (int r = 0; r < 10; ++r) {
    uint64_t p0 = (uint64_t)0xD2511F53u * c[0];
    uint64_t p1 = (uint64_t)0xCD9E8D57u * c[2];
    uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0, n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1;
    c[1] = (uint32_t)p1;
    c[3] = (uint32_t)p0;
    c[0] = n0;
    c[2] = n2;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}
__device__ inline float unit24(uint32_t v) { return (float)(v >> 8) * (1.0f / 16777216.0f); }

// EulerParticlesTool.cu:5-25 findFluidGrid: fluid SDF < 0 and not solid.
__device__ inline bool seedCell(const float* fsdf, const uint8_t* sidx, long long c) {
  return fsdf[c] < 0.f && !(sidx && sidx[c]);
}

__global__ void kSeedCount(long long n, const float* __restrict__ fsdf, const uint8_t* __restrict__ sidx,
                           unsigned int* __restrict__ blockCounts, int cellsPerBlock) {
  long long b0 = (long long)blockIdx.x * cellsPerBlock;
  unsigned int cnt = 0;
  for (long long c = b0 + threadIdx.x; c < b0 + cellsPerBlock && c < n; c += blockDim.x) cnt += seedCell(fsdf, sidx, c);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  __shared__ unsigned int s[32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += s[i];
    blockCounts[blockIdx.x] = t;
  }
}
cudaError_t launchSeedCount(const Dim3i& r, const float* fluidSDF, const uint8_t* solidIdx, unsigned int* blockCounts,
                            int cellsPerBlock, cudaStream_t s) {
  long long n = r.size();
  int nb = (int)((n + cellsPerBlock - 1) / cellsPerBlock);
  kSeedCount<<<nb, kThreads, 0, s>>>(n, fluidSDF, solidIdx, blockCounts, cellsPerBlock);
  return cudaGetLastError();
}

__global__ void kSeedScan(unsigned int* counts, int n, unsigned long long* total) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    unsigned long long s = 0;
    for (int i = 0; i < n; ++i) { unsigned int c = counts[i]; counts[i] = (unsigned int)s; s += c; }
    *total = s;
  }
}
cudaError_t launchSeedScan(unsigned int* blockCounts, int nBlocks, unsigned long long* total, cudaStream_t s) {
  kSeedScan<<<1, 1, 0, s>>>(blockCounts, nBlocks, total);
  return cudaGetLastError();
}

// EulerParticles.cpp:156-176: particle k of the f-th fluid cell (cells in
// linear order) at ((x + u) h + o) with u from Philox(cell, k; seed).
__global__ void kSeedWrite(Geom g, const float* __restrict__ fsdf, const uint8_t* __restrict__ sidx,
                           const unsigned int* __restrict__ blockOff, int cellsPerBlock, int ppc,
                           unsigned long long seed, float* __restrict__ pos) {
  long long n = g.r.size();
  long long b0 = (long long)blockIdx.x * cellsPerBlock;
  __shared__ unsigned int warpBase[32];
  __shared__ unsigned int runBase;
  if (threadIdx.x == 0) runBase = blockOff[blockIdx.x];
  __syncthreads();
  for (long long c0 = b0; c0 < b0 + cellsPerBlock && c0 < n; c0 += blockDim.x) {
    long long c = c0 + threadIdx.x;
    bool f = c < b0 + cellsPerBlock && c < n && seedCell(fsdf, sidx, c);
    unsigned int ball = __ballot_sync(0xffffffffu, f);
    unsigned int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) warpBase[w] = __popc(ball);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned int s = runBase;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { unsigned int t = warpBase[i]; warpBase[i] = s; s += t; }
      runBase = s;
    }
    __syncthreads();
    if (f) {
      unsigned long long rank = warpBase[w] + __popc(ball & ((1u << lane) - 1u));
      int x, y, z;
      cellCoord(c, g.r, x, y, z);
      for (int k = 0; k < ppc; ++k) {
        uint32_t ctr[4] = {(uint32_t)c, (uint32_t)((unsigned long long)c >> 32), (uint32_t)k, 0u};
        philox10(ctr, (uint32_t)seed, (uint32_t)(seed >> 32));
        float* q = pos + 3 * (rank * ppc + k);
        q[0] = __fadd_rn(__fmul_rn(__fadd_rn((float)x, unit24(ctr[0])), g.hx), g.ox);
        q[1] = __fadd_rn(__fmul_rn(__fadd_rn((float)y, unit24(ctr[1])), g.hy), g.oy);
        q[2] = __fadd_rn(__fmul_rn(__fadd_rn((float)z, unit24(ctr[2])), g.hz), g.oz);
      }
    }
    __syncthreads();
  }
}
cudaError_t launchSeedWrite(const Geom& g, const float* fluidSDF, const uint8_t* solidIdx,
                            const unsigned int* blockOffsets, int cellsPerBlock, int ppc, unsigned long long seed,
                            float* pos, cudaStream_t s) {
  long long n = g.r.size();
  int nb = (int)((n + cellsPerBlock - 1) / cellsPerBlock);
  kSeedWrite<<<nb, kThreads, 0, s>>>(g, fluidSDF, solidIdx, blockOffsets, cellsPerBlock, ppc, seed, pos);
  return cudaGetLastError();
}

// Particle velocity update before advection:
//   PIC  (ParticleInCell.cpp:102-104):       v = G2P(vin)
//   FLIP (FluidImplicitParticle.cpp:107-119): v += G2P(vin - prev)
//   MIX  (MixPICAndFLIP.cpp:112-129):        v = (1-m)(v + G2P(vin - prev)) + m G2P(vin)
// with prev = the previous step's P2G output, or prev = 0 on the first FLIP step.
template <int ALG>
__global__ void kParticleVelUpdate(Geom g, int mode, ConstFaceField vin, ConstFaceField prev, int first, float mixing,
                                   const float* __restrict__ pos, float* __restrict__ vel, long long P) {
  const float keep = (float)(1.0 - (double)mixing);
  HFG_FOR(p, P) {
    float px = pos[3 * p], py = pos[3 * p + 1], pz = pos[3 * p + 2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      Geom fg = faceGeom(g, a);
      float v = vel[3 * p + a];
      if (mode == MODE_PIC) {
        v = g2p<ALG>(vin.c[a], fg, px, py, pz);
      } else {
        float pic = (mode == MODE_MIX) ? g2p<ALG>(vin.c[a], fg, px, py, pz) : 0.f;
        float dv;
        if (first) {
          dv = g2p<ALG>(vin.c[a], fg, px, py, pz);
        } else {
          // G2P of the face-wise difference vin - prev
          Taps t;
          taps<ALG == G2PNEAREST ? LINEAR : ALG>(fg, px, py, pz, t);
          constexpr int A = ALG == G2PNEAREST ? LINEAR : ALG, n = TapsN<A>::n;
          const TapRows<A> at(fg, t);
          dv = 0.f;
          if (ALG == G2PNEAREST) {
            long long i = binCell(fg, px, py, pz);
            dv = __fsub_rn(__ldg(vin.c[a] + i), __ldg(prev.c[a] + i));
          } else {
#pragma unroll
            for (int z = 0; z < n; ++z)
#pragma unroll
              for (int y = 0; y < n; ++y)
#pragma unroll
                for (int x = 0; x < n; ++x) {
                  float w = t.w[0][x] * t.w[1][y] * t.w[2][z];
                  const unsigned i = at(x, y, z);
                  dv += w * __fsub_rn(__ldg(vin.c[a] + i), __ldg(prev.c[a] + i));
                }
          }
        }
        v = __fadd_rn(dv, v);
        if (mode == MODE_MIX) {
          v = __fmul_rn(v, keep);
          v = fmaf(mixing, pic, v);
        }
      }
      vel[3 * p + a] = v;
    }
  }
}

__device__ inline void blockMaxToGlobal(float m, unsigned int* dst);

// LINEAR transfers (the configuration of every benchmark scene), fused with the
// first velocity sample of the substep loop that follows
// (EulerParticles.cpp:249-251): one sampler per particle serves the PIC sample,
// the FLIP difference and all three components.  The PIC sample comes from the
// corner tables of vin and is also v0 of the substeps, with max |v0|.
template <typename I>
__global__ void kParticleVelUpdateLinear(Geom g, int mode, FaceQuads vinQ, ConstFaceField vin, ConstFaceField prev,
                                         int first, float mixing, const float* __restrict__ pos,
                                         float* __restrict__ vel, long long P, float* __restrict__ v0,
                                         SubstepState* st) {
  const float keep = (float)(1.0 - (double)mixing);
  const I stride = (I)gridDim.x * blockDim.x;
  float m = 0.f;
  HFG_FOR_T(I, p, P) {
    if (p + stride < (I)P) {  // the next iteration's lines (two or four ahead gained less)
      prefetchL2(pos + 3 * (p + stride));
      prefetchL2(vel + 3 * (p + stride));
    }
    FaceSampler fs(vinQ, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], FaceSampler::IndexClamp{});
    float pic[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      pic[a] = fs.sampleQuads(vinQ, a);
      v0[3 * p + a] = pic[a];
      m = fmaxf(m, fabsf(pic[a]));
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float v = vel[3 * p + a];
      if (mode == MODE_PIC) {
        v = pic[a];
      } else {
        float dv = first ? pic[a] : fs.sampleDiff(g, a, vin.c[a], prev.c[a]);
        v = __fadd_rn(dv, v);
        if (mode == MODE_MIX) {
          v = __fmul_rn(v, keep);
          v = fmaf(mixing, pic[a], v);
        }
      }
      vel[3 * p + a] = v;
    }
  }
  blockMaxToGlobal(m, &st[0].maxAbsBits);
}

cudaError_t launchParticleVelUpdate(const Geom& g, int mode, int alg, ConstFaceField vin, ConstFaceField prev,
                                    int firstFlip, float mixing, const float* pos, float* vel, long long P,
                                    cudaStream_t s, const FaceQuads* vinQ, float* v0, SubstepState* st) {
  if (P <= 0) return cudaSuccess;
  int gr = gridFor(P);
  switch (alg) {
    case LINEAR:
      if (!vinQ || !v0 || !st) return cudaErrorInvalidValue;
      if (index32(P))
        kParticleVelUpdateLinear<int><<<gr, kThreads, 0, s>>>(g, mode, *vinQ, vin, prev, firstFlip, mixing, pos, vel,
                                                              P, v0, st);
      else
        kParticleVelUpdateLinear<long long><<<gr, kThreads, 0, s>>>(g, mode, *vinQ, vin, prev, firstFlip, mixing, pos,
                                                                    vel, P, v0, st);
      break;
    case QUADRATIC: kParticleVelUpdate<QUADRATIC><<<gr, kThreads, 0, s>>>(g, mode, vin, prev, firstFlip, mixing, pos, vel, P); break;
    case CUBIC: kParticleVelUpdate<CUBIC><<<gr, kThreads, 0, s>>>(g, mode, vin, prev, firstFlip, mixing, pos, vel, P); break;
    case G2PNEAREST: kParticleVelUpdate<G2PNEAREST><<<gr, kThreads, 0, s>>>(g, mode, vin, prev, firstFlip, mixing, pos, vel, P); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// max of m over the block, then atomically into *dst (bits of a float >= 0)
__device__ inline void blockMaxToGlobal(float m, unsigned int* dst) {
  __shared__ float s[32];
  m = warpMaxF(m);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    int nw = blockDim.x >> 5;
    float v = (int)threadIdx.x < nw ? s[threadIdx.x] : 0.f;
    v = warpMaxF(v);
    if (threadIdx.x == 0) atomicMax(dst, __float_as_uint(v));
  }
}

// Corner tables of the three face grids (FaceQuads), one component per
// blockIdx.y; consecutive threads take consecutive jx.
__global__ void kFaceQuads(Dim3i r, ConstFaceField v, float4* q0, float4* q1, float4* q2) {
  const int a = blockIdx.y;
  const unsigned nx = (unsigned)(r.x + (a == 0)), ny = (unsigned)(r.y + (a == 1)), nz = (unsigned)(r.z + (a == 2));
  const unsigned lx = nx + 1, ly = ny + 1;
  const long long n = (long long)lx * ly * (nz + 2);
  const float* __restrict__ f = a == 0 ? v.c[0] : (a == 1 ? v.c[1] : v.c[2]);
  float4* __restrict__ out = a == 0 ? q0 : (a == 1 ? q1 : q2);
  HFG_FOR(e, n) {
    const unsigned t = (unsigned)(e / lx), jx = (unsigned)(e - (long long)t * lx);
    const unsigned L = t / ly, jy = t - L * ly;
    const unsigned z = L == 0 ? 0 : (L > nz ? nz - 1 : L - 1);
    const unsigned x0 = jx > 0 ? jx - 1 : 0, x1 = jx < nx ? jx : nx - 1;
    const unsigned y0 = jy > 0 ? jy - 1 : 0, y1 = jy < ny ? jy : ny - 1;
    const unsigned b0 = (z * ny + y0) * nx, b1 = (z * ny + y1) * nx;
    const float f00 = __ldg(f + b0 + x0), f01 = __ldg(f + b0 + x1), f10 = __ldg(f + b1 + x0), f11 = __ldg(f + b1 + x1);
    out[e] = make_float4(f00, __fsub_rn(f01, f00), f10, __fsub_rn(f11, f10));
  }
}
long long faceQuadCount(const Dim3i& r, int a) {
  return (long long)(r.x + (a == 0) + 1) * (r.y + (a == 1) + 1) * (r.z + (a == 2) + 2);
}
cudaError_t launchFaceQuads(const Dim3i& r, ConstFaceField v, float4* const out[3], cudaStream_t s) {
  long long n = faceQuadCount(r, 0);
  dim3 grid(gridFor(n), 3);
  kFaceQuads<<<grid, kThreads, 0, s>>>(r, v, out[0], out[1], out[2]);
  return cudaGetLastError();
}

// First velocity sample of the substep loop (EulerParticles.cpp:249-251):
// v0 = trilinear(vel, pos) and max |v0| over every component.
template <typename I>
__global__ void kSubstepBegin(Geom g, FaceQuads vel, const float* __restrict__ pos, float* __restrict__ v0,
                              long long P, SubstepState* st) {
  float m = 0.f;
  HFG_FOR_T(I, p, P) {
    float v[3];
    sampleFaceQuads(vel, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], v);
    v0[3 * p] = v[0]; v0[3 * p + 1] = v[1]; v0[3 * p + 2] = v[2];
    m = fmaxf(m, fmaxf(fabsf(v[0]), fmaxf(fabsf(v[1]), fabsf(v[2]))));
  }
  blockMaxToGlobal(m, &st[0].maxAbsBits);
}
cudaError_t launchSubstepBegin(const Geom& g, FaceQuads vel, const float* pos, float* v0, long long P,
                               SubstepState* st, cudaStream_t s) {
  if (index32(P))
    kSubstepBegin<int><<<gridFor(P > 0 ? P : 1), kThreads, 0, s>>>(g, vel, pos, v0, P, st);
  else
    kSubstepBegin<long long><<<gridFor(P > 0 ? P : 1), kThreads, 0, s>>>(g, vel, pos, v0, P, st);
  return cudaGetLastError();
}

// Substep size rule of EulerParticles.cpp:253-275, evaluated identically by
// every thread from the slot's state.
__device__ inline float substepSize(const SubstepState& s, float dt, float cfl, float minH, bool& last) {
  float amax = __uint_as_float(s.maxAbsBits);
  float d = (amax != 0.f) ? __fdiv_rn(__fmul_rn(cfl, minH), amax) : dt;
  last = false;
  if (__fadd_rn(s.subTime, d) >= dt) {
    d = __fsub_rn(dt, s.subTime);
    last = true;
  } else if (__fadd_rn(s.subTime, __fmul_rn(2.f, d)) >= dt) {
    d = (float)(0.5 * (double)__fsub_rn(dt, s.subTime));
  }
  return d;
}

// One RK1/2/3 substep (EulerParticles.cpp:277-318).  After the last substep the
// box clamp of fixParticlesPosWithBoundarys (EulerParticlesTool.cu:310-333) is
// applied to the first `nclamp` particles; otherwise the next v0 and its max
// are produced for slot+1.
// One particle's substep: RK1/2/3 from its v0, the box clamp after the last
// substep, otherwise the next v0 sampled and stored; returns max |v0 next|.
template <typename I>
__device__ __forceinline__ float substepParticle(const Geom& g, const FaceQuads& vel, float* __restrict__ pos,
                                                 float* __restrict__ v0, I p, int acc, float ds, float half, float tq,
                                                 float a29, float a39, float a49, bool last, bool clampIt) {
  float q[3] = {pos[3 * p], pos[3 * p + 1], pos[3 * p + 2]};
  float w0[3] = {v0[3 * p], v0[3 * p + 1], v0[3 * p + 2]};
  float m = 0.f;
  QuadCache qc;
  bool fresh = true;  // no entry cached yet
  if (acc == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = fmaf(ds, w0[a], q[a]);
  } else if (acc == 1) {
    float mid[3], w1[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) mid[a] = fmaf(half, w0[a], q[a]);
    sampleFaceQuadsCached(vel, mid[0], mid[1], mid[2], w1, qc, true);
    fresh = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = fmaf(ds, w1[a], q[a]);
  } else {
    // q + a29 w0 + a39 w1 + a49 w2, in that order, accumulated as soon as
    // each sample is known so that fewer values stay live across a sample
    float mid[3], tf[3], acc3[3], w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mid[a] = fmaf(half, w0[a], q[a]);
      acc3[a] = fmaf(a29, w0[a], q[a]);
    }
    sampleFaceQuadsCached(vel, mid[0], mid[1], mid[2], w, qc, true);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      tf[a] = fmaf(tq, w[a], q[a]);
      acc3[a] = fmaf(a39, w[a], acc3[a]);
    }
    sampleFaceQuadsCached(vel, tf[0], tf[1], tf[2], w, qc, false);
    fresh = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = fmaf(a49, w[a], acc3[a]);
  }
  if (last) {
    if (clampIt) {  // the box bounds are formed here, from the kernel parameters
      const float bmin[3] = {g.ox, g.oy, g.oz};
      const float bmax[3] = {g.ox + (float)g.r.x * g.hx, g.oy + (float)g.r.y * g.hy, g.oz + (float)g.r.z * g.hz};
#pragma unroll
      for (int a = 0; a < 3; ++a) q[a] = fmaxf(bmin[a], fminf(q[a], bmax[a]));
    }
  } else {
    float v[3];
    sampleFaceQuadsCached(vel, q[0], q[1], q[2], v, qc, fresh);
    v0[3 * p] = v[0]; v0[3 * p + 1] = v[1]; v0[3 * p + 2] = v[2];
    m = fmaxf(fabsf(v[0]), fmaxf(fabsf(v[1]), fabsf(v[2])));
  }
  pos[3 * p] = q[0]; pos[3 * p + 1] = q[1]; pos[3 * p + 2] = q[2];
  return m;
}

// The RK coefficients of a substep of size ds (EulerParticles.cpp:281-301).
struct SubstepCoef {
  float ds, half, tq, a29, a39, a49;
  SubstepCoef() = default;
  __device__ explicit SubstepCoef(float d)
      : ds(d), half((float)(0.5 * (double)d)), tq((float)(0.75 * (double)d)), a29((float)(2.0 / 9.0 * (double)d)),
        a39((float)(3.0 / 9.0 * (double)d)), a49((float)(4.0 / 9.0 * (double)d)) {}
};

// One RK1/2/3 substep (EulerParticles.cpp:277-318).  After the last substep the
// box clamp of fixParticlesPosWithBoundarys (EulerParticlesTool.cu:310-333) is
// applied to the first `nclamp` particles; otherwise the next v0 and its max
// are produced for slot+1.  ACC: the RK order (0, 1, 2), fixed per
// instantiation so that the particle loop carries no branch on it.
// One wave of blocks, each thread walking its share, so that neighbouring
// particles' table entries are in L1 and L2 together: with four waves a 256^3
// step's substeps (31.4 M particles, RK3) took 12.5 ms, with one 11.0.  512
// threads against 256: 7.6 M particles on 160^3 1.20 against 1.26 ms a call,
// alike at 256^3 and below 1 M particles; 1.5 or 3 waves 14 ms.
constexpr int kSubstepThreads = 512, kSubstepPerSM = 2;
template <typename I, int ACC>
__global__ void __launch_bounds__(kSubstepThreads, kSubstepPerSM) kSubstep(Geom g, FaceQuads vel, float* __restrict__ pos,
                                                  float* __restrict__ v0, long long P, float dt, float cfl,
                                                  long long nclamp, SubstepState* st, int slot) {
  const SubstepState cur = st[slot];
  if (cur.finished) {
    // carry the finished state forward so later speculative launches no-op
    if (blockIdx.x == 0 && threadIdx.x == 0) st[slot + 1] = cur;
    return;
  }
  // the substep size and RK coefficients, formed once per block: held in
  // shared memory, a use is one load where registers would have to give way
  // to recomputing them (FP64 products) inside the particle loop
  __shared__ SubstepCoef sk;
  __shared__ int sLast;
  if (threadIdx.x == 0) {
    bool l;
    sk = SubstepCoef(substepSize(cur, dt, cfl, fminf(fminf(g.hx, g.hy), g.hz), l));
    sLast = l ? 1 : 0;
  }
  __syncthreads();
  const SubstepCoef& k = sk;
  const bool last = sLast != 0;
  float m = 0.f;
  const I stride = (I)gridDim.x * blockDim.x;
  HFG_FOR_T(I, p, P) {
    // the stream loads of a later iteration are DRAM misses; ask for them now
    // so that the chain of samples below does not start with one
    if (p + stride < (I)P) {
      prefetchL2(pos + 3 * (p + stride));
      prefetchL2(v0 + 3 * (p + stride));
    }
    m = fmaxf(m, substepParticle<I>(g, vel, pos, v0, p, ACC, k.ds, k.half, k.tq, k.a29, k.a39, k.a49, last,
                                    (long long)p < nclamp));
  }
  if (!last) blockMaxToGlobal(m, &st[slot + 1].maxAbsBits);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st[slot + 1].subTime = __fadd_rn(cur.subTime, k.ds);
    st[slot + 1].finished = last ? 1 : 0;
    st[slot + 1].count = cur.count + 1;
  }
}

// The substep `slot` of many scenes in one launch (the batched mode).  Scene
// s owns blocks [chunkStart[s], chunkStart[s + 1]), each a chunk of
// kMultiChunk of its particles; a block finds its scene by binary search and
// runs that scene's substep with the scene's own CFL state, exactly as
// kSubstep would.  Scenes whose substeps are finished do nothing.
constexpr int kMultiChunk = 8 * kThreads;
__global__ void __launch_bounds__(256, 3) kSubstepMulti(const SubstepTask* __restrict__ tasks,
                                                       const long long* __restrict__ chunkStart, int nScenes,
                                                       int slot) {
  __shared__ int sc;
  __shared__ FaceQuads sq;
  if (threadIdx.x == 0) {
    int lo = 0, hi = nScenes - 1;  // the last scene whose first chunk is <= blockIdx.x
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (chunkStart[mid] <= (long long)blockIdx.x) lo = mid;
      else hi = mid - 1;
    }
    sc = lo;
    sq = tasks[lo].vel;
  }
  __syncthreads();
  const SubstepTask& T = tasks[sc];
  const long long chunk = (long long)blockIdx.x - chunkStart[sc];
  const SubstepState cur = T.st[slot];
  if (cur.finished) {
    if (chunk == 0 && threadIdx.x == 0) T.st[slot + 1] = cur;
    return;
  }
  const Geom g = T.g;
  // the scene's tables and sampling constants, read from shared memory where
  // used (held in registers they spill)
  const FaceQuads& vel = sq;
  const float minH = fminf(fminf(g.hx, g.hy), g.hz);
  bool last;
  const SubstepCoef k(substepSize(cur, T.dt, T.cfl, minH, last));
  float m = 0.f;
  // the chunk's particles, indexed in 32 bits from the chunk's start
  const long long p0 = chunk * kMultiChunk;
  const int n = (int)(min(T.P, p0 + kMultiChunk) - p0);
  const long long nclamp = T.nclamp - p0;
  float* pos = T.pos + 3 * p0;
  float* v0 = T.v0 + 3 * p0;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    m = fmaxf(m, substepParticle<int>(g, vel, pos, v0, i, T.acc, k.ds, k.half, k.tq, k.a29, k.a39, k.a49, last,
                                      (long long)i < nclamp));
  if (!last) blockMaxToGlobal(m, &T.st[slot + 1].maxAbsBits);
  if (chunk == 0 && threadIdx.x == 0) {
    T.st[slot + 1].subTime = __fadd_rn(cur.subTime, k.ds);
    T.st[slot + 1].finished = last ? 1 : 0;
    T.st[slot + 1].count = cur.count + 1;
  }
}
long long multiSubstepChunks(long long P) { return (P + kMultiChunk - 1) / kMultiChunk; }
cudaError_t launchSubstepMulti(const SubstepTask* tasks, const long long* chunkStart, int nScenes,
                               long long totalChunks, int slot, cudaStream_t s) {
  if (nScenes <= 0 || totalChunks <= 0) return cudaSuccess;
  kSubstepMulti<<<(unsigned)totalChunks, kThreads, 0, s>>>(tasks, chunkStart, nScenes, slot);
  return cudaGetLastError();
}

// finished flag and substep count of every scene's state slot `slot`, into
// host-mapped memory (two ints per scene)
__global__ void kGatherSubstepStates(const SubstepTask* __restrict__ tasks, int nScenes, int slot, int* out) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nScenes; s += gridDim.x * blockDim.x) {
    const SubstepState v = tasks[s].st[slot];
    out[2 * s] = v.finished;
    out[2 * s + 1] = v.count;
  }
}
cudaError_t launchGatherSubstepStates(const SubstepTask* tasks, int nScenes, int slot, int* out, cudaStream_t s) {
  if (nScenes <= 0) return cudaSuccess;
  kGatherSubstepStates<<<(nScenes + 255) / 256, 256, 0, s>>>(tasks, nScenes, slot, out);
  return cudaGetLastError();
}

cudaError_t launchSubstep(const Geom& g, FaceQuads vel, float* pos, float* v0, long long P, int acc, float dt,
                          float cfl, long long nclamp, SubstepState* st, int slot, cudaStream_t s) {
  const int grid = gridFor(P > 0 ? P : 1, kSubstepThreads, kSubstepPerSM);
#define HFG_SUBSTEP(I, A) kSubstep<I, A><<<grid, kSubstepThreads, 0, s>>>(g, vel, pos, v0, P, dt, cfl, nclamp, st, slot)
  if (index32(P)) {
    if (acc == 0) HFG_SUBSTEP(int, 0);
    else if (acc == 1) HFG_SUBSTEP(int, 1);
    else HFG_SUBSTEP(int, 2);
  } else {
    if (acc == 0) HFG_SUBSTEP(long long, 0);
    else if (acc == 1) HFG_SUBSTEP(long long, 1);
    else HFG_SUBSTEP(long long, 2);
  }
#undef HFG_SUBSTEP
  return cudaGetLastError();
}

// Adds (value, weight) pairs to two neighbouring entries: one 16-byte atomic
// where the pair lies on a 16-byte boundary, else two of 8 bytes.
__device__ __forceinline__ void addPair(float2* p, float2 a, float2 b) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    atomicAdd(reinterpret_cast<float4*>(p), make_float4(a.x, a.y, b.x, b.y));
  } else {
    atomicAdd(p, a);
    atomicAdd(p + 1, b);
  }
}

// P2G of one particle to a grid, value and weight packed as float2
// (accumulateParticles2CCSField, EulerParticlesTool.cu:79-196).  The kernel is
// bound by the atomics at L2, so a row of four taps goes out as 16-byte atomics
// (two, or one and two 8-byte ones, by the row's alignment), and the taps that a
// quadratic kernel leaves without weight (37 of 64) are skipped; a value that
// is not finite still reaches them, as 0 times it is not 0.  0.9 M particles,
// 97 x 64 x 83, cubic: this kernel 0.86 -> 0.67 ms, a call 0.90 -> 0.70.  (The linear
// kernel's corners sent this way: 2.40 -> 2.50 ms at 256^3, so it keeps its own
// atomics.)
template <int ALG>
__device__ inline void p2gScatter(const Geom& fg, float px, float py, float pz, float val, float2* acc) {
  if (ALG == P2GSUM) {
    atomicAdd(&acc[binCell(fg, px, py, pz)].x, val);
    return;
  }
  Taps t;
  taps<ALG>(fg, px, py, pz, t);
  constexpr int n = TapsN<ALG>::n, s = TapsN<ALG>::shift;
  const int x0 = t.base[0] + s;
  const bool inRow = x0 >= 0 && x0 + n <= fg.r.x;
  const bool skip0 = ALG == QUADRATIC && fabsf(val) <= FLT_MAX;  // taps of weight 0 add nothing
#pragma unroll
  for (int z = 0; z < n; ++z)
#pragma unroll
    for (int y = 0; y < n; ++y) {
      if (skip0 && (t.w[1][y] == 0.f || t.w[2][z] == 0.f)) continue;
      float2 c[n];
#pragma unroll
      for (int x = 0; x < n; ++x) {
        const float w = t.w[0][x] * t.w[1][y] * t.w[2][z];
        c[x] = make_float2(w * val, w);
      }
      if (!inRow) {
#pragma unroll
        for (int x = 0; x < n; ++x)
          atomicAdd(acc + linc(t.base[0] + x + s, t.base[1] + y + s, t.base[2] + z + s, fg.r), c[x]);
        continue;
      }
      float2* row = acc + linc(x0, t.base[1] + y + s, t.base[2] + z + s, fg.r);
      if (n == 2) {
        atomicAdd(row, c[0]);
        atomicAdd(row + 1, c[1]);
      } else {
        const bool lo = !(skip0 && t.w[0][0] == 0.f), hi = !(skip0 && t.w[0][n - 1] == 0.f);
        if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
          if (lo) addPair(row, c[0], c[1]);
          else atomicAdd(row + 1, c[1]);
          if (hi) addPair(row + 2, c[n - 2], c[n - 1]);
          else atomicAdd(row + 2, c[n - 2]);
        } else {
          if (lo) atomicAdd(row, c[0]);
          addPair(row + 1, c[1], c[n - 2]);
          if (hi) atomicAdd(row + 3, c[n - 1]);
        }
      }
    }
}

// LINEAR P2G to the three face grids.  Particles are stored in seeding order
// (the particles of a cell next to each other) and move coherently, so the
// lanes of an aligned pair, quad or octet of a warp often share all eight
// corners of a component.  Such a group first sums its contributions with
// lane shuffles (levels skipped when no lane of the warp merges there), and one
// lane adds the sums to the grid: up to eight times fewer L2 atomics.  The
// sums differ from lane-by-lane atomics in the order of the additions only,
// as the order of the atomics does anyway.
__global__ void kP2GFaceLinear(Geom g, const float* __restrict__ pos, const float* __restrict__ vel, long long P,
                               float2* a0, float2* a1, float2* a2) {
  constexpr unsigned kAll = 0xffffffffu;
  float2* acc[3] = {a0, a1, a2};
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * blockDim.x;
  // warp-uniform trip count: every lane takes part in the shuffles
  for (long long p0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); p0 < P; p0 += stride) {
    const long long p = p0 + lane;
    const bool live = p < P;
    FaceSampler fs(g, live ? pos[3 * p] : g.ox, live ? pos[3 * p + 1] : g.oy, live ? pos[3 * p + 2] : g.oz);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      unsigned idx[8];
      float w[8];
      fs.corners(g, a, idx, w);
      const float val = live ? vel[3 * p + a] : 0.f;
      float vx[8], vw[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        vx[k] = w[k] * val;
        vw[k] = w[k];
      }
      // lanes with the same clamped floor indices (AxisW::j, -1 .. n - 1, which
      // fix both corners of an axis) share all eight corners; the key is
      // their linear index in a grid one larger per axis, less a constant, in
      // 32-bit unsigned arithmetic: distinct triples give distinct keys, and
      // the keys that wrap below zero land above 2^32 - 2^31, never on a dead
      // lane's 0x80000000 | lane
      const AxisW& X = a == 0 ? fs.fc[0] : fs.cc[0];
      const AxisW& Y = a == 1 ? fs.fc[1] : fs.cc[1];
      const AxisW& Z = a == 2 ? fs.fc[2] : fs.cc[2];
      const unsigned lx = (unsigned)(g.r.x + (a == 0) + 1), ly = (unsigned)(g.r.y + (a == 1) + 1);
      const unsigned key = live ? ((unsigned)Z.j * ly + (unsigned)Y.j) * lx + (unsigned)X.j : 0x80000000u | (unsigned)lane;
      const unsigned m = __match_any_sync(kAll, key);
      int group = 1;
#pragma unroll
      for (int lvl = 1; lvl <= 4; lvl <<= 1) {
        const unsigned gm = (lvl == 1 ? 0x3u : (lvl == 2 ? 0xFu : 0xFFu));
        const bool merge = group == lvl && ((m >> (lane & ~(2 * lvl - 1))) & gm) == gm;
        if (!__any_sync(kAll, merge)) break;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float ox = __shfl_xor_sync(kAll, vx[k], lvl), ow = __shfl_xor_sync(kAll, vw[k], lvl);
          if (merge) {
            vx[k] += ox;
            vw[k] += ow;
          }
        }
        if (merge) group = 2 * lvl;
      }
      if (live && (lane & (group - 1)) == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) atomicAdd(acc[a] + idx[k], make_float2(vx[k], vw[k]));
      }
    }
  }
}

template <int ALG>
__global__ void kP2GFace(Geom g, const float* __restrict__ pos, const float* __restrict__ vel, long long P,
                         float2* a0, float2* a1, float2* a2) {
  HFG_FOR(p, P) {
    float px = pos[3 * p], py = pos[3 * p + 1], pz = pos[3 * p + 2];
    p2gScatter<ALG>(faceGeom(g, 0), px, py, pz, vel[3 * p], a0);
    p2gScatter<ALG>(faceGeom(g, 1), px, py, pz, vel[3 * p + 1], a1);
    p2gScatter<ALG>(faceGeom(g, 2), px, py, pz, vel[3 * p + 2], a2);
  }
}
cudaError_t launchP2GFace(const Geom& g, int alg, const float* pos, const float* vel, long long P, float2* acc[3],
                          cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  int gr = gridFor(P);
  switch (alg) {
    case LINEAR: kP2GFaceLinear<<<gr, kThreads, 0, s>>>(g, pos, vel, P, acc[0], acc[1], acc[2]); break;
    case QUADRATIC: kP2GFace<QUADRATIC><<<gr, kThreads, 0, s>>>(g, pos, vel, P, acc[0], acc[1], acc[2]); break;
    case CUBIC: kP2GFace<CUBIC><<<gr, kThreads, 0, s>>>(g, pos, vel, P, acc[0], acc[1], acc[2]); break;
    case P2GSUM: kP2GFace<P2GSUM><<<gr, kThreads, 0, s>>>(g, pos, vel, P, acc[0], acc[1], acc[2]); break;
    default: break;  // G2PNEAREST has no P2G branch in the reference: nothing is accumulated
  }
  return cudaGetLastError();
}

template <int ALG>
__global__ void kP2GCell(Geom g, const float* __restrict__ pos, const float* __restrict__ val, long long P,
                         float2* acc) {
  HFG_FOR(p, P) p2gScatter<ALG>(g, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], val[p], acc);
}
cudaError_t launchP2GCell(const Geom& g, int alg, const float* pos, const float* val, long long P, float2* acc,
                          cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  int gr = gridFor(P);
  switch (alg) {
    case LINEAR: kP2GCell<LINEAR><<<gr, kThreads, 0, s>>>(g, pos, val, P, acc); break;
    case QUADRATIC: kP2GCell<QUADRATIC><<<gr, kThreads, 0, s>>>(g, pos, val, P, acc); break;
    case CUBIC: kP2GCell<CUBIC><<<gr, kThreads, 0, s>>>(g, pos, val, P, acc); break;
    case P2GSUM: kP2GCell<P2GSUM><<<gr, kThreads, 0, s>>>(g, pos, val, P, acc); break;
    default: break;
  }
  return cudaGetLastError();
}

// P2G of the four scalars the particles carry (colour and fluid domain) to the
// cells in one pass: the weights are the same for all, so a corner takes one
// 16-byte atomic for the values and one for the weight instead of four pairs.
// 0.46 M particles on 64^3, with the clearing and the normalisation: the
// advection stage of a step 0.31 -> 0.22 ms.
template <int ALG>
__global__ void kP2GCells(Geom g, const float* __restrict__ pos, const float* __restrict__ vec,
                          const float* __restrict__ scalar, long long P, float4* acc, float* weight) {
  HFG_FOR(p, P) {
    const float px = pos[3 * p], py = pos[3 * p + 1], pz = pos[3 * p + 2];
    const float4 v = make_float4(vec[3 * p], vec[3 * p + 1], vec[3 * p + 2], scalar[p]);
    if (ALG == P2GSUM) {
      atomicAdd(acc + binCell(g, px, py, pz), v);
      continue;
    }
    Taps t;
    taps<ALG>(g, px, py, pz, t);
    constexpr int n = TapsN<ALG>::n, s = TapsN<ALG>::shift;
#pragma unroll
    for (int z = 0; z < n; ++z)
#pragma unroll
      for (int y = 0; y < n; ++y)
#pragma unroll
        for (int x = 0; x < n; ++x) {
          const float w = t.w[0][x] * t.w[1][y] * t.w[2][z];
          const long long i = linc(t.base[0] + x + s, t.base[1] + y + s, t.base[2] + z + s, g.r);
          atomicAdd(acc + i, make_float4(w * v.x, w * v.y, w * v.z, w * v.w));
          atomicAdd(weight + i, w);
        }
  }
}
cudaError_t launchP2GCells(const Geom& g, int alg, const float* pos, const float* vec, const float* scalar, long long P,
                           float4* acc, float* weight, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  const int gr = gridFor(P);
  switch (alg) {
    case LINEAR: kP2GCells<LINEAR><<<gr, kThreads, 0, s>>>(g, pos, vec, scalar, P, acc, weight); break;
    case QUADRATIC: kP2GCells<QUADRATIC><<<gr, kThreads, 0, s>>>(g, pos, vec, scalar, P, acc, weight); break;
    case CUBIC: kP2GCells<CUBIC><<<gr, kThreads, 0, s>>>(g, pos, vec, scalar, P, acc, weight); break;
    case P2GSUM: kP2GCells<P2GSUM><<<gr, kThreads, 0, s>>>(g, pos, vec, scalar, P, acc, weight); break;
    default: break;
  }
  return cudaGetLastError();
}
__global__ void kNormalizeCells(long long n, const float4* __restrict__ acc, const float* __restrict__ weight,
                                float* __restrict__ o0, float* __restrict__ o1, float* __restrict__ o2,
                                float* __restrict__ o3) {
  HFG_FOR(i, n) {
    float4 a = acc[i];
    const float w = weight[i];
    if (w > 0.f) a = make_float4(__fdiv_rn(a.x, w), __fdiv_rn(a.y, w), __fdiv_rn(a.z, w), __fdiv_rn(a.w, w));
    o0[i] = a.x;
    o1[i] = a.y;
    o2[i] = a.z;
    o3[i] = a.w;
  }
}
cudaError_t launchNormalizeCells(long long n, const float4* acc, const float* weight, float* const out[4],
                                 cudaStream_t s) {
  kNormalizeCells<<<gridFor(n), kThreads, 0, s>>>(n, acc, weight, out[0], out[1], out[2], out[3]);
  return cudaGetLastError();
}

// normalizeCCSField (EulerParticlesTool.cu:290-308), the three face grids in one
// launch, fused with the copy kept as the next FLIP "previous grid velocity"
// (MixPICAndFLIP.cpp:135) and the unit-field external-force axpys
// (ExternalForcesSolver.cpp:57-58).
__global__ void kNormalizeFaces(NormalizeFaces f) {
  const int a = blockIdx.y;
  const float2* __restrict__ acc = a == 0 ? f.acc[0] : (a == 1 ? f.acc[1] : f.acc[2]);
  float* __restrict__ out = a == 0 ? f.out[0] : (a == 1 ? f.out[1] : f.out[2]);
  float* __restrict__ copy = a == 0 ? f.copy[0] : (a == 1 ? f.copy[1] : f.copy[2]);
  const float add = a == 0 ? f.add[0] : (a == 1 ? f.add[1] : f.add[2]);
  const float add2 = a == 0 ? f.add2[0] : (a == 1 ? f.add2[1] : f.add2[2]);
  const long long n = a == 0 ? f.n[0] : (a == 1 ? f.n[1] : f.n[2]);
  HFG_FOR(i, n) {
    const float2 w = acc[i];
    float v = w.y > 0.f ? __fdiv_rn(w.x, w.y) : w.x;
    if (copy) copy[i] = v;
    if (f.doAdd) v = __fadd_rn(add, v);
    if (f.doAdd2) v = __fadd_rn(add2, v);
    out[i] = v;
  }
}
cudaError_t launchNormalizeFaces(const NormalizeFaces& f, cudaStream_t s) {
  kNormalizeFaces<<<dim3(gridFor(std::max({f.n[0], f.n[1], f.n[2]})), 3), kThreads, 0, s>>>(f);
  return cudaGetLastError();
}
__global__ void kNormalize(long long n, const float2* __restrict__ acc, float* __restrict__ out) {
  HFG_FOR(i, n) {
    const float2 a = acc[i];
    out[i] = a.y > 0.f ? __fdiv_rn(a.x, a.y) : a.x;
  }
}
cudaError_t launchNormalize(long long n, const float2* acc, float* out, cudaStream_t s) {
  kNormalize<<<gridFor(n), kThreads, 0, s>>>(n, acc, out);
  return cudaGetLastError();
}

template <int ALG>
__global__ void kG2PFace(Geom g, ConstFaceField f, const float* __restrict__ pos, long long P, float* __restrict__ out) {
  HFG_FOR(p, P) {
    float px = pos[3 * p], py = pos[3 * p + 1], pz = pos[3 * p + 2];
#pragma unroll
    for (int a = 0; a < 3; ++a) out[3 * p + a] = g2p<ALG>(f.c[a], faceGeom(g, a), px, py, pz);
  }
}
// LINEAR: one sampler (weights and base indices of each axis formed once, with
// a reciprocal) serves the three components, 32-bit indices.  7.6 M particles
// on 160^3: 173 -> 139 us, 134 with unchecked samples (the check stands between
// the components' loads; one for all three, which keeps or makes again what the
// weighted sums need, took 153 to 193).
template <typename I>
__global__ void kG2PFaceLinear(const __grid_constant__ LerpGrid lg, ConstFaceField f, const float* __restrict__ pos, long long P,
                               float* __restrict__ out) {
  HFG_FOR_T(I, p, P) {
    const LerpSampler fs(lg, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2]);
    float v[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = fs.sample<true>(lg, a, f.c[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) out[3 * p + a] = v[a];
  }
}
cudaError_t launchG2PFace(const Geom& g, int alg, ConstFaceField f, const float* pos, long long P, float* out,
                          cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  int gr = gridFor(P);
  switch (alg) {
    case LINEAR:
      if (index32(P)) kG2PFaceLinear<int><<<gr, kThreads, 0, s>>>(makeLerpGrid(g), f, pos, P, out);
      else kG2PFaceLinear<long long><<<gr, kThreads, 0, s>>>(makeLerpGrid(g), f, pos, P, out);
      break;
    case QUADRATIC: kG2PFace<QUADRATIC><<<gr, kThreads, 0, s>>>(g, f, pos, P, out); break;
    case CUBIC: kG2PFace<CUBIC><<<gr, kThreads, 0, s>>>(g, f, pos, P, out); break;
    case G2PNEAREST: kG2PFace<G2PNEAREST><<<gr, kThreads, 0, s>>>(g, f, pos, P, out); break;
    default: return cudaMemsetAsync(out, 0, sizeof(float) * 3 * P, s);  // P2GSUM: G2P writes 0 (:223)
  }
  return cudaGetLastError();
}

template <int ALG>
__global__ void kG2PCell(Geom g, const float* __restrict__ f, const float* __restrict__ pos, long long P,
                         float* __restrict__ out, int span, int comp) {
  HFG_FOR(p, P) out[span * p + comp] = g2p<ALG>(f, g, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2]);
}
cudaError_t launchG2PCell(const Geom& g, int alg, const float* f, const float* pos, long long P, float* out, int span,
                          int comp, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  int gr = gridFor(P);
  switch (alg) {
    case LINEAR: kG2PCell<LINEAR><<<gr, kThreads, 0, s>>>(g, f, pos, P, out, span, comp); break;
    case QUADRATIC: kG2PCell<QUADRATIC><<<gr, kThreads, 0, s>>>(g, f, pos, P, out, span, comp); break;
    case CUBIC: kG2PCell<CUBIC><<<gr, kThreads, 0, s>>>(g, f, pos, P, out, span, comp); break;
    case G2PNEAREST: kG2PCell<G2PNEAREST><<<gr, kThreads, 0, s>>>(g, f, pos, P, out, span, comp); break;
    default: break;
  }
  return cudaGetLastError();
}

__global__ void kSampleFace(Geom g, ConstFaceField f, const float* __restrict__ pos, long long M, float* __restrict__ out) {
  HFG_FOR(i, M) {
    float v[3];
    sampleFace(f, g, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], v);
    out[3 * i] = v[0]; out[3 * i + 1] = v[1]; out[3 * i + 2] = v[2];
  }
}
cudaError_t launchSampleFace(const Geom& g, ConstFaceField f, const float* pos, long long M, float* out, cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  kSampleFace<<<gridFor(M), kThreads, 0, s>>>(g, f, pos, M, out);
  return cudaGetLastError();
}
__global__ void kSampleCell(Geom g, const float* __restrict__ f, const float* __restrict__ pos, long long M,
                            float* __restrict__ out) {
  HFG_FOR(i, M) out[i] = trilerp(f, g, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]);
}
cudaError_t launchSampleCell(const Geom& g, const float* f, const float* pos, long long M, float* out, cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  kSampleCell<<<gridFor(M), kThreads, 0, s>>>(g, f, pos, M, out);
  return cudaGetLastError();
}

// ===========================================================================
// Semi-Lagrangian advection (SemiLagrangian.cpp:135-347): back-trace each
// face / cell centre through `vel` with RK1/2/3, then sample the source field
// there.  The position fields and the nine axpys of the reference are fused
// into one pass per output grid.
// ===========================================================================
__device__ inline void axpyPt(float a, const float v[3], float p[3]) {
  if (fabsf(a) < FLT_EPSILON) return;  // plusAlphaX skip
#pragma unroll
  for (int k = 0; k < 3; ++k) p[k] = fmaf(a, v[k], p[k]);
}

// SAMP 0 and -1: trilinear, plain and CHECKED; 1 to 4: the cubic samplers
constexpr int kChecked = -1;
template <int SAMP>
__device__ inline void sampleVel(ConstFaceField vel, const Geom& g, const LerpGrid& lg, float px, float py, float pz,
                                 float v[3]) {
  if (SAMP <= 0) {
    const LerpSampler fs(lg, px, py, pz);
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = fs.sample<SAMP == kChecked>(lg, a, vel.c[a]);
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = cubicSample<SAMP>(vel.c[a], faceGeom(g, a), px, py, pz);
  }
}

// CSemiLagrangian::backTrace (SemiLagrangian.cpp:188-347); every velocity
// sample uses the advection's sampling algorithm.
template <int SAMP>
__device__ inline void backTrace(ConstFaceField vel, const Geom& g, const LerpGrid& lg, float dt, int acc, const float in[3], float out[3]) {
  float v0[3], v1[3], v2[3], mid[3], tf[3];
  out[0] = in[0]; out[1] = in[1]; out[2] = in[2];
  sampleVel<SAMP>(vel, g, lg, in[0], in[1], in[2], v0);
  if (acc == 0) {
    axpyPt(-dt, v0, out);
    return;
  }
  mid[0] = in[0]; mid[1] = in[1]; mid[2] = in[2];
  axpyPt(-0.5f * dt, v0, mid);
  sampleVel<SAMP>(vel, g, lg, mid[0], mid[1], mid[2], v1);
  if (acc == 1) {
    axpyPt(-dt, v1, out);
    return;
  }
  tf[0] = in[0]; tf[1] = in[1]; tf[2] = in[2];
  axpyPt(-0.75f * dt, v1, tf);
  sampleVel<SAMP>(vel, g, lg, tf[0], tf[1], tf[2], v2);
  axpyPt(-(float)(2.0 / 9.0) * dt, v0, out);
  axpyPt(-(float)(3.0 / 9.0) * dt, v1, out);
  axpyPt(-(float)(4.0 / 9.0) * dt, v2, out);
}

// The passes run over the planes of their grid (the face axis in blockIdx.z), a
// thread walking zPer planes of one column (they share most corner lines), its
// cell found with one 32-bit division.  Against 64-bit divisions, a
// sequential loop over the axes, two floors per coordinate and weighted sums:
// 375 -> 256 us (128^3, RK3, faces and one cell field).
__device__ __forceinline__ float slLerp(const LerpGrid& lg, int a, const float* __restrict__ f, const float q[3]) {
  const LerpSampler fs(lg, q[0], q[1], q[2]);
  // a is the block's: three forms with constant index selection
  return a == 0 ? fs.sample<false>(lg, 0, f) : (a == 1 ? fs.sample<false>(lg, 1, f) : fs.sample<false>(lg, 2, f));
}
// A point whose linear result is not finite, again with checked samples (a sample
// of the velocity that is not finite makes the result so): component a of a face
// field, or a cell field (3).  A thread goes over its points again for it, and
// the blocks are held to the registers that the first pass needs: 128^3, RK3,
// 260 us; with every sample checked 300, with this called as the point is made
// 273, without any check 258.
__device__ __noinline__ float slChecked(LerpGrid lg, ConstFaceField vel, int acc, float dt, float px, float py, float pz,
                                         int a, const float* f) {
  const float p[3] = {px, py, pz};
  float q[3];
  backTrace<kChecked>(vel, Geom{}, lg, dt, acc, p, q);
  return LerpSampler(lg, q[0], q[1], q[2]).sample<true>(lg, a, f);
}
// SemiLagrangian.cpp:60-97 sample points: entry (x, y, z) of the faces of axis
// a, or of the cells (3)
__device__ __forceinline__ void slPoint(const Geom& g, int a, int x, int y, int z, float p[3]) {
  const float fx = a == 0 ? (float)x : __fadd_rn((float)x, 0.5f), fy = a == 1 ? (float)y : __fadd_rn((float)y, 0.5f),
              fz = a == 2 ? (float)z : __fadd_rn((float)z, 0.5f);
  p[0] = __fadd_rn(__fmul_rn(fx, g.hx), g.ox);
  p[1] = __fadd_rn(__fmul_rn(fy, g.hy), g.oy);
  p[2] = __fadd_rn(__fmul_rn(fz, g.hz), g.oz);
}
constexpr int kSLThreads = 128;
// the planes of this thread: runs of zPer, gridDim.y of them apart
__device__ __forceinline__ int slFirst(int zPer) { return blockIdx.y * zPer; }
__device__ __forceinline__ int slNext(int z, int zPer) {
  return (z + 1) % zPer ? z + 1 : z + 1 + ((int)gridDim.y - 1) * zPer;
}
template <int SAMP>
__global__ void __launch_bounds__(kSLThreads, SAMP == 0 ? 8 : 1) kSLFace(Geom g, const __grid_constant__ LerpGrid lg, int zPer, int acc, float dt, ConstFaceField vel, ConstFaceField in, FaceField out, float ax,
                        float ay, float az, int doAdd, float bx, float by, float bz, int doAdd2) {
  const int a = blockIdx.z;
  const unsigned nx = (unsigned)(g.r.x + (a == 0)), ny = (unsigned)(g.r.y + (a == 1)), plane = nx * ny;
  const int nz = g.r.z + (a == 2);
  const float add = a == 0 ? ax : (a == 1 ? ay : az), add2 = a == 0 ? bx : (a == 1 ? by : bz);
  const float* __restrict__ src = a == 0 ? in.c[0] : (a == 1 ? in.c[1] : in.c[2]);
  float* __restrict__ dst = a == 0 ? out.c[0] : (a == 1 ? out.c[1] : out.c[2]);
  bool bad = false;
  HFG_FOR_U(i, plane) {
    const unsigned y = i / nx, x = i - y * nx;
    for (int z = slFirst(zPer); z < nz; z = slNext(z, zPer)) {
      float p[3], q[3];
      slPoint(g, a, x, y, z, p);
      backTrace<SAMP>(vel, g, lg, dt, acc, p, q);
      float v = SAMP == 0 ? slLerp(lg, a, src, q) : sampleAlg<SAMP>(src, faceGeom(g, a), q[0], q[1], q[2]);
      if (doAdd) v = __fadd_rn(add, v);
      if (doAdd2) v = __fadd_rn(add2, v);
      dst[(unsigned)z * plane + i] = v;
      if (SAMP == 0) bad |= notFinite(v);
    }
  }
  if (!bad) return;
  HFG_FOR_U(i, plane) {
    const unsigned y = i / nx, x = i - y * nx;
    for (int z = slFirst(zPer); z < nz; z = slNext(z, zPer)) {
      if (!notFinite(dst[(unsigned)z * plane + i])) continue;
      float p[3];
      slPoint(g, a, x, y, z, p);
      float v = slChecked(lg, vel, acc, dt, p[0], p[1], p[2], a, src);
      if (doAdd) v = __fadd_rn(add, v);
      if (doAdd2) v = __fadd_rn(add2, v);
      dst[(unsigned)z * plane + i] = v;
    }
  }
}
namespace {
// Runs of four planes where that leaves a thousand threads to an SM, else
// shorter ones (one plane on the small grids).
int slPlanes(const Dim3i& r) {
  return (int)std::max(1LL, std::min(4LL, (long long)(r.x + 1) * (r.y + 1) * (r.z + 1) / (numSMs() * 1024LL)));
}
// blocks over a plane of at most (nx + 1) (ny + 1) entries and runs of zPer planes
dim3 planeGrid(const Dim3i& r, int threads, int axes, int zPer) {
  const long long plane = (long long)(r.x + 1) * (r.y + 1);
  return dim3((unsigned)std::min<long long>((plane + threads - 1) / threads, 1 << 20),
              (unsigned)std::min((r.z + zPer) / zPer, 65535), axes);
}
}  // namespace
cudaError_t launchSLFace(const Geom& g, int acc, float dt, ConstFaceField vel, ConstFaceField in, FaceField out,
                         const float add[3], int doAdd, const float add2[3], int doAdd2, cudaStream_t s,
                         int sampling) {
#define HFG_SL_FACE(S)                                                                                              \
  kSLFace<S><<<planeGrid(g.r, kSLThreads, 3, slPlanes(g.r)), kSLThreads, 0, s>>>(g, makeLerpGrid(g), slPlanes(g.r), acc, dt, vel, in, out, add[0], add[1], add[2], doAdd, add2[0], \
                                                    add2[1], add2[2], doAdd2)
  switch (sampling) {
    case 1: HFG_SL_FACE(1); break;
    case 2: HFG_SL_FACE(2); break;
    case 3: HFG_SL_FACE(3); break;
    case 4: HFG_SL_FACE(4); break;
    default: HFG_SL_FACE(0);
  }
#undef HFG_SL_FACE
  return cudaGetLastError();
}

struct CellFields {
  const float* in[4];
  float* out[4];
};
template <int SAMP>
__global__ void __launch_bounds__(kSLThreads, SAMP == 0 ? 8 : 1) kSLCell(Geom g, const __grid_constant__ LerpGrid lg, int zPer, int acc, float dt, ConstFaceField vel, CellFields cf, int nf) {
  const unsigned nx = (unsigned)g.r.x, plane = nx * (unsigned)g.r.y;
  bool bad = false;
  HFG_FOR_U(i, plane) {
    const unsigned y = i / nx, x = i - y * nx;
    for (int z = slFirst(zPer); z < g.r.z; z = slNext(z, zPer)) {
      float p[3], q[3];
      slPoint(g, 3, x, y, z, p);
      backTrace<SAMP>(vel, g, lg, dt, acc, p, q);
      const unsigned c = (unsigned)z * plane + i;
      if (SAMP == 0) {
        const LerpSampler fs(lg, q[0], q[1], q[2]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < nf) {
            const float v = fs.sample<false>(lg, 3, cf.in[k]);
            cf.out[k][c] = v;
            bad |= notFinite(v);
          }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < nf) cf.out[k][c] = sampleAlg<SAMP>(cf.in[k], g, q[0], q[1], q[2]);
      }
    }
  }
  if (!bad) return;
  HFG_FOR_U(i, plane) {
    const unsigned y = i / nx, x = i - y * nx;
    for (int z = slFirst(zPer); z < g.r.z; z = slNext(z, zPer)) {
      const unsigned c = (unsigned)z * plane + i;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k >= nf || !notFinite(cf.out[k][c])) continue;
        float p[3];
        slPoint(g, 3, x, y, z, p);
        cf.out[k][c] = slChecked(lg, vel, acc, dt, p[0], p[1], p[2], 3, cf.in[k]);
      }
    }
  }
}
cudaError_t launchSLCell(const Geom& g, int acc, float dt, ConstFaceField vel, const float* const* in, float* const* out,
                         int nfields, cudaStream_t s, int sampling) {
  CellFields cf{};
  for (int k = 0; k < nfields && k < 4; ++k) { cf.in[k] = in[k]; cf.out[k] = out[k]; }
  const int nf = nfields < 4 ? nfields : 4;
  const int zPer = slPlanes(g.r);
  const dim3 grid = planeGrid(g.r, kSLThreads, 1, zPer);
  const LerpGrid lg = makeLerpGrid(g);
  switch (sampling) {
    case 1: kSLCell<1><<<grid, kSLThreads, 0, s>>>(g, lg, zPer, acc, dt, vel, cf, nf); break;
    case 2: kSLCell<2><<<grid, kSLThreads, 0, s>>>(g, lg, zPer, acc, dt, vel, cf, nf); break;
    case 3: kSLCell<3><<<grid, kSLThreads, 0, s>>>(g, lg, zPer, acc, dt, vel, cf, nf); break;
    case 4: kSLCell<4><<<grid, kSLThreads, 0, s>>>(g, lg, zPer, acc, dt, vel, cf, nf); break;
    default: kSLCell<0><<<grid, kSLThreads, 0, s>>>(g, lg, zPer, acc, dt, vel, cf, nf);
  }
  return cudaGetLastError();
}

// Sampling of a cell-centred scalar grid (FieldMathTool.cu:470-573) or of
// the three face grids (:783-1128) at n points with an ESamplingAlgorithm.
template <int SAMP>
__global__ void kSampleAlg(Geom g, int face, ConstFaceField f, const float* __restrict__ pos, long long n,
                           float* __restrict__ out) {
  HFG_FOR(i, n) {
    const float px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
    if (face) {
#pragma unroll
      for (int a = 0; a < 3; ++a) out[3 * i + a] = sampleAlg<SAMP>(f.c[a], faceGeom(g, a), px, py, pz);
    } else {
      out[i] = sampleAlg<SAMP>(f.c[0], g, px, py, pz);
    }
  }
}
cudaError_t launchSampleAlg(const Geom& g, int face, ConstFaceField f, const float* pos, long long n, int sampling,
                            float* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (sampling) {
    case 1: kSampleAlg<1><<<gridFor(n), kThreads, 0, s>>>(g, face, f, pos, n, out); break;
    case 2: kSampleAlg<2><<<gridFor(n), kThreads, 0, s>>>(g, face, f, pos, n, out); break;
    case 3: kSampleAlg<3><<<gridFor(n), kThreads, 0, s>>>(g, face, f, pos, n, out); break;
    case 4: kSampleAlg<4><<<gridFor(n), kThreads, 0, s>>>(g, face, f, pos, n, out); break;
    default: kSampleAlg<0><<<gridFor(n), kThreads, 0, s>>>(g, face, f, pos, n, out);
  }
  return cudaGetLastError();
}

__global__ void kAddConst(long long n, float* __restrict__ v, float a) {
  HFG_FOR(i, n) v[i] = __fadd_rn(a, v[i]);
}
cudaError_t launchAddConst(long long n, float* v, float a, cudaStream_t s) {
  kAddConst<<<gridFor(n), kThreads, 0, s>>>(n, v, a);
  return cudaGetLastError();
}

// ===========================================================================
// Self-test of the bounded waits.  Every wait of the TMA-fed and cooperative
// kernels is bounded: past its limit it records an error and returns, so the
// context stays usable.  These two kernels make the shared wait helpers run
// out on purpose, on conditions that nothing will ever satisfy, without any
// fault: an mbarrier phase expecting bytes no copy will deliver, and a grid
// barrier expecting one arrival more than the grid has blocks.
// ===========================================================================
__global__ void kSelftestMbarrier(unsigned long long waitNs, int* out) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbarInit(&bar, 1);
    mbarFenceInit();
    mbarExpectTx(&bar, 16);  // this thread arrives; 16 bytes stay pending for good
    const bool done = mbarWait(&bar, 0, globalNs() + waitNs);
    out[0] = done ? 0 : 1;
  }
}
__global__ void kSelftestGridBarrier(unsigned* words, int* out) {
  // words: error, then three mailboxes (the third block does not exist)
  gridArrive(words + 1, 1u, gridDim.x + 1);
  const bool ok = gridWait(words + 1, 1u, words, gridDim.x + 1);
  if (threadIdx.x == 0 && blockIdx.x == 0) out[1] = ok ? 0 : 1;
}
cudaError_t launchSelftestWaits(unsigned long long waitNs, unsigned* words, int* out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(words, 0, 10 * sizeof(unsigned), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0xff, 2 * sizeof(int), s);
  if (e != cudaSuccess) return e;
  kSelftestMbarrier<<<1, 32, 0, s>>>(waitNs, out);
  kSelftestGridBarrier<<<2, 32, 0, s>>>(words, out);
  return cudaGetLastError();
}

}  // namespace hfg
