// hfg_pressure.cu -- the matrix-free pressure Poisson system and its CG on
// sm_100a.
//
// The reference stores A as 4 floats per cell (buildPressureMatrixA,
// EulerSolverTool.cu:58-126) and runs CG with cuBLAS calls and three blocking
// host reads per iteration (CuMatrixFreePCG.cpp:22-65).  Here A is rebuilt in
// registers from a 16-bit stencil code per cell, every CG iteration is two
// kernels with FP64 block reductions finished by the last block (no host
// round trip), or, where the fluid fits the GPU's shared memory, a whole solve
// is one launch (the resident CG below), and the stencil kernels are 2.5-D: a 32x8 thread tile marches
// along z keeping the below / current / above planes in registers, so the z
// neighbours cost no extra loads and no division is needed for indexing.
#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "hfg_kernels.h"

namespace hfg {

namespace {
constexpr int TX = 32, TY = 8;

struct CgGrid {
  dim3 grid, block;
  int zPer;
};

// Enough blocks to fill every SM several times over, each marching >= 4 planes.
CgGrid cgGrid(const Dim3i& r) {
  CgGrid g;
  g.block = dim3(TX, TY, 1);
  int bx = (r.x + TX - 1) / TX, by = (r.y + TY - 1) / TY;
  long long tiles = (long long)bx * by;
  long long want = (long long)numSMs() * 16;
  int zc = (int)std::max<long long>(1, (want + tiles - 1) / tiles);
  zc = std::min(zc, std::max(1, r.z / 4));
  g.zPer = (r.z + zc - 1) / zc;
  zc = (r.z + g.zPer - 1) / g.zPer;
  g.grid = dim3(bx, by, zc);
  return g;
}

__device__ __forceinline__ bool nbFluid(Code k, int d) { return (k >> (7 + d)) & 1; }

// Diagonal in the reference's accumulation order (EulerSolverTool.cu:85-120).
__device__ __forceinline__ float diagOf(Code k, float sx, float sy, float sz) {
  if (!(k & 1)) return 1.f;
  float d = 0.f;
  if (k & 2) d += sx;
  if (k & 4) d += sx;
  if (k & 8) d += sy;
  if (k & 16) d += sy;
  if (k & 32) d += sz;
  if (k & 64) d += sz;
  return d;
}

// PC: 0 identity, 1 Jacobi, 2 z supplied by the caller (multigrid)
template <int PC>
__device__ __forceinline__ float precondZ(Code k, float rv, float sx, float sy, float sz) {
  return PC == 1 ? __fdiv_rn(rv, diagOf(k, sx, sy, sz)) : rv;
}

__device__ inline bool cgStop(const CgState* st, double rr) {
  double rn = sqrt(rr);
  if (st->tolMode == 0) return sqrt(rn) < st->tol;  // CuMatrixFreePCG.cpp:28,51
  double bn = sqrt(st->bb);
  return bn == 0.0 || rn / bn < st->tol;
}

// (A v)_c for a fluid cell given v at the centre and at its six neighbours
// (fdmMatrixVectorMul, EulerSolverTool.cu:219-226: products in float, sum in
// double as the reference's `: 0.0` ternaries make it).
__device__ __forceinline__ float applyRow(Code k, float sx, float sy, float sz, float vc, float vl, float vr, float vd,
                                          float vu, float vb, float vf) {
  if (!(k & 1)) return vc;
  double acc = (double)__fmul_rn(diagOf(k, sx, sy, sz), vc);
  if (nbFluid(k, 0)) acc += (double)__fmul_rn(-sx, vl);
  if (nbFluid(k, 1)) acc += (double)__fmul_rn(-sx, vr);
  if (nbFluid(k, 2)) acc += (double)__fmul_rn(-sy, vd);
  if (nbFluid(k, 3)) acc += (double)__fmul_rn(-sy, vu);
  if (nbFluid(k, 4)) acc += (double)__fmul_rn(-sz, vb);
  if (nbFluid(k, 5)) acc += (double)__fmul_rn(-sz, vf);
  return (float)acc;
}
}  // namespace


// ---------------------------------------------------------------------------
__global__ void kStencilCode(Dim3i r, int px, const uint8_t* __restrict__ mk, Code* __restrict__ code,
                             CgCode* __restrict__ cgc, int zPer) {
  int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
  if (x >= px || y >= r.y) return;
  int z0 = blockIdx.z * zPer, z1 = min(z0 + zPer, r.z);
  long long plane = (long long)r.x * r.y;
  for (int z = z0; z < z1; ++z) {
    long long c = (long long)z * plane + (long long)y * r.x + x;
    long long o = ((long long)z * r.y + y) * px + x;
    Code k = 0;
    if (x < r.x && mk[c] == kFluid) {
      k = 1;
      const bool in[6] = {x > 0, x + 1 < r.x, y > 0, y + 1 < r.y, z > 0, z + 1 < r.z};
      const long long d6[6] = {-1, 1, -(long long)r.x, (long long)r.x, -plane, plane};
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if (!in[d]) continue;
        uint8_t m = mk[c + d6[d]];
        if (m != kSolid) k |= (Code)(1u << (1 + d));
        if (m == kFluid) k |= (Code)(1u << (7 + d));
      }
    }
    code[o] = k;
    if (cgc) cgc[o] = (CgCode)(k & 0x7f);
  }
}
cudaError_t launchStencilCode(const Dim3i& r, int px, const uint8_t* markers, Code* code, cudaStream_t s,
                              CgCode* cgc) {
  CgGrid g = cgGrid(Dim3i{px, r.y, r.z});
  kStencilCode<<<g.grid, g.block, 0, s>>>(r, px, markers, code, cgc, g.zPer);
  return cudaGetLastError();
}

// The reference's stored matrix [diag, +x, +y, +z] (EulerSolverTool.cu:58-126),
// bit-exact: used by the operator API and its tests only.
__global__ void kMatrixA(Dim3i r, float sx, float sy, float sz, const Code* __restrict__ code, float* __restrict__ A) {
  long long n = r.size();
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    Code k = code[c];
    float a0 = diagOf(k, sx, sy, sz), a1 = 0.f, a2 = 0.f, a3 = 0.f;
    if (k & 1) {
      if (nbFluid(k, 1)) a1 = -sx;
      if (nbFluid(k, 3)) a2 = -sy;
      if (nbFluid(k, 5)) a3 = -sz;
    }
    A[4 * c] = a0; A[4 * c + 1] = a1; A[4 * c + 2] = a2; A[4 * c + 3] = a3;
  }
}
cudaError_t launchMatrixA(const Dim3i& r, float sx, float sy, float sz, const Code* code, float* A, cudaStream_t s) {
  int blocks = (int)std::min<long long>((r.size() + 255) / 256, (long long)numSMs() * 16);
  kMatrixA<<<blocks, 256, 0, s>>>(r, sx, sy, sz, code, A);
  return cudaGetLastError();
}

// y = A x (fdmMatrixVectorMulInvoker, EulerSolverTool.cu:706-720)
__global__ void kApplyA(Dim3i r, float sx, float sy, float sz, const Code* __restrict__ code,
                        const float* __restrict__ xin, float* __restrict__ y, int zPer) {
  int x = blockIdx.x * TX + threadIdx.x, yy = blockIdx.y * TY + threadIdx.y;
  if (x >= r.x || yy >= r.y) return;
  int z0 = blockIdx.z * zPer, z1 = min(z0 + zPer, r.z);
  long long plane = (long long)r.x * r.y;
  long long c = (long long)z0 * plane + (long long)yy * r.x + x;
  float below = z0 > 0 ? xin[c - plane] : 0.f, cur = xin[c];
  for (int z = z0; z < z1; ++z, c += plane) {
    float above = z + 1 < r.z ? xin[c + plane] : 0.f;
    Code k = code[c];
    float vl = x > 0 ? xin[c - 1] : 0.f, vr = x + 1 < r.x ? xin[c + 1] : 0.f;
    float vd = yy > 0 ? xin[c - r.x] : 0.f, vu = yy + 1 < r.y ? xin[c + r.x] : 0.f;
    y[c] = applyRow(k, sx, sy, sz, cur, vl, vr, vd, vu, below, above);
    below = cur;
    cur = above;
  }
}
cudaError_t launchApplyA(const Dim3i& r, float sx, float sy, float sz, const Code* code, const float* x, float* y,
                         cudaStream_t s) {
  CgGrid g = cgGrid(r);
  kApplyA<<<g.grid, g.block, 0, s>>>(r, sx, sy, sz, code, x, y, g.zPer);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// RHS: divergence (FieldMathTool.cu:370-395) + solid terms
// (EulerSolverTool.cu:128-197), fused with the CG set-up of
// CuMatrixFreePCG.cpp:22-37 (x0 = 0 so r = b).
// b of one cell: -div u plus the solid-face terms (FieldMathTool.cu:370-395,
// EulerSolverTool.cu:128-197), in the reference's operation order; 0 for
// non-fluid cells.
__device__ __forceinline__ float rhsAt(const Geom& g, const ConstFaceField& v, const ConstFaceField& svArr,
                                       const SolidVelTable& svTab, const uint8_t* __restrict__ mk, int x, int y,
                                       int z) {
  const Dim3i R = g.r;
  const long long plane = (long long)R.x * R.y;
  const long long c = (long long)z * plane + (long long)y * R.x + x;
  if (mk[c] != kFluid) return 0.f;
  const float ix = 1.0f / g.hx, iy = 1.0f / g.hy, iz = 1.0f / g.hz;
  const long long fxRow = R.x + 1, fxPlane = (long long)(R.x + 1) * R.y;
  const long long fyPlane = (long long)R.x * (R.y + 1);
  long long uL = (long long)z * fxPlane + (long long)y * fxRow + x, uR = uL + 1;
  long long vD = (long long)z * fyPlane + (long long)y * R.x + x, vU = vD + R.x;
  long long wB = c, wF = c + plane;
  float L = v.c[0][uL], Rr = v.c[0][uR], D = v.c[1][vD], U = v.c[1][vU], B = v.c[2][wB], F = v.c[2][wF];
  float div = __fadd_rn(__fadd_rn(__fdiv_rn(__fsub_rn(Rr, L), g.hx), __fdiv_rn(__fsub_rn(U, D), g.hy)),
                        __fdiv_rn(__fsub_rn(F, B), g.hz));
  float b = -div;
  uint8_t me = svTab.solidIdx ? svTab.solidIdx[c] : 0;
  auto sv = [&](int axis, long long f, long long nb, bool nbIsHi) -> float {
    if (svArr.c[0]) return svArr.c[axis][f];
    uint8_t o = svTab.solidIdx[nb];
    return nbIsHi ? solidFaceVel(svTab, me, o, axis) : solidFaceVel(svTab, o, me, axis);
  };
  long long cl = x > 0 ? c - 1 : c, cr = x + 1 < R.x ? c + 1 : c;
  long long cd = y > 0 ? c - R.x : c, cu = y + 1 < R.y ? c + R.x : c;
  long long cb = z > 0 ? c - plane : c, cf = z + 1 < R.z ? c + plane : c;
  if (mk[cl] == kSolid) b = __fsub_rn(b, __fmul_rn(ix, __fsub_rn(L, sv(0, uL, cl, false))));
  if (mk[cr] == kSolid) b = __fadd_rn(b, __fmul_rn(ix, __fsub_rn(Rr, sv(0, uR, cr, true))));
  if (mk[cd] == kSolid) b = __fsub_rn(b, __fmul_rn(iy, __fsub_rn(D, sv(1, vD, cd, false))));
  if (mk[cu] == kSolid) b = __fadd_rn(b, __fmul_rn(iy, __fsub_rn(U, sv(1, vU, cu, true))));
  if (mk[cb] == kSolid) b = __fsub_rn(b, __fmul_rn(iz, __fsub_rn(B, sv(2, wB, cb, false))));
  if (mk[cf] == kSolid) b = __fadd_rn(b, __fmul_rn(iz, __fsub_rn(F, sv(2, wF, cf, true))));
  return b;
}

// Divergence residual of a projected field: sum of b^2 over the fluid cells
// (FP64, last-block reduction) and max |b| (ordered-bits atomic max).
__global__ void kDivergenceNorm(Geom g, ConstFaceField v, ConstFaceField svArr, SolidVelTable svTab,
                                const uint8_t* __restrict__ mk, double* partials, unsigned* ticket,
                                double* sumOut, unsigned* maxBits) {
  double s2 = 0.0, dummy = 0.0;
  float mx = 0.f;
  const long long n = g.r.size();
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(c % g.r.x);
    const long long t = c / g.r.x;
    const int y = (int)(t % g.r.y), z = (int)(t / g.r.y);
    float b = rhsAt(g, v, svArr, svTab, mk, x, y, z);
    s2 += (double)b * (double)b;
    mx = fmaxf(mx, fabsf(b));
  }
  mx = warpMaxF(mx);
  if ((threadIdx.x & 31) == 0) atomicMax(maxBits, __float_as_uint(mx));
  if (gridSum2(s2, dummy, partials, ticket) && flatTid() == 0) {
    *sumOut = s2;
    *ticket = 0;
  }
}

// The final residual check of a pressure solve, in FP64 on the GPU:
// ||b - A x||^2 and ||b||^2 over the fluid cells.  b is recomputed from the
// unprojected velocity (rhsAt, the reference's operation order), the entries
// of A are the FP32 system's scales promoted to FP64 (fdmMatrixVectorMul,
// EulerSolverTool.cu:199-227, with diagonal and neighbour terms from the
// stencil code) and x is read as stored (FP32 or FP64).  The CG's own
// recurrence residual drifts from this once FP32 round-off builds up.
__global__ void kTrueResidual(Geom g, ConstFaceField v, SolidVelTable svTab, const uint8_t* __restrict__ mk,
                              const Code* __restrict__ code, const void* __restrict__ xv, int xDouble, double sx,
                              double sy, double sz, double* partials, unsigned* ticket, double* out) {
  double rr = 0.0, bb = 0.0;
  const Dim3i R = g.r;
  const long long px = cgPitch(R.x), pl = px * R.y;
  const ConstFaceField none{{nullptr, nullptr, nullptr}};
  auto X = [&](long long i) -> double {
    return xDouble ? ((const double*)xv)[i] : (double)((const float*)xv)[i];
  };
  const long long n = R.size();
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    if (mk[c] != kFluid) continue;
    const int x = (int)(c % R.x);
    const long long t = c / R.x;
    const int y = (int)(t % R.y), z = (int)(t / R.y);
    const double b = (double)rhsAt(g, v, none, svTab, mk, x, y, z);
    const long long o = ((long long)z * R.y + y) * px + x;
    const Code k = code[o];
    double diag = 0.0;
    if (k & 2) diag += sx;
    if (k & 4) diag += sx;
    if (k & 8) diag += sy;
    if (k & 16) diag += sy;
    if (k & 32) diag += sz;
    if (k & 64) diag += sz;
    double ax = diag * X(o);
    if (nbFluid(k, 0)) ax -= sx * X(o - 1);
    if (nbFluid(k, 1)) ax -= sx * X(o + 1);
    if (nbFluid(k, 2)) ax -= sy * X(o - px);
    if (nbFluid(k, 3)) ax -= sy * X(o + px);
    if (nbFluid(k, 4)) ax -= sz * X(o - pl);
    if (nbFluid(k, 5)) ax -= sz * X(o + pl);
    const double r = b - ax;
    rr += r * r;
    bb += b * b;
  }
  if (gridSum2(rr, bb, partials, ticket) && flatTid() == 0) {
    out[0] = rr;
    out[1] = bb;
    *ticket = 0;
  }
}
cudaError_t launchTrueResidual(const Geom& g, ConstFaceField v, const SolidVelTable& svTab, const uint8_t* markers,
                               const Code* code, const void* x, bool xDouble, float sx, float sy, float sz,
                               double* scratch, unsigned* ticket, double* out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  kTrueResidual<<<divergenceBlocks(), 256, 0, s>>>(g, v, svTab, markers, code, x, xDouble ? 1 : 0, (double)sx,
                                                   (double)sy, (double)sz, scratch, ticket, out);
  return cudaGetLastError();
}

template <int PC>
__global__ void __launch_bounds__(TX* TY) kRhsInit(Geom g, ConstFaceField v, ConstFaceField svArr, SolidVelTable svTab,
                                                   const uint8_t* __restrict__ mk, const Code* __restrict__ code,
                                                   float sAx, float sAy, float sAz, float* __restrict__ bOut,
                                                   float* __restrict__ r, void* __restrict__ xv, int xDouble,
                                                   float* __restrict__ p, double* partials, CgState* st, int zPer) {
  const Dim3i R = g.r;
  const int px = cgPitch(R.x);
  int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
  double bb = 0.0, rzs = 0.0;
  if (x >= R.x && x < px && y < R.y) {  // pitch padding: inert cells
    int z0 = blockIdx.z * zPer, z1 = min(z0 + zPer, R.z);
    for (int z = z0; z < z1; ++z) {
      long long o = ((long long)z * R.y + y) * px + x;
      r[o] = 0.f;
      if (xDouble) ((double*)xv)[o] = 0.0;
      else ((float*)xv)[o] = 0.f;
      p[o] = 0.f;
    }
  }
  if (x < R.x && y < R.y) {
    int z0 = blockIdx.z * zPer, z1 = min(z0 + zPer, R.z);
    const long long plane = (long long)R.x * R.y;
    for (int z = z0; z < z1; ++z) {
      long long c = (long long)z * plane + (long long)y * R.x + x;
      float b = rhsAt(g, v, svArr, svTab, mk, x, y, z);
      if (bOut) bOut[c] = b;
      long long o = ((long long)z * R.y + y) * px + x;
      r[o] = b;
      if (xDouble) ((double*)xv)[o] = 0.0;
      else ((float*)xv)[o] = 0.f;
      p[o] = 0.f;
      float zz = precondZ<PC>(code[o], b, sAx, sAy, sAz);
      bb += (double)b * (double)b;
      rzs += (double)b * (double)zz;
    }
  }
  if (gridSum2(bb, rzs, partials, &st->ticket) && flatTid() == 0) {
    st->bb = bb;
    st->rr = bb;
    st->rz = rzs;
    st->iter = 0;
    st->beta = 0.f;
    st->alpha = 0.f;
    st->done = cgStop(st, bb) || st->maxIter <= 0;  // CuMatrixFreePCG.cpp:28-32
    st->ticket = 0;
  }
}
cudaError_t launchRhsInit(const Geom& gm, ConstFaceField v, ConstFaceField svArr, const SolidVelTable& svTab,
                          const uint8_t* markers, const Code* code, float ax, float ay, float az, float* b, float* r,
                          void* x, bool xDouble, float* p, double* partials, CgState* st, int precond,
                          cudaStream_t s) {
  CgGrid g = cgGrid(cgDims(gm.r));
  const int xd = xDouble ? 1 : 0;
  if (precond == 1)
    kRhsInit<1><<<g.grid, g.block, 0, s>>>(gm, v, svArr, svTab, markers, code, ax, ay, az, b, r, x, xd, p, partials,
                                           st, g.zPer);
  else
    kRhsInit<0><<<g.grid, g.block, 0, s>>>(gm, v, svArr, svTab, markers, code, ax, ay, az, b, r, x, xd, p, partials,
                                           st, g.zPer);
  return cudaGetLastError();
}

cudaError_t launchDivergenceNorm(const Geom& g, ConstFaceField v, const SolidVelTable& svTab,
                                 const uint8_t* markers, double* scratch, unsigned* ticketAndMax, double* sumOut,
                                 cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(ticketAndMax, 0, 2 * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  ConstFaceField none{{nullptr, nullptr, nullptr}};
  kDivergenceNorm<<<divergenceBlocks(), 256, 0, s>>>(g, v, none, svTab, markers, scratch, ticketAndMax, sumOut,
                                                     ticketAndMax + 1);
  return cudaGetLastError();
}

namespace {
// ---------------------------------------------------------------------------
// Fast row of A for the CG: the diagonal and its reciprocal come from a
// 128-entry table per launch, indexed by the whole 7-bit CG code (fluid bit
// and the six "not solid" bits; the entries are summed in the reference's
// order), and the six off-diagonal terms are FP32 FMAs on the neighbour
// values.  The non-fluid codes hold (-1, 1): the Jacobi preconditioner then
// needs no test of the fluid bit (r * 1 = r), and a negative diagonal marks
// a non-fluid cell (a fluid diagonal is a sum of positive scales, or 0).
struct DiagTab {
  float2 e[128];  // (diagonal, its reciprocal)
};

__device__ __forceinline__ void buildDiagTab(DiagTab& t, float sx, float sy, float sz) {
  const int tid = flatTid();
  if (tid < 128) {
    float d = -1.f, inv = 1.f;
    if (tid & 1) {
      d = diagOf((Code)tid, sx, sy, sz);
      inv = d != 0.f ? 1.0f / d : 0.f;
    }
    t.e[tid] = make_float2(d, inv);
  }
}

// Row sum of A at a fluid cell: d vc minus the six off-diagonal terms, d the
// diagonal of the cell's code.  The neighbour values need no masks here.  The
// CG vectors p, r and z are zero at every cell that is not fluid: b is zero
// there, the row of A is the identity, and the Jacobi and multigrid
// preconditioners write zero there, so r -= alpha A p and p = z + beta p keep
// them zero.  The halo outside the grid arrives zero-filled and the pitch
// padding is zero too.  So the only neighbours that add anything are the
// fluid ones, as in the reference's off-diagonal terms, and the sum is the
// masked sum up to the sign of a zero.  At a non-fluid cell the row is the
// identity and every CG vector stays zero for the whole solve (the RHS kernel
// zeroes x, r and p there, and the updates add alpha or beta times zero), so
// the CG kernels neither form the row nor store anything there.
__device__ __forceinline__ float rowSum(float d, float sx, float sy, float sz, float vc, float vl, float vr, float vd,
                                        float vu, float vb, float vf) {
  float q = d * vc;
  q = fmaf(-sx, vl + vr, q);
  q = fmaf(-sy, vd + vu, q);
  q = fmaf(-sz, vb + vf, q);
  return q;
}

template <int PC>
__device__ __forceinline__ float fastZ(float inv, float rv) {
  if (PC != 1) return rv;
  return rv * inv;
}

// ---------------------------------------------------------------------------
// TMA plumbing.  Each CG block owns a 32 x 8 column of the pitched grid and
// marches along z; one elected thread streams the planes ahead of the
// consumers into a ring of shared-memory stages with cp.async.bulk.tensor,
// completion tracked by one mbarrier per stage.  The halo boxes start 4
// floats (8 codes) left of the tile so that every box starts on a 16-byte
// boundary; boxes outside the grid arrive zero-filled.
constexpr int CTX = 32, CTY = 8;     // threads per block (x, y)
constexpr int RY = 2;                // rows per thread: thread (tx, ty) owns rows ty and ty + CTY
constexpr int CTR = CTY * RY;        // 16 tile rows per plane
static_assert(2 * CTR == CTX, "one warp computes both halo columns (one lane per halo cell)");
constexpr int HXF = 4, HXC = 16;     // left pad of the float / code halo boxes (16 bytes)
constexpr int FW = CTX + 2 * HXF;    // 40 floats
constexpr int CW = CTX + 2 * HXC;    // 64 codes
constexpr int FH = CTR + 2;          // 18 rows
constexpr int kDirStages = 4, kUpdStages = 5;
constexpr unsigned long long kWaitNs = 2000000000ull;  // a stage that takes 2 s to land is an error

__device__ __forceinline__ void tmaLoad3(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smemAddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smemAddr(bar))
      : "memory");
}

// Marks the solve failed; the host sees `error` and stops.
__device__ __forceinline__ void cgFail(CgState* st, int code) {
  atomicExch(&st->error, code);
  atomicExch(&st->done, 1);
}

// Blocks that gave up still drain every stage they issued (bounded) before
// the shared memory is released.
template <int S>
__device__ void drainStages(uint64_t* bar, const int* issued, int waited) {
  unsigned long long deadline = globalNs() + kWaitNs;
  for (int i = waited; i < issued[0]; ++i)
    if (!mbarWait(&bar[i % S], (unsigned)((i / S) & 1), deadline)) break;
}

struct __align__(128) DirStage {
  alignas(128) float r[FH][FW];
  alignas(128) float po[FH][FW];
  alignas(128) CgCode code[FH][CW];
};
constexpr unsigned kDirStageBytes = sizeof(float) * FH * FW * 2 + sizeof(CgCode) * FH * CW;

// TX: the pressure iterate x in FP32 (the reference's Real) or FP64.
template <class TX> struct __align__(128) UpdStage {
  alignas(128) float p[FH][FW];
  alignas(128) float r[CTR][CTX];
  alignas(128) TX x[CTR][CTX];
  alignas(128) CgCode code[CTR][CTX];
};
template <class TX>
constexpr unsigned kUpdStageBytes = sizeof(float) * (FH * FW + CTR * CTX) + sizeof(TX) * CTR * CTX + sizeof(CgCode) * CTR * CTX;
template <class TX> constexpr int kUpdStagesT = sizeof(TX) == 8 ? 4 : kUpdStages;  // keeps static shared memory < 48 KB

struct CgLaunch {
  dim3 grid, block;
  int zPer;
};

// The CG schedule of a solve (launchCgSchedule), in one int array:
//   [0, cols)            the lowest plane holding a fluid cell of each tile
//                        column (CTX x CTR cells of the pitched grid, all z),
//   [cols, 2 cols)       the highest (a range no plane meets: no fluid),
//   [2 cols]             the number of work items,
//   [schedItemsOffset)   the items (column, z0, z1, 0): one per CG block, the
//                        fluid planes of the active columns cut into chunks
//                        so that the items about fill one wave of blocks.
// A block past the last item only joins the reductions.  Null: the dense
// grid, block (x, y, z) on tile (x, y) and planes [z zPer, (z + 1) zPer).
static_assert(CTX == kCgTileX && CTR == kCgTileY, "the schedule's tile is the CG kernels' tile");

// A work item that is not a run of planes of a column of this grid (or a
// count beyond the grid) is not used: the block stays idle and the solve
// reports error 4.
__device__ __forceinline__ bool cgBlockWork(const int* sched, const Dim3i& P, int zPer, int& x0, int& y0, int& z0,
                                            int& z1, CgState* st) {
  if (!sched) {
    x0 = blockIdx.x * CTX;
    y0 = blockIdx.y * CTR;
    z0 = blockIdx.z * zPer;
    z1 = min(z0 + zPer, P.z);
    return true;
  }
  x0 = y0 = z0 = z1 = 0;
  const int tilesX = (P.x + CTX - 1) / CTX, cols = tilesX * ((P.y + CTR - 1) / CTR);
  const int n = __ldg(sched + 2 * cols);
  if (n < 0 || n > (int)gridDim.x) {
    if (threadIdx.x == 0 && threadIdx.y == 0) cgFail(st, 4);
    return false;
  }
  if ((int)blockIdx.x >= n) return false;
  const int4 w = __ldg(reinterpret_cast<const int4*>(sched + schedItemsOffset(cols)) + blockIdx.x);
  if (w.x < 0 || w.x >= cols || w.y < 0 || w.y >= w.z || w.z > P.z) {
    if (threadIdx.x == 0 && threadIdx.y == 0) cgFail(st, 4);
    return false;
  }
  x0 = (w.x % tilesX) * CTX;
  y0 = (w.x / tilesX) * CTR;
  z0 = w.y;
  z1 = w.z;
  return true;
}

// Tiles over (x, y), z split into chunks so that the blocks fill whole waves
// of the resident slots (wave count x chunk length minimal, chunks of at
// least 3 planes).
int residentBlocks(const void* kernel) {
  static std::mutex mu;
  static std::map<const void*, int> cache;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(kernel);
  if (it != cache.end()) return it->second;
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, CTX * CTY, 0) != cudaSuccess || per <= 0) per = 1;
  cache[kernel] = per;
  return per;
}

}  // namespace

// Work items of a CG schedule: one wave of the CG kernels of this
// preconditioner (the fewest resident blocks of the direction and both update
// kernels, at most kSchedPerSM per SM).
constexpr int kSchedPerSM = 8;
int cgScheduleTarget(int precond, bool xDouble);

// ---------------------------------------------------------------------------
// Launch shapes picked by measurement.  autotuneCg (driven by the solver)
// times the CG kernels of a grid for every z-chunk length in kTuneZPer and
// records the fastest per kernel family; cgLaunch prefers a recorded shape to
// its cost model.  The table is process wide and can be saved and loaded.
namespace {
constexpr int kTuneZPer[] = {3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 48, 64};
std::mutex g_tuneMu;
std::map<std::string, int> g_tune;  // "cg<family> nx ny nz" -> zPer

std::string tuneKey(int family, const Dim3i& cg) {
  return "cg" + std::to_string(family) + " " + std::to_string(cg.x) + " " + std::to_string(cg.y) + " " +
         std::to_string(cg.z);
}
int tunedZPer(int family, const Dim3i& cg) {
  std::lock_guard<std::mutex> lk(g_tuneMu);
  auto it = g_tune.find(tuneKey(family, cg));
  return it == g_tune.end() ? -1 : it->second;
}
}  // namespace

void setTunedCgZPer(int family, const Dim3i& cg, int zPer) {
  std::lock_guard<std::mutex> lk(g_tuneMu);
  if (zPer > 0) g_tune[tuneKey(family, cg)] = zPer;
  else g_tune.erase(tuneKey(family, cg));
}
int tunedCgZPer(int family, const Dim3i& cg) { return tunedZPer(family, cg); }
std::vector<int> cgZPerCandidates(const Dim3i& cg) {
  std::vector<int> v;
  for (int z : kTuneZPer)
    if (z <= cg.z) v.push_back(z);
  if (v.empty()) v.push_back(cg.z);
  return v;
}
bool saveTuning(const char* path) {
  std::lock_guard<std::mutex> lk(g_tuneMu);
  FILE* f = std::fopen(path, "w");
  if (!f) return false;
  std::fprintf(f, "# hfgrid launch shapes: cg<family 0 direction, 1 update> px ny nz zPer\n");
  for (const auto& kv : g_tune) std::fprintf(f, "%s %d\n", kv.first.c_str(), kv.second);
  return std::fclose(f) == 0;
}
int loadTuning(const char* path) {
  FILE* f = std::fopen(path, "r");
  if (!f) return -1;
  char name[16];
  int x, y, z, per, n = 0;
  char line[256];
  while (std::fgets(line, sizeof line, f)) {
    if (line[0] == '#') continue;
    if (std::sscanf(line, "%15s %d %d %d %d", name, &x, &y, &z, &per) != 5) continue;
    if ((std::string(name) != "cg0" && std::string(name) != "cg1") || per < 1 || per > z) continue;
    setTunedCgZPer(name[2] - '0', Dim3i{x, y, z}, per);
    ++n;
  }
  std::fclose(f);
  return n;
}

namespace {
// family: 0 for kCgDirection, 1 for kCgUpdate (the key of the tuning table).
// With a schedule the grid is one block per possible work item.
template <class K>
CgLaunch cgLaunch(const Dim3i& cg, K kernel, int family, const int* sched = nullptr, int precond = 1,
                  bool xDouble = false) {
  CgLaunch L;
  L.block = dim3(CTX, CTY, 1);
  if (sched) {
    L.zPer = 0;
    L.grid = dim3(cgScheduleTarget(precond, xDouble) + cgColumns(cg), 1, 1);
    return L;
  }
  int bx = (cg.x + CTX - 1) / CTX, by = (cg.y + CTR - 1) / CTR;
  const int tuned = tunedZPer(family, cg);
  if (tuned > 0) {
    L.zPer = std::min(tuned, cg.z);
    L.grid = dim3(bx, by, (cg.z + L.zPer - 1) / L.zPer);
    return L;
  }
  long long slots = (long long)numSMs() * residentBlocks((const void*)kernel);
  long long tiles = (long long)bx * by;
  long long best = -1;
  int bestPer = cg.z;
  // chunks of at least 3 planes: on small grids one-plane chunks pay the
  // ring's fill and a block's set-up for every plane (64^3: 16.1 us per
  // iteration with 1 plane, 15.2 with 3, 15.3 with 4, 19.2 with 8; 96^3:
  // 22.3 with 3, 24.1 with 4)
  for (int zPer = std::min(3, cg.z); zPer <= cg.z; ++zPer) {
    long long zc = (cg.z + zPer - 1) / zPer;
    long long waves = (tiles * zc + slots - 1) / slots;
    long long cost = waves * (zPer + 2);  // +2: pipeline fill per block
    if (best < 0 || cost < best) {
      best = cost;
      bestPer = zPer;
    }
  }
  L.zPer = bestPer;
  L.grid = dim3(bx, by, (cg.z + bestPer - 1) / bestPer);
  return L;
}

// CG direction: p = z + beta p_old (scal then axpy with 1), q = A p and the
// reduction p.q; the last block forms alpha = r.z / p.Ap
// (CuMatrixFreePCG.cpp:40-47, :56-60).  Stage i of the ring holds raw (z or r,
// p_old, code) of plane z0 + i with a one-cell halo; p of each plane (with
// halo) is formed once into a double-buffered tile, p above / below the
// current plane stay in registers.  PC: 0 identity, 1 Jacobi, 2 z from
// memory (multigrid).
template <int PC>
__global__ void __launch_bounds__(CTX* CTY, 4)
    kCgDirection(const __grid_constant__ CUtensorMap mZ, const __grid_constant__ CUtensorMap mPo,
                 const __grid_constant__ CUtensorMap mCode, Dim3i P, float sx, float sy, float sz,
                 const CgCode* __restrict__ code, const float* __restrict__ zr, const float* __restrict__ pOld,
                 float* __restrict__ pNew, double* partials, CgState* st, int zPer, const int* __restrict__ colZ) {
  __shared__ DirStage stg[kDirStages];
  __shared__ float pt[2][FH][CTX + 2];
  __shared__ DiagTab tab;
  __shared__ __align__(8) uint64_t bar[kDirStages];
  __shared__ int issued;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * CTX + tx;
  int x0 = 0, y0 = 0, z0 = 0, z1 = 0;
  auto issue = [&](int i) {
    DirStage& S = stg[i % kDirStages];
    uint64_t* b = &bar[i % kDirStages];
    mbarExpectTx(b, kDirStageBytes);
    tmaLoad3(&S.r[0][0], &mZ, x0 - HXF, y0 - 1, z0 + i, b);
    tmaLoad3(&S.po[0][0], &mPo, x0 - HXF, y0 - 1, z0 + i, b);
    tmaLoad3(&S.code[0][0], &mCode, x0 - HXC, y0 - 1, z0 + i, b);
  };
  if (tid == 0) {
    for (int s = 0; s < kDirStages; ++s) mbarInit(&bar[s], 1);
    mbarFenceInit();
  }
  buildDiagTab(tab, sx, sy, sz);
  __syncthreads();
  waitPrevGrid();
  if (st->done) return;  // the same value in every thread
  allowNextGrid();
  // a block with no work item (sched) writes nothing and adds zero to the
  // reduction; the schedule was written before the kernels before this one
  const bool active = cgBlockWork(colZ, P, zPer, x0, y0, z0, z1, st);
  const int nPlanes = active ? z1 - z0 : 0, nLoad = nPlanes + 1;  // plane z1 is the last "above"
  if (tid == 0) {
    int n = active ? min(kDirStages, nLoad) : 0;
    for (int i = 0; i < n; ++i) issue(i);
    issued = n;
  }
  const float beta = st->beta;
  const unsigned long long deadline = globalNs() + kWaitNs;
  const int x = x0 + tx;
  const unsigned plane = (unsigned)P.x * (unsigned)P.y;
  bool in[RY];
  unsigned c[RY];
  float below[RY], cur[RY], above[RY];
  float dCur[RY], dAbove[RY];
#pragma unroll
  for (int j = 0; j < RY; ++j) {
    const int y = y0 + ty + j * CTY;
    in[j] = x < P.x && y < P.y;
    c[j] = (unsigned)z0 * plane + (unsigned)y * (unsigned)P.x + (unsigned)x;
    // p of the plane below the chunk, own cell only
    below[j] = 0.f;
    if (active && in[j] && z0 > 0) {
      unsigned b = c[j] - plane;
      below[j] = fmaf(beta, __ldg(pOld + b), fastZ<PC>(tab.e[__ldg(code + b)].y, __ldg(zr + b)));
    }
  }
  // p of stage i's plane into tile t: the thread's RY cells, the x halo of its
  // rows and, for the edge warps, the y halo rows; own p and diagonals returned
  auto formTile = [&](int i, float (*t)[CTX + 2], float* v, float* dOwn) {
    const DirStage& S = stg[i % kDirStages];
    auto pAt = [&](int row, int colF, int colC) {
      return fmaf(beta, S.po[row][colF], fastZ<PC>(tab.e[S.code[row][colC]].y, S.r[row][colF]));
    };
#pragma unroll
    for (int j = 0; j < RY; ++j) {
      const int row = ty + 1 + j * CTY;
      const float2 e = tab.e[S.code[row][tx + HXC]];
      v[j] = fmaf(beta, S.po[row][tx + HXF], fastZ<PC>(e.y, S.r[row][tx + HXF]));
      dOwn[j] = e.x;
      t[row][tx + 1] = v[j];
    }
    // the halo ring, one warp-wide pass per side: warps 0 and CTY-1 take the
    // rows below and above; warp 3 takes both columns, lane l -> row
    // 1 + (l & 15), left for l < 16, right otherwise
    if (ty == 0) t[0][tx + 1] = pAt(0, tx + HXF, tx + HXC);
    if (ty == CTY - 1) t[CTR + 1][tx + 1] = pAt(CTR + 1, tx + HXF, tx + HXC);
    if (ty == 3) {
      const int row = 1 + (tx & (CTR - 1));
      const bool right = tx >= CTR;
      t[row][right ? CTX + 1 : 0] = pAt(row, right ? HXF + CTX : HXF - 1, right ? HXC + CTX : HXC - 1);
    }
  };
  bool ok = !active || mbarWait(&bar[0], 0, deadline);
  if (ok && active) formTile(0, pt[0], cur, dCur);
  int waited = active ? 1 : 0;
  bool fail = __syncthreads_or(!ok);
  if (active && !fail && tid == 0 && kDirStages < nLoad) issue(kDirStages), issued = kDirStages + 1;
  double acc = 0.0;  // FP64 dot partials: each product rounded to FP64, summed in FP64
  for (int i = 0; i < nPlanes && !fail; ++i) {
    ok = mbarWait(&bar[(i + 1) % kDirStages], (unsigned)(((i + 1) / kDirStages) & 1), deadline);
    waited = i + 2;
    if (ok) formTile(i + 1, pt[(i + 1) & 1], above, dAbove);
    float (*t)[CTX + 2] = pt[i & 1];
#pragma unroll
    for (int j = 0; j < RY; ++j) {
      if (in[j] && ok && dCur[j] >= 0.f) {  // fluid cells only
        const int row = ty + 1 + j * CTY;
        float q = rowSum(dCur[j], sx, sy, sz, cur[j], t[row][tx], t[row][tx + 2], t[row - 1][tx + 1],
                         t[row + 1][tx + 1], below[j], above[j]);
        pNew[c[j]] = cur[j];
        acc = fma((double)cur[j], (double)q, acc);
      }
      below[j] = cur[j];
      cur[j] = above[j];
      dCur[j] = dAbove[j];
      c[j] += plane;
    }
    fail = __syncthreads_or(!ok);
    if (!fail && tid == 0 && i + 1 + kDirStages < nLoad) issue(i + 1 + kDirStages), issued = i + 2 + kDirStages;
  }
  if (fail) {
    if (tid == 0) {
      cgFail(st, 1);
      drainStages<kDirStages>(bar, &issued, waited);
    }
    return;
  }
  double pq = acc, dummy = 0.0;
  if (gridSum2(pq, dummy, partials, &st->ticket) && flatTid() == 0) {
    st->pAp = pq;
    st->alpha = (float)(st->rz / pq);
    st->ticket = 0;
  }
}

// CG update: x += alpha p, r -= alpha A p (A p recomputed from the stored p
// of the stage ring), z = M^-1 r, the reductions r.r and r.z; the last block
// checks convergence and forms beta (CuMatrixFreePCG.cpp:49-63).  The
// |alpha| < FLT_EPSILON skip of CCuDenseVector::plusAlphaX
// (CuDenseVector.cpp:178) is kept.  The dot products accumulate in FP64 from
// the first product: per-thread partials over one z-column segment, then a
// fixed-order FP64 reduction over the grid.
template <int PC, class TX>
__global__ void __launch_bounds__(CTX* CTY, 4)
    kCgUpdate(const __grid_constant__ CUtensorMap mP, const __grid_constant__ CUtensorMap mR,
              const __grid_constant__ CUtensorMap mX, const __grid_constant__ CUtensorMap mCode, Dim3i P, float sx,
              float sy, float sz, const float* __restrict__ p, TX* __restrict__ xv, float* __restrict__ r,
              double* partials, CgState* st, int zPer, const int* __restrict__ colZ) {
  constexpr int kUpdStages = kUpdStagesT<TX>;
  using Stage = UpdStage<TX>;
  __shared__ Stage stg[kUpdStages];
  __shared__ DiagTab tab;
  __shared__ __align__(8) uint64_t bar[kUpdStages];
  __shared__ int issued;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * CTX + tx;
  int x0 = 0, y0 = 0, z0 = 0, z1 = 0;
  auto issue = [&](int i) {
    Stage& S = stg[i % kUpdStages];
    uint64_t* b = &bar[i % kUpdStages];
    mbarExpectTx(b, kUpdStageBytes<TX>);
    tmaLoad3(&S.p[0][0], &mP, x0 - HXF, y0 - 1, z0 + i, b);
    tmaLoad3(&S.r[0][0], &mR, x0, y0, z0 + i, b);
    tmaLoad3(&S.x[0][0], &mX, x0, y0, z0 + i, b);
    tmaLoad3(&S.code[0][0], &mCode, x0, y0, z0 + i, b);
  };
  if (tid == 0) {
    for (int s = 0; s < kUpdStages; ++s) mbarInit(&bar[s], 1);
    mbarFenceInit();
  }
  buildDiagTab(tab, sx, sy, sz);
  __syncthreads();
  waitPrevGrid();
  if (st->done) return;  // the same value in every thread
  allowNextGrid();
  const bool active = cgBlockWork(colZ, P, zPer, x0, y0, z0, z1, st);  // as in kCgDirection
  const int nPlanes = active ? z1 - z0 : 0, nLoad = nPlanes + 1;
  if (tid == 0) {
    int n = active ? min(kUpdStages, nLoad) : 0;
    for (int i = 0; i < n; ++i) issue(i);
    issued = n;
  }
  const float alpha = st->alpha;
  const bool skip = fabsf(alpha) < FLT_EPSILON;
  const unsigned long long deadline = globalNs() + kWaitNs;
  const int x = x0 + tx;
  const unsigned plane = (unsigned)P.x * (unsigned)P.y;
  bool in[RY];
  unsigned c[RY];
  float below[RY], cur[RY];
#pragma unroll
  for (int j = 0; j < RY; ++j) {
    const int y = y0 + ty + j * CTY;
    in[j] = x < P.x && y < P.y;
    c[j] = (unsigned)z0 * plane + (unsigned)y * (unsigned)P.x + (unsigned)x;
    below[j] = (active && in[j] && z0 > 0) ? __ldg(p + c[j] - plane) : 0.f;
  }
  bool ok = !active || mbarWait(&bar[0], 0, deadline);
#pragma unroll
  for (int j = 0; j < RY; ++j) cur[j] = (ok && active) ? stg[0].p[ty + 1 + j * CTY][tx + HXF] : 0.f;
  int waited = active ? 1 : 0;
  bool fail = __syncthreads_or(!ok);
  double arr = 0.0, arz = 0.0;  // FP64 dot partials
  for (int i = 0; i < nPlanes && !fail; ++i) {
    ok = mbarWait(&bar[(i + 1) % kUpdStages], (unsigned)(((i + 1) / kUpdStages) & 1), deadline);
    waited = i + 2;
    const Stage& A = stg[(i + 1) % kUpdStages];
    const Stage& S = stg[i % kUpdStages];
#pragma unroll
    for (int j = 0; j < RY; ++j) {
      const int row = ty + 1 + j * CTY, ir = ty + j * CTY;
      float above = ok ? A.p[row][tx + HXF] : 0.f;
      if (in[j] && ok) {
        CgCode k = S.code[ir][tx];
        const float2 e = tab.e[k];
        float rv = S.r[ir][tx];
        if (!skip && (k & 1)) {  // x, r and z stay zero off the fluid
          float q = rowSum(e.x, sx, sy, sz, cur[j], S.p[row][tx + HXF - 1], S.p[row][tx + HXF + 1],
                           S.p[row - 1][tx + HXF], S.p[row + 1][tx + HXF], below[j], above);
          if (sizeof(TX) == 8)  // FP64 accumulation: x + alpha p, each operation rounded once
            xv[c[j]] = (TX)__dadd_rn((double)S.x[ir][tx], __dmul_rn((double)alpha, (double)cur[j]));
          else
            xv[c[j]] = (TX)fmaf(alpha, cur[j], (float)S.x[ir][tx]);
          rv = fmaf(-alpha, q, rv);
          r[c[j]] = rv;
        }
        float zz = fastZ<PC>(e.y, rv);
        arr = fma((double)rv, (double)rv, arr);
        arz = fma((double)rv, (double)zz, arz);
      }
      below[j] = cur[j];
      cur[j] = above;
      c[j] += plane;
    }
    fail = __syncthreads_or(!ok);
    if (!fail && tid == 0 && i + kUpdStages < nLoad) issue(i + kUpdStages), issued = i + 1 + kUpdStages;
  }
  if (fail) {
    if (tid == 0) {
      cgFail(st, 1);
      drainStages<kUpdStages>(bar, &issued, waited);
    }
    return;
  }
  double rr = arr, rz = arz;
  if (gridSum2(rr, rz, partials, &st->ticket) && flatTid() == 0) {
    st->rr = rr;
    st->iter += 1;
    bool stop = cgStop(st, rr);
    if (PC != 2) {  // with multigrid the V-cycle's last sweep forms r.z and beta
      st->beta = (float)(rz / st->rz);
      st->rz = rz;
    }
    st->done = st->error || stop || st->iter >= st->maxIter;
    st->ticket = 0;
  }
}

// The two kernels on small grids, between the launches of a V-cycle (z from
// memory): a cell to a thread at a time, every load of a cell in flight at
// once.  There is nothing to stream on such a grid, and the ring's set-up and
// fill, the plane barriers and a reduction over many blocks were most of the
// time: with a V-cycle's launches around them, the
// CG stage of a 64^3 step 1.43 -> 1.36 ms.  The operations and their order are the marching kernels';
// neighbours that are solid or outside hold zero and are not loaded, which the
// cell's code tells without coordinates.
// This form / the marching kernels, us a CG iteration with its V-cycle: 24^3 55.3 /
// 59.1, 64^3 80.6 / 84.7, 80^3 (0.51 M cells) 103.5 / 108.4, 96^3 113.0 / 116.3,
// 112^3 128.3 / 127.5, 128^3 139.2 / 132.7.  The crossing is near 1.2 M cells; the
// line keeps to sizes where the gain is clear.
constexpr long long kCgSmallGrid = 1 << 19;          // cells of a small grid, at most
constexpr int kSmallThreads = 256, kSmallCells = 4;  // cells of a thread
struct CgNb {
  float l, r, d, u, b, f;
};
template <class G>
__device__ __forceinline__ CgNb cgNeighbours(CgCode k, unsigned c, unsigned nx, unsigned plane, G get) {
  CgNb n;
  n.l = k & 2 ? get(c - 1) : 0.f;
  n.r = k & 4 ? get(c + 1) : 0.f;
  n.d = k & 8 ? get(c - nx) : 0.f;
  n.u = k & 16 ? get(c + nx) : 0.f;
  n.b = k & 32 ? get(c - plane) : 0.f;
  n.f = k & 64 ? get(c + plane) : 0.f;
  return n;
}
__global__ void __launch_bounds__(kSmallThreads)
    kCgDirectionSmall(Dim3i P, float sx, float sy, float sz, const CgCode* __restrict__ code,
                      const float* __restrict__ z, const float* __restrict__ pOld, float* __restrict__ pNew,
                      double* partials, CgState* st) {
  const unsigned nx = (unsigned)P.x, plane = nx * (unsigned)P.y, n = plane * (unsigned)P.z;
  const unsigned c0 = blockIdx.x * (kSmallThreads * kSmallCells) + threadIdx.x;
  CgCode k[kSmallCells];  // the codes do not change within a solve
#pragma unroll
  for (int j = 0; j < kSmallCells; ++j) {
    const unsigned c = c0 + j * kSmallThreads;
    k[j] = c < n ? __ldg(code + c) : (CgCode)0;
  }
  waitPrevGrid();
  if (st->done) return;
  allowNextGrid();
  const float beta = st->beta;
  auto pAt = [&](unsigned i) { return fmaf(beta, __ldg(pOld + i), __ldg(z + i)); };
  double acc = 0.0, dummy = 0.0;
#pragma unroll
  for (int j = 0; j < kSmallCells; ++j) {
    if (!(k[j] & 1)) continue;
    const unsigned c = c0 + j * kSmallThreads;
    const float pc = pAt(c);
    const CgNb v = cgNeighbours(k[j], c, nx, plane, pAt);
    const float q = rowSum(diagOf((Code)k[j], sx, sy, sz), sx, sy, sz, pc, v.l, v.r, v.d, v.u, v.b, v.f);
    pNew[c] = pc;
    acc = fma((double)pc, (double)q, acc);
  }
  if (gridSum2(acc, dummy, partials, &st->ticket) && flatTid() == 0) {
    st->pAp = acc;
    st->alpha = (float)(st->rz / acc);
    st->ticket = 0;
  }
}
template <class TX>
__global__ void __launch_bounds__(kSmallThreads)
    kCgUpdateSmall(Dim3i P, float sx, float sy, float sz, const CgCode* __restrict__ code, const float* __restrict__ p,
                   TX* __restrict__ x, float* __restrict__ r, double* partials, CgState* st) {
  const unsigned nx = (unsigned)P.x, plane = nx * (unsigned)P.y, n = plane * (unsigned)P.z;
  const unsigned c0 = blockIdx.x * (kSmallThreads * kSmallCells) + threadIdx.x;
  CgCode k[kSmallCells];
#pragma unroll
  for (int j = 0; j < kSmallCells; ++j) {
    const unsigned c = c0 + j * kSmallThreads;
    k[j] = c < n ? __ldg(code + c) : (CgCode)0;
  }
  waitPrevGrid();
  if (st->done) return;
  allowNextGrid();
  const float alpha = st->alpha;
  const bool skip = fabsf(alpha) < FLT_EPSILON;
  double rr = 0.0, dummy = 0.0;
#pragma unroll
  for (int j = 0; j < kSmallCells; ++j) {
    if (!(k[j] & 1)) continue;
    const unsigned c = c0 + j * kSmallThreads;
    float rv = r[c];
    if (!skip) {
      const float pc = __ldg(p + c);
      const CgNb v = cgNeighbours(k[j], c, nx, plane, [&](unsigned i) { return __ldg(p + i); });
      const float q = rowSum(diagOf((Code)k[j], sx, sy, sz), sx, sy, sz, pc, v.l, v.r, v.d, v.u, v.b, v.f);
      if (sizeof(TX) == 8)
        x[c] = (TX)__dadd_rn((double)x[c], __dmul_rn((double)alpha, (double)pc));
      else
        x[c] = (TX)fmaf(alpha, pc, (float)x[c]);
      rv = fmaf(-alpha, q, rv);
      r[c] = rv;
    }
    rr = fma((double)rv, (double)rv, rr);
  }
  if (gridSum2(rr, dummy, partials, &st->ticket) && flatTid() == 0) {
    st->rr = rr;
    st->iter += 1;
    st->done = st->error || cgStop(st, rr) || st->iter >= st->maxIter;
    st->ticket = 0;
  }
}
int smallBlocks(const Dim3i& cg) {
  return (int)((cg.size() + kSmallThreads * kSmallCells - 1) / (kSmallThreads * kSmallCells));
}

// ---------------------------------------------------------------------------
// The resident CG: whole solves in one cooperative launch, for systems whose
// fluid fits the shared memory of the GPU.
//
// The kernel pair above streams r, p, x and the codes past every SM twice per
// iteration and pays two launches, two ring fills and a block barrier per
// plane for it; on small grids the launches alone are most of an iteration.
// Here one block per SM keeps its share of the system for the whole solve:
// p (with halo) and the codes in shared memory, and x, r and A p in registers
// when the share is small (at most kResKL quads of cells to a thread), else x
// and r stream from L2.  A thread works on four cells in x at a time, so the
// addresses, the code test and the wide loads serve four.  An iteration is
//   p = z + beta p on the block's cells and, from the neighbours' z, on its
//     halo; A p; the grid reduction p.Ap -> alpha;
//   x += alpha p, r -= alpha A p; z at the share's faces published to zG; the
//     grid reductions r.r and r.z -> beta, and the stop test;
// with the operations of kCgDirection and kCgUpdate on every cell, so the
// iterates agree with theirs up to the order of the FP64 dot-product sums.
// Every block sums the partials in the same fixed order and forms the same
// scalars; the two grid reductions are the only waits (bounded at 2 s).
//
// Shares: the fluid runs of the tile columns (sched's extents) laid end to
// end and cut into equal parts of n planes of 32 x 16 cells; a part covers
// one or a few segments of columns, each with a halo plane at both ends.
// A system whose parts do not fit leaves the state untouched (resident = 2)
// and is solved by the kernel pair.
// Small systems (at most 16 shares in the register form) run as one cluster of
// 16 blocks instead of a grid: the reductions then go through the cluster's
// shared memory and hardware barrier: 6.6 -> 5.2 us per iteration at 33^3.
// Measured (B200, Jacobi), us per iteration, pair -> resident: 33^3 dam break
// 17.8 -> 6.9, 128^3 31.5 -> 10.4, 160^3 -> 15.6, 256^3 (4.0 M fluid cells)
// 62 -> 34.  What bounds it now: the two reductions (about 2.5 us each) on the
// small grids, issue slots (row sums, FP64 dot products) on the large ones.
// 512 threads with up to 128 registers: 768 (80) and 1024 (64, spills) took 50
// and 63 us at 256^3 where 512 took 45 (with one shared reduction array).
constexpr int RTH = 512;                       // threads of a block
constexpr int RQ = CTX / 4, RPT = RQ * CTR;    // a plane of a tile: 128 quads of 4 cells in x, one thread each
constexpr int RG = RTH / RPT;                  // planes in hand at once
static_assert(RQ == 8 && RTH % RPT == 0, "a warp holds four rows of eight quads");
// A plane in shared memory: rows -1 .. 16 of 32 floats, then the columns left
// and right of the tile (16 floats each).
constexpr int RXL = (CTR + 2) * CTX, RXR = RXL + CTR, RPL = RXR + CTR;
constexpr int kResPlanes = 96, kResSegs = 32;  // planes and segments of one block, at most
constexpr int kResGrid = 256;                  // blocks, at most
constexpr int kResMinPlanes = 2;
constexpr int kResCluster = 16;                // blocks of the cluster form
constexpr int kResCols = 1024 / RTH;           // tile columns per thread of the share plan
constexpr int kResKL = 4;                      // quads of a thread held in registers

struct ResShared {
  DiagTab tab;
  int4 plane[kResPlanes];  // x0, y0, z, -
  int2 at[kResPlanes];     // linear index of the tile origin; float offset of the plane | first or last of its segment
  int4 seg[kResSegs];      // tile column, first plane, planes, first local plane
  int segSlot[kResSegs];   // slot of the segment's lower halo plane
  int hist[kResGrid];
  double red[2][RTH / 32];
  double tot[2][kResGrid / 32];
  double mail[2][2][kResCluster];  // cluster form: the other blocks' partials, by epoch parity and value
  int scan[32];
  int total, nSegs, maxSegs, ok;
};

// 16-byte accesses that other SMs see whole: a partial sum and its tag.
struct Tagged {
  double v;
  unsigned long long tag;
};
__device__ __forceinline__ void putTagged(Tagged* p, double v, unsigned long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ Tagged getTagged(const Tagged* p) {
  Tagged r;
  long long v;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(v), "=l"(r.tag)
               : "l"(p)
               : "memory");
  r.v = __longlong_as_double(v);
  return r;
}

// One grid reduction of a (and b) over blocks 0 .. m-1; every thread gets the
// totals.  Every block has a mailbox with a slot for each block: a block puts
// its partial sum, tagged with the epoch, into its slot of all m mailboxes and
// polls its own.  So a reduction is one store and one load deep, and no line
// is polled by more than one SM (with one shared array that all blocks polled,
// an iteration took 13.5 us instead of 10.4 at 128^3).  The mailboxes of two
// epochs alternate: a slot is written again only after every block has passed
// the epoch between.  PUBLISH: global writes before the call are visible to
// every block after it.  False once a wait ran out here or in another block.
template <int NV, bool PUBLISH>
__device__ __forceinline__ bool resReduce(double& a, double& b, ResShared& sh, Tagged* box, unsigned epoch, int m,
                                          CgState* st) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  a = warpSumD(a);
  if (NV > 1) b = warpSumD(b);
  if (lane == 0) {
    sh.red[0][w] = a;
    if (NV > 1) sh.red[1][w] = b;
  }
  __syncthreads();
  constexpr int U = kResGrid / 32;
  static_assert(U <= RTH / 32 && RTH / 32 <= 32, "one warp per 32 blocks");
  const unsigned long long tag = epoch + 1ull;
  if (32 * w < m) {  // warp w serves blocks 32 w .. 32 w + 31
    const int j = 32 * w + lane;
    const double a0 = __shfl_sync(0xffffffffu, warpSumD(lane < RTH / 32 ? sh.red[0][lane] : 0.0), 0);
    double b0 = 0.0;
    if (NV > 1) b0 = __shfl_sync(0xffffffffu, warpSumD(lane < RTH / 32 ? sh.red[1][lane] : 0.0), 0);
    // mailbox of block k: box[((epoch & 1) * m + k) * 2 m + ...]
    Tagged* all = box + (size_t)(epoch & 1) * m * 2 * m;
    if (j < m) {
      if (PUBLISH) __threadfence();
      Tagged* to = all + (size_t)j * 2 * m + blockIdx.x;
      putTagged(to, a0, tag);
      if (NV > 1) putTagged(to + m, b0, tag);
    }
    const Tagged* mine = all + (size_t)blockIdx.x * 2 * m;
    Tagged v[NV];
    unsigned long long deadline = 0;
    for (int spin = 0;; ++spin) {
      bool here = true;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        v[k] = Tagged{0.0, tag};
        if (j < m) v[k] = getTagged(mine + k * m + j);
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) here = here && v[k].tag == tag;
      if (__all_sync(0xffffffffu, here)) break;
      if ((spin & 63) == 63) {
        const unsigned long long now = globalNs();
        if (deadline == 0) deadline = now + kWaitNs;
        const bool give = now > deadline || ldAcquire((const unsigned*)&st->error) != 0u;
        if (__any_sync(0xffffffffu, give)) {
          if (lane == 0) {
            cgFail(st, 2);
            sh.ok = 0;
          }
          break;
        }
      }
    }
    if (PUBLISH) __threadfence();
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const double sum = warpSumD(v[k].v);
      if (lane == 0) sh.tot[k][w] = sum;
    }
  }
  __syncthreads();
  a = b = 0.0;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (32 * u < m) {
      a += sh.tot[0][u];
      if (NV > 1) b += sh.tot[1][u];
    }
  return sh.ok != 0;
}

// The same reduction over the m blocks of one cluster: the partials go straight
// into the other blocks' shared memory and the cluster's hardware barrier is
// the only wait.  It makes global writes before it visible to the cluster too.
template <int NV>
__device__ __forceinline__ void resReduceCluster(double& a, double& b, ResShared& sh, unsigned epoch, int m) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  a = warpSumD(a);
  if (NV > 1) b = warpSumD(b);
  if (lane == 0) {
    sh.red[0][w] = a;
    if (NV > 1) sh.red[1][w] = b;
  }
  __syncthreads();
  const int par = epoch & 1;
  if (w == 0) {
    const double a0 = __shfl_sync(0xffffffffu, warpSumD(lane < RTH / 32 ? sh.red[0][lane] : 0.0), 0);
    double b0 = 0.0;
    if (NV > 1) b0 = __shfl_sync(0xffffffffu, warpSumD(lane < RTH / 32 ? sh.red[1][lane] : 0.0), 0);
    const int k = lane >> 4, to = lane & (kResCluster - 1);  // value k to block `to`
    if (k < NV && to < m) {
      unsigned remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smemAddr(&sh.mail[par][k][blockIdx.x])), "r"(to));
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(k ? b0 : a0) : "memory");
    }
  }
  clusterArrive();
  clusterWait();
  a = b = 0.0;
  for (int j = 0; j < m; ++j) {
    a += sh.mail[par][0][j];
    if (NV > 1) b += sh.mail[par][1][j];
  }
}

struct ResArgs {
  Dim3i P;
  float sx, sy, sz;
  const CgCode* code;
  float *r, *x, *p, *zG;
  Tagged* box;
  CgState* st;
  int maxIters;  // iterations of this launch
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
constexpr unsigned kAllInner = 0x7f7f7f7fu;  // four fluid cells, no neighbour solid or outside

// Diagonals and reciprocals of four cells; a cell off the fluid has diagonal -1.
__device__ __forceinline__ void diag4(const DiagTab& t, unsigned c4, float4& d, float4& inv) {
  const float2 e = t.e[0x7f];
  d = make_float4(e.x, e.x, e.x, e.x);
  inv = make_float4(e.y, e.y, e.y, e.y);
  if (c4 != kAllInner) {
    const float2 e0 = t.e[c4 & 0xff], e1 = t.e[(c4 >> 8) & 0xff], e2 = t.e[(c4 >> 16) & 0xff], e3 = t.e[c4 >> 24];
    d = make_float4(e0.x, e1.x, e2.x, e3.x);
    inv = make_float4(e0.y, e1.y, e2.y, e3.y);
  }
}
template <int PC>
__device__ __forceinline__ float4 z4(float4 inv, float4 r) {
  return make_float4(fastZ<PC>(inv.x, r.x), fastZ<PC>(inv.y, r.y), fastZ<PC>(inv.z, r.z), fastZ<PC>(inv.w, r.w));
}
__device__ __forceinline__ float4 fma4(float s, float4 a, float4 b) {
  return make_float4(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y), fmaf(s, a.z, b.z), fmaf(s, a.w, b.w));
}
// four rows of A (0 off the fluid)
__device__ __forceinline__ float4 rows4(const ResArgs& A, float4 d, float4 c, float l, float r, float4 dn, float4 up,
                                        float4 be, float4 ab) {
  float4 q = make_float4(rowSum(d.x, A.sx, A.sy, A.sz, c.x, l, c.y, dn.x, up.x, be.x, ab.x),
                         rowSum(d.y, A.sx, A.sy, A.sz, c.y, c.x, c.z, dn.y, up.y, be.y, ab.y),
                         rowSum(d.z, A.sx, A.sy, A.sz, c.z, c.y, c.w, dn.z, up.z, be.z, ab.z),
                         rowSum(d.w, A.sx, A.sy, A.sz, c.w, c.z, r, dn.w, up.w, be.w, ab.w));
  if (d.x < 0.f) q.x = 0.f;
  if (d.y < 0.f) q.y = 0.f;
  if (d.z < 0.f) q.z = 0.f;
  if (d.w < 0.f) q.w = 0.f;
  return q;
}
__device__ __forceinline__ void dot4(double& s, float4 a, float4 b) {
  s = fma((double)a.x, (double)b.x, s);
  s = fma((double)a.y, (double)b.y, s);
  s = fma((double)a.z, (double)b.z, s);
  s = fma((double)a.w, (double)b.w, s);
}

// The solve of one block's share.  KL > 0: at most KL quads per thread, x, r
// and A p in registers; KL = 0: any number, x and r in global memory and A p
// formed twice.  Cells off the fluid hold zeros in every vector.
template <int PC, int KL, bool CLUSTER>
__device__ void resSolve(const ResArgs& A, ResShared& sh, float* __restrict__ tile, const unsigned* __restrict__ codeS,
                         int nb, int m) {
  const int tid = threadIdx.x, grp = tid / RPT, cell = tid % RPT, row = cell / RQ, col = cell % RQ;
  const Dim3i P = A.P;
  CgState* st = A.st;
  constexpr int KR = KL > 0 ? KL : 1, RU = 6;
  float4 rR[KR], xR[KR], qR[KR];
  const int nSegs = sh.nSegs;
  // this thread's planes, its quad in a plane and the cells beside it
  const int per = (nb + RG - 1) / RG, i0 = min(nb, grp * per), i1 = min(nb, i0 + per);
  const int own = (row + 1) * CTX + 4 * col;
  const int left = col == 0 ? RXL + row : own - 1, right = col == RQ - 1 ? RXR + row : own + 4;
  const unsigned off = (unsigned)row * (unsigned)P.x + 4u * (unsigned)col;
  const bool faceXY = row == 0 || row == CTR - 1 || col == 0 || col == RQ - 1;
  float* __restrict__ gr = A.r;
  float* __restrict__ gx = A.x;

  // halo quads: rows -1 and 16 of every plane, then the halo planes of every segment
  const int hq = 2 * RQ * nb, hAll = hq + 2 * RPT * nSegs;
  auto haloQuad = [&](int h, int& t) -> int {
    int gx0, gy, gz;
    if (h < hq) {
      const int i = h >> 4, hi = (h >> 3) & 1, c = h & 7;
      const int4 pl = sh.plane[i];
      gx0 = pl.x + 4 * c;
      gy = hi ? pl.y + CTR : pl.y - 1;
      gz = pl.z;
      t = (sh.at[i].y & ~1) + (hi ? CTR + 1 : 0) * CTX + 4 * c;
    } else {
      const int k = h - hq, s = k >> 8, hi = (k >> 7) & 1, rw = (k >> 3) & 15, c = k & 7;
      const int4 sg = sh.seg[s];
      const int4 pl = sh.plane[sg.w];
      gx0 = pl.x + 4 * c;
      gy = pl.y + rw;
      gz = hi ? sg.y + sg.z : sg.y - 1;
      t = (sh.segSlot[s] + (hi ? sg.z + 1 : 0)) * RPL + (rw + 1) * CTX + 4 * c;
    }
    return gx0 < P.x && (unsigned)gy < (unsigned)P.y && (unsigned)gz < (unsigned)P.z ? (gz * P.y + gy) * P.x + gx0 : -1;
  };
  // halo columns: 16 cells left and 16 right of every plane
  auto haloCol = [&](int h, int& t) -> int {
    const int i = h >> 5, hi = (h >> 4) & 1, rw = h & 15;
    const int4 pl = sh.plane[i];
    const int gx1 = hi ? pl.x + CTX : pl.x - 1, gy = pl.y + rw;
    t = (sh.at[i].y & ~1) + (hi ? RXR : RXL) + rw;
    return (unsigned)gx1 < (unsigned)P.x && gy < P.y ? (pl.z * P.y + gy) * P.x + gx1 : -1;
  };
  auto publish = [&](int2 at, unsigned c, float4 z) {
    if (faceXY || (at.y & 1)) __stcg(reinterpret_cast<float4*>(A.zG + c), z);
  };

  // the share as the last launch (or the RHS kernel) left it
  for (int h = tid; h < hAll; h += RTH) {
    int t;
    const int g = haloQuad(h, t);
    if (g >= 0) st4(tile + t, ld4(A.p + g));
  }
  for (int h = tid; h < 32 * nb; h += RTH) {
    int t;
    const int g = haloCol(h, t);
    if (g >= 0) tile[t] = A.p[g];
  }
  for (int i = i0; i < i1; ++i) {
    const unsigned c4 = codeS[i * RPT + cell];
    if (!c4) continue;
    const int2 at = sh.at[i];
    const unsigned c = (unsigned)at.x + off;
    float4 d, inv;
    diag4(sh.tab, c4, d, inv);
    st4(tile + (at.y & ~1) + own, ld4(A.p + c));
    publish(at, c, z4<PC>(inv, ld4(gr + c)));
  }
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  if (KL > 0) {
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      rR[k] = xR[k] = qR[k] = zero;
      if (i0 + k < i1 && codeS[(i0 + k) * RPT + cell]) {
        const unsigned c = (unsigned)sh.at[i0 + k].x + off;
        rR[k] = ld4(gr + c);
        xR[k] = ld4(gx + c);
      }
    }
  }
  float beta = st->beta, alpha = st->alpha;
  double rz = st->rz, rr = st->rr, pAp = st->pAp;
  int iter = st->iter, done = 0;
  const int maxIter = st->maxIter;
  unsigned epoch = 0;
  double a = 0.0, b = 0.0;
  auto reduce1 = [&](bool publish) -> bool {
    if (CLUSTER) {
      resReduceCluster<1>(a, b, sh, epoch++, m);
      return true;
    }
    return publish ? resReduce<1, true>(a, b, sh, A.box, epoch++, m, st)
                   : resReduce<1, false>(a, b, sh, A.box, epoch++, m, st);
  };
  auto reduce2 = [&]() -> bool {
    if (CLUSTER) {
      resReduceCluster<2>(a, b, sh, epoch++, m);
      return true;
    }
    return resReduce<2, true>(a, b, sh, A.box, epoch++, m, st);
  };
  if (!reduce1(true)) return;  // every share's z is out

  for (int it = 0; it < A.maxIters; ++it) {
    // p on the halo and on the share
    for (int h0 = tid; h0 < hAll; h0 += 2 * RTH) {
      float4 zv[2];
      int t[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int h = h0 + u * RTH;
        int g = -1;
        if (h < hAll) g = haloQuad(h, t[u]);
        if (g >= 0) zv[u] = __ldcg(reinterpret_cast<const float4*>(A.zG + g));
        else t[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (t[u] >= 0) st4(tile + t[u], fma4(beta, ld4(tile + t[u]), zv[u]));
    }
    for (int h0 = tid; h0 < 32 * nb; h0 += 2 * RTH) {
      float zv[2];
      int t[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int h = h0 + u * RTH;
        int g = -1;
        if (h < 32 * nb) g = haloCol(h, t[u]);
        if (g >= 0) zv[u] = __ldcg(A.zG + g);
        else t[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (t[u] >= 0) tile[t[u]] = fmaf(beta, tile[t[u]], zv[u]);
    }
    if (KL > 0) {
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        if (i0 + k >= i1) continue;
        const unsigned c4 = codeS[(i0 + k) * RPT + cell];
        if (!c4) continue;
        float4 d, inv;
        diag4(sh.tab, c4, d, inv);
        float* t = tile + (sh.at[i0 + k].y & ~1) + own;
        st4(t, fma4(beta, ld4(t), z4<PC>(inv, rR[k])));
      }
    } else {
      for (int ib = i0; ib < i1; ib += RU) {  // RU planes' loads in flight
        unsigned c4[RU];
        float4 rv[RU];
#pragma unroll
        for (int u = 0; u < RU; ++u) {
          c4[u] = ib + u < i1 ? codeS[(ib + u) * RPT + cell] : 0u;
          if (c4[u]) rv[u] = ld4(gr + (unsigned)sh.at[ib + u].x + off);
        }
#pragma unroll
        for (int u = 0; u < RU; ++u) {
          if (!c4[u]) continue;
          float4 d, inv;
          diag4(sh.tab, c4[u], d, inv);
          float* t = tile + (sh.at[ib + u].y & ~1) + own;
          st4(t, fma4(beta, ld4(t), z4<PC>(inv, rv[u])));
        }
      }
    }
    __syncthreads();
    a = b = 0.0;
    if (KL > 0) {
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        if (i0 + k >= i1) continue;
        const unsigned c4 = codeS[(i0 + k) * RPT + cell];
        if (!c4) continue;
        float4 d, inv;
        diag4(sh.tab, c4, d, inv);
        const float* t = tile + (sh.at[i0 + k].y & ~1);
        const float4 pc = ld4(t + own);
        qR[k] = rows4(A, d, pc, t[left], t[right], ld4(t + own - CTX), ld4(t + own + CTX), ld4(t + own - RPL),
                      ld4(t + own + RPL));
        dot4(a, pc, qR[k]);
      }
    } else {
      const float* tp = nullptr;
      float4 be = zero, pc = zero;
      for (int i = i0; i < i1; ++i) {
        const float* t = tile + (sh.at[i].y & ~1);
        if (t != tp) {  // the first plane of a segment
          be = ld4(t + own - RPL);
          pc = ld4(t + own);
        }
        const float4 ab = ld4(t + own + RPL);
        const unsigned c4 = codeS[i * RPT + cell];
        if (c4) {
          float4 d, inv;
          diag4(sh.tab, c4, d, inv);
          dot4(a, pc, rows4(A, d, pc, t[left], t[right], ld4(t + own - CTX), ld4(t + own + CTX), be, ab));
        }
        be = pc;
        pc = ab;
        tp = t + RPL;
      }
    }
    if (!reduce1(false)) return;
    pAp = a;
    alpha = (float)(rz / pAp);
    const bool skip = fabsf(alpha) < FLT_EPSILON;
    a = b = 0.0;
    if (KL > 0) {
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        if (i0 + k >= i1) continue;
        const unsigned c4 = codeS[(i0 + k) * RPT + cell];
        if (!c4) continue;
        const int2 at = sh.at[i0 + k];
        float4 d, inv;
        diag4(sh.tab, c4, d, inv);
        if (!skip) {
          xR[k] = fma4(alpha, ld4(tile + (at.y & ~1) + own), xR[k]);
          rR[k] = fma4(-alpha, qR[k], rR[k]);
        }
        const float4 zz = z4<PC>(inv, rR[k]);
        publish(at, (unsigned)at.x + off, zz);
        dot4(a, rR[k], rR[k]);
        dot4(b, rR[k], zz);
      }
    } else {
      const float* tp = nullptr;
      float4 be = zero, pc = zero;
      float4 rn = zero, xn = zero;  // r and x of the next plane, loaded one plane ahead
      if (i0 < i1 && codeS[i0 * RPT + cell]) {
        const unsigned c = (unsigned)sh.at[i0].x + off;
        rn = ld4(gr + c);
        xn = ld4(gx + c);
      }
      for (int i = i0; i < i1; ++i) {
        const int2 at = sh.at[i];
        const float* t = tile + (at.y & ~1);
        float4 rv = rn, xv = xn;
        if (i + 1 < i1 && codeS[(i + 1) * RPT + cell]) {
          const unsigned c = (unsigned)sh.at[i + 1].x + off;
          rn = ld4(gr + c);
          xn = ld4(gx + c);
        }
        if (t != tp) {
          be = ld4(t + own - RPL);
          pc = ld4(t + own);
        }
        const float4 ab = ld4(t + own + RPL);
        const unsigned c4 = codeS[i * RPT + cell];
        if (c4) {
          const unsigned c = (unsigned)at.x + off;
          float4 d, inv;
          diag4(sh.tab, c4, d, inv);
          if (!skip) {
            const float4 q = rows4(A, d, pc, t[left], t[right], ld4(t + own - CTX), ld4(t + own + CTX), be, ab);
            st4(gx + c, fma4(alpha, pc, xv));
            rv = fma4(-alpha, q, rv);
            st4(gr + c, rv);
          }
          const float4 zz = z4<PC>(inv, rv);
          publish(at, c, zz);
          dot4(a, rv, rv);
          dot4(b, rv, zz);
        }
        be = pc;
        pc = ab;
        tp = t + RPL;
      }
    }
    if (!reduce2()) return;
    rr = a;
    ++iter;
    beta = (float)(b / rz);
    rz = b;
    done = cgStop(st, rr) || iter >= maxIter;
    if (done) break;
  }
  // x for the caller; r and p for the next launch
  if (KL > 0) {
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      if (i0 + k < i1 && codeS[(i0 + k) * RPT + cell]) {
        const unsigned c = (unsigned)sh.at[i0 + k].x + off;
        st4(gx + c, xR[k]);
        st4(gr + c, rR[k]);
      }
    }
  }
  if (!done)
    for (int i = i0; i < i1; ++i)
      if (codeS[i * RPT + cell]) {
        const int2 at = sh.at[i];
        st4(A.p + (unsigned)at.x + off, ld4(tile + (at.y & ~1) + own));
      }
  if (blockIdx.x == 0 && tid == 0) {
    st->alpha = alpha;
    st->beta = beta;
    st->rz = rz;
    st->rr = rr;
    st->pAp = pAp;
    st->iter = iter;
    st->done = done;
    st->resident = 1;
  }
}

template <int PC, bool CLUSTER>
__global__ void __launch_bounds__(RTH, 1) kCgResident(ResArgs A, const int* __restrict__ sched, int cols, int dynBytes) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ __align__(16) ResShared sh;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (A.st->done) return;
  buildDiagTab(sh.tab, A.sx, A.sy, A.sz);
  // prefix sum of the columns' fluid planes, kResCols columns per thread
  int lo[kResCols], len[kResCols], inc = 0;
#pragma unroll
  for (int j = 0; j < kResCols; ++j) {
    const int c = kResCols * tid + j;
    lo[j] = len[j] = 0;
    if (c < cols) {
      lo[j] = __ldg(sched + c);
      const int hi = __ldg(sched + cols + c);
      len[j] = hi >= lo[j] ? hi - lo[j] + 1 : 0;
    }
    inc += len[j];
  }
  const int mine = inc;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += v;
  }
  if (lane == 31) sh.scan[w] = inc;
  for (int i = tid; i < kResGrid; i += RTH) sh.hist[i] = 0;
  if (tid == 0) {
    sh.nSegs = sh.maxSegs = 0;
    sh.ok = 1;
  }
  __syncthreads();
  if (w == 0) {
    const int v = lane < RTH / 32 ? sh.scan[lane] : 0;
    int vi = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, vi, d);
      if (lane >= d) vi += u;
    }
    sh.scan[lane] = vi - v;
    if (lane == 31) sh.total = vi;
  }
  __syncthreads();
  const int S = sh.total, first = sh.scan[w] + inc - mine;
  const int n = max(kResMinPlanes, (S + (int)gridDim.x - 1) / (int)gridDim.x);
  const int m = (S + n - 1) / n;  // blocks with a share
  // segments of every share: the fit is decided alike in every block
  for (int j = 0, pre = first; j < kResCols; pre += len[j++])
    if (len[j] > 0)
      for (int b = pre / n; b <= (pre + len[j] - 1) / n; ++b) atomicMax(&sh.maxSegs, atomicAdd(&sh.hist[b], 1) + 1);
  __syncthreads();
  const int maxSegs = sh.maxSegs;
  const long long need = (long long)(n + 2 * maxSegs) * RPL * sizeof(float) + (long long)n * (CTX * CTR);
  if (n > (CLUSTER ? RG * kResKL : kResPlanes) || maxSegs > kResSegs || need > dynBytes) {
    if (blockIdx.x == 0 && tid == 0) A.st->resident = 2;
    return;
  }
  if ((int)blockIdx.x >= m) return;
  // this block's segments, tile slots and planes
  const int b0 = blockIdx.x * n, b1 = min(S, b0 + n), nb = b1 - b0;
  for (int j = 0, pre = first; j < kResCols; pre += len[j++]) {
    const int s0 = max(pre, b0), s1 = min(pre + len[j], b1);
    if (len[j] > 0 && s0 < s1)
      sh.seg[atomicAdd(&sh.nSegs, 1)] = make_int4(kResCols * tid + j, lo[j] + s0 - pre, s1 - s0, s0 - b0);
  }
  __syncthreads();
  const int nSegs = sh.nSegs;
  if (tid == 0) {
    int slot = 0;
    for (int s = 0; s < nSegs; ++s) {
      sh.segSlot[s] = slot;
      slot += sh.seg[s].z + 2;
    }
  }
  __syncthreads();
  const int tilesX = (A.P.x + CTX - 1) / CTX;
  if (tid < nb) {
    for (int s = 0; s < nSegs; ++s) {
      const int4 sg = sh.seg[s];
      const int k = tid - sg.w;
      if (k < 0 || k >= sg.z) continue;
      const int x0 = (sg.x % tilesX) * CTX, y0 = (sg.x / tilesX) * CTR, z = sg.y + k;
      const int edge = k == 0 || k == sg.z - 1;
      sh.plane[tid] = make_int4(x0, y0, z, 0);
      sh.at[tid] = make_int2((z * A.P.y + y0) * A.P.x + x0, (sh.segSlot[s] + 1 + k) * RPL | edge);
    }
  }
  float* tile = reinterpret_cast<float*>(dyn);
  unsigned* codeS = reinterpret_cast<unsigned*>(tile + (n + 2 * maxSegs) * RPL);
  for (int i = tid; i < (nb + 2 * nSegs) * RPL; i += RTH) tile[i] = 0.f;
  __syncthreads();
  for (int h = tid; h < nb * RPT; h += RTH) {
    const int i = h / RPT, cell = h % RPT, row = cell / RQ, col = cell % RQ;
    const int4 pl = sh.plane[i];
    unsigned c4 = 0;
    if (pl.x + 4 * col < A.P.x && pl.y + row < A.P.y)
      c4 = __ldg(reinterpret_cast<const unsigned*>(A.code + (unsigned)sh.at[i].x + (unsigned)row * (unsigned)A.P.x +
                                                   4u * (unsigned)col));
    // cells off the fluid carry no bits, so four of them are code 0
    const unsigned fl = c4 & 0x01010101u;
    codeS[h] = c4 & (fl * 0xffu);
  }
  __syncthreads();
  if (CLUSTER) {
    // a block's shared memory may be written once it has started
    clusterArrive();
    clusterWait();
    resSolve<PC, kResKL, true>(A, sh, tile, codeS, nb, m);
  } else if ((n + RG - 1) / RG <= kResKL) {
    resSolve<PC, kResKL, false>(A, sh, tile, codeS, nb, m);
  } else {
    resSolve<PC, 0, false>(A, sh, tile, codeS, nb, m);
  }
}

// Tensor map of a pitched 3-D array (x fastest) with the given box.
cudaError_t encodeMap(CUtensorMap* m, const void* base, CUtensorMapDataType type, unsigned esize, const Dim3i& cg,
                      unsigned bx, unsigned by) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    encode = (Encode)fn;
  }
  cuuint64_t dims[3] = {(cuuint64_t)cg.x, (cuuint64_t)cg.y, (cuuint64_t)cg.z};
  cuuint64_t strides[2] = {(cuuint64_t)cg.x * esize, (cuuint64_t)cg.x * cg.y * esize};
  cuuint32_t box[3] = {bx, by, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(m, type, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
}  // namespace

cudaError_t makeHaloMap(const Dim3i& cg, const float* v, CUtensorMap* m) {
  return encodeMap(m, v, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, cg, FW, FH);
}

cudaError_t makeCgMaps(const Dim3i& cg, const CgCode* code, const float* r, const void* x, bool xDouble,
                       const float* p0, const float* p1, CgMaps* m) {
  if (cg.x % 16 != 0) return cudaErrorInvalidValue;  // rows of 8-bit codes must start on 16-byte boundaries
  cudaError_t e;
  if ((e = encodeMap(&m->codeH, code, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, cg, CW, FH)) != cudaSuccess) return e;
  if ((e = encodeMap(&m->codeI, code, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, cg, CTX, CTR)) != cudaSuccess) return e;
  if ((e = encodeMap(&m->rH, r, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, cg, FW, FH)) != cudaSuccess) return e;
  if ((e = encodeMap(&m->rI, r, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, cg, CTX, CTR)) != cudaSuccess) return e;
  if ((e = encodeMap(&m->xI, x, xDouble ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                     xDouble ? 8 : 4, cg, CTX, CTR)) != cudaSuccess)
    return e;
  if ((e = encodeMap(&m->pH[0], p0, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, cg, FW, FH)) != cudaSuccess) return e;
  return encodeMap(&m->pH[1], p1, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, cg, FW, FH);
}

void cgWarmLaunchCache() {
  residentBlocks((const void*)kCgDirection<0>);
  residentBlocks((const void*)kCgDirection<1>);
  residentBlocks((const void*)kCgDirection<2>);
  residentBlocks((const void*)kCgUpdate<0, float>);
  residentBlocks((const void*)kCgUpdate<1, float>);
  residentBlocks((const void*)kCgUpdate<2, float>);
  residentBlocks((const void*)kCgUpdate<0, double>);
  residentBlocks((const void*)kCgUpdate<1, double>);
  residentBlocks((const void*)kCgUpdate<2, double>);
}

bool cgResidentEligible(const Dim3i& cg, int precond, bool xDouble) {
  return (precond == 0 || precond == 1) && !xDouble && cgColumns(cg) <= kResCols * RTH && cg.size() < (1ll << 30);
}

namespace {
int residentGrid(const Dim3i& cg) {
  const long long planes = (long long)cgColumns(cg) * cg.z;
  return (int)std::max(1LL, std::min({(planes + kResMinPlanes - 1) / kResMinPlanes, (long long)numSMs(),
                                      (long long)kResGrid}));
}
}  // namespace
// Shared memory of a cluster block: RG kResKL planes of up to 8 segments.
constexpr int kResClusterBytes = (RG * kResKL + 2 * 8) * RPL * 4 + RG * kResKL * CTX * CTR;
namespace {
const void* clusterKernel(int precond) {
  return precond == 1 ? (const void*)kCgResident<1, true> : (const void*)kCgResident<0, true>;
}
}  // namespace
bool cgClusterEligible(const Dim3i& cg, int precond, bool xDouble) {
  // The fluid is seldom more than a quarter of the grid's planes.  A system that
  // turns out too large costs one launch and one host read, 28 us a solve; one
  // that fits gains 1.8 us an iteration at 15 fluid planes, 1.2 at 50, 0.7 at 120
  // and 0.2 beyond 160 (of 6.4 to 8.3 us for the grid)
  if (!cgResidentEligible(cg, precond, xDouble) ||
      (long long)cgColumns(cg) * cg.z > 4LL * kResCluster * RG * kResKL)
    return false;
  int size = 0;
  return clusterSize(clusterKernel(precond), RTH, kResClusterBytes, &size) == cudaSuccess && size > 0;
}
cudaError_t launchCgCluster(const Dim3i& cg, float sx, float sy, float sz, const CgCode* code, float* r, float* x,
                            float* p, float* zG, CgState* st, int precond, const int* sched, int maxIters,
                            cudaStream_t s) {
  auto* k = precond == 1 ? kCgResident<1, true> : kCgResident<0, true>;
  int size = 0;
  cudaError_t e = clusterSize((const void*)k, RTH, kResClusterBytes, &size);
  if (e != cudaSuccess) return e;
  const long long planes = (long long)cgColumns(cg) * cg.z;
  while (size > 1 && (long long)(size / 2) * kResMinPlanes >= planes) size /= 2;
  ResArgs A{cg, sx, sy, sz, code, r, x, p, zG, nullptr, st, maxIters};
  return launchCluster(k, size, RTH, kResClusterBytes, s, A, sched, cgColumns(cg), kResClusterBytes);
}
namespace {
constexpr size_t mailboxBytes(size_t blocks) { return 2 * blocks * 2 * blocks * sizeof(Tagged); }
}  // namespace
size_t cgResidentBytes(const Dim3i& cg) { return mailboxBytes(residentGrid(cg)); }
size_t cgResidentBytesMost() { return mailboxBytes(kResGrid); }

cudaError_t launchCgResident(const Dim3i& cg, float sx, float sy, float sz, const CgCode* code, float* r, float* x,
                             float* p, float* zG, void* mailboxes, CgState* st, int precond, const int* sched,
                             int maxIters, cudaStream_t s) {
  const void* k = precond == 1 ? (const void*)kCgResident<1, false> : (const void*)kCgResident<0, false>;
  int dev = 0, optin = 0;
  cudaFuncAttributes fa{};
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return e;
  int dynBytes = (optin - (int)fa.sharedSizeBytes) & ~15;
  if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, dynBytes)) != cudaSuccess) return e;
  int cols = cgColumns(cg);
  const int grid = residentGrid(cg);
  // the tags of an earlier launch must not look like this one's
  if ((e = cudaMemsetAsync(mailboxes, 0, cgResidentBytes(cg), s)) != cudaSuccess) return e;
  ResArgs A{cg, sx, sy, sz, code, r, x, p, zG, static_cast<Tagged*>(mailboxes), st, maxIters};
  void* args[] = {&A, (void*)&sched, &cols, &dynBytes};
  return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(RTH), args, (size_t)dynBytes, s);
}

namespace {
__global__ void kZeroOffFluid(long long n, const CgCode* __restrict__ code, float* __restrict__ x) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
    if (!(code[c] & 1)) x[c] = 0.f;
}
}  // namespace
cudaError_t launchZeroOffFluid(const Dim3i& cg, const CgCode* code, float* x, cudaStream_t s) {
  kZeroOffFluid<<<(unsigned)std::min((cg.size() + 255) / 256, 8LL * numSMs()), 256, 0, s>>>(cg.size(), code, x);
  return cudaGetLastError();
}

int cgScheduleTarget(int precond, bool xDouble) {
  int per = kSchedPerSM;
  auto take = [&](const void* k) { per = std::min(per, residentBlocks(k)); };
  if (precond == 1) {
    take((const void*)kCgDirection<1>);
    take(xDouble ? (const void*)kCgUpdate<1, double> : (const void*)kCgUpdate<1, float>);
  } else if (precond == 2) {
    take((const void*)kCgDirection<2>);
    take(xDouble ? (const void*)kCgUpdate<2, double> : (const void*)kCgUpdate<2, float>);
  } else {
    take((const void*)kCgDirection<0>);
    take(xDouble ? (const void*)kCgUpdate<0, double> : (const void*)kCgUpdate<0, float>);
  }
  return numSMs() * std::max(1, per);
}

int cgScheduleInts(const Dim3i& cg) {
  const int cols = cgColumns(cg);
  return schedItemsOffset(cols) + 4 * (numSMs() * kSchedPerSM + cols);
}

int cgPartialsNeeded(const Dim3i& r) {
  const Dim3i cg = cgDims(r);
  CgGrid g = cgGrid(cg);
  long long n = (long long)g.grid.x * g.grid.y * g.grid.z;
  // the CG kernels, at the shortest z chunk any launch shape (tuned or not) uses
  const long long tiles = (long long)((cg.x + CTX - 1) / CTX) * ((cg.y + CTR - 1) / CTR);
  n = std::max(n, tiles * ((cg.z + std::min(3, cg.z) - 1) / std::min(3, cg.z)));
  n = std::max(n, (long long)numSMs() * kSchedPerSM + tiles);  // a schedule's grid
  return 2 * (int)n;
}

cudaError_t launchCgDirection(const Dim3i& cg, float sx, float sy, float sz, const CUtensorMap& mZ,
                              const CUtensorMap& mPo, const CUtensorMap& mCode, const CgCode* code, const float* zr,
                              const float* pOld, float* pNew, double* partials, CgState* st, int precond,
                              cudaStream_t s, const int* colZ, bool xDouble) {
  switch (precond) {
    case 1: {
      CgLaunch L = cgLaunch(cg, kCgDirection<1>, 0, colZ, 1, xDouble);
      cudaError_t e = launchPdl(kCgDirection<1>, L.grid, L.block, s, mZ, mPo, mCode, cg, sx, sy, sz, code, zr, pOld,
                                pNew, partials, st, L.zPer, colZ);
      if (e != cudaSuccess) return e;
      break;
    }
    case 2: {
      if (cg.size() <= kCgSmallGrid)
        return launchPdl(kCgDirectionSmall, dim3(smallBlocks(cg)), dim3(kSmallThreads), s, cg, sx, sy, sz, code, zr, pOld,
                         pNew, partials, st);
      CgLaunch L = cgLaunch(cg, kCgDirection<2>, 0, colZ, 2, xDouble);
      cudaError_t e = launchPdl(kCgDirection<2>, L.grid, L.block, s, mZ, mPo, mCode, cg, sx, sy, sz, code, zr, pOld,
                                pNew, partials, st, L.zPer, colZ);
      if (e != cudaSuccess) return e;
      break;
    }
    default: {
      CgLaunch L = cgLaunch(cg, kCgDirection<0>, 0, colZ, 0, xDouble);
      cudaError_t e = launchPdl(kCgDirection<0>, L.grid, L.block, s, mZ, mPo, mCode, cg, sx, sy, sz, code, zr, pOld,
                                pNew, partials, st, L.zPer, colZ);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaGetLastError();
}

cudaError_t launchCgUpdate(const Dim3i& cg, float sx, float sy, float sz, const CUtensorMap& mP, const CUtensorMap& mR,
                           const CUtensorMap& mX, const CUtensorMap& mCode, const CgCode* code, const float* p, void* x, bool xDouble,
                           float* r, double* partials, CgState* st, int precond, cudaStream_t s, const int* colZ) {
  if (precond == 2 && cg.size() <= kCgSmallGrid)
    return xDouble ? launchPdl(kCgUpdateSmall<double>, dim3(smallBlocks(cg)), dim3(kSmallThreads), s, cg, sx, sy, sz,
                               code, p, (double*)x, r, partials, st)
                   : launchPdl(kCgUpdateSmall<float>, dim3(smallBlocks(cg)), dim3(kSmallThreads), s, cg, sx, sy, sz,
                               code, p, (float*)x, r, partials, st);
#define HFG_CG_UPDATE(PCV, TXV)                                                                                   \
  {                                                                                                               \
    CgLaunch L = cgLaunch(cg, kCgUpdate<PCV, TXV>, 1, colZ, PCV, xDouble);                                                             \
    cudaError_t e = launchPdl(kCgUpdate<PCV, TXV>, L.grid, L.block, s, mP, mR, mX, mCode, cg, sx, sy, sz, p,      \
                              (TXV*)x, r, partials, st, L.zPer, colZ);                                        \
    if (e != cudaSuccess) return e;                                                                             \
  }
  if (xDouble) {
    if (precond == 1) HFG_CG_UPDATE(1, double)
    else if (precond == 2) HFG_CG_UPDATE(2, double)
    else HFG_CG_UPDATE(0, double)
  } else {
    if (precond == 1) HFG_CG_UPDATE(1, float)
    else if (precond == 2) HFG_CG_UPDATE(2, float)
    else HFG_CG_UPDATE(0, float)
  }
#undef HFG_CG_UPDATE
  return cudaGetLastError();
}

// Fluid extent of every CG tile column: one block per (column, z slice)
// reduces the fluid planes of its slice; the column's range is their
// min / max (atomics into colZ, set up by the launcher).
__global__ void kFluidColumns(Dim3i cg, const CgCode* __restrict__ code, int zPer, int* colZ) {
  const int x = blockIdx.x * CTX + threadIdx.x, y = blockIdx.y * CTR + threadIdx.y;
  const int z0 = blockIdx.z * zPer, z1 = min(z0 + zPer, cg.z);
  int lo = 0x7fffffff, hi = -1;
  if (x < cg.x && y < cg.y)
    for (int z = z0; z < z1; ++z)
      if (code[((long long)z * cg.y + y) * cg.x + x] & 1) {
        lo = min(lo, z);
        hi = z;
      }
  __shared__ int sl[CTR], sh[CTR];
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (threadIdx.x == 0) { sl[threadIdx.y] = lo; sh[threadIdx.y] = hi; }
  __syncthreads();
  if (threadIdx.y == 0 && threadIdx.x < CTR) {
    lo = __reduce_min_sync(0x0000ffffu, sl[threadIdx.x]);
    hi = __reduce_max_sync(0x0000ffffu, sh[threadIdx.x]);
    if (threadIdx.x == 0 && hi >= 0) {
      const unsigned cols = gridDim.x * gridDim.y, t = blockIdx.y * gridDim.x + blockIdx.x;
      atomicMin(colZ + t, lo);
      atomicMax(colZ + cols + t, hi);
    }
  }
}
int cgColumns(const Dim3i& cg) { return ((cg.x + CTX - 1) / CTX) * ((cg.y + CTR - 1) / CTR); }

// The work items of a schedule from the columns' fluid extents: chunks of
// zLen = max(zMin, ceil(S / target)) planes, S the fluid planes of all active
// columns, so the items are at most target + (active columns); they are
// written column by column, bottom to top.  One block.
constexpr int kListThreads = 1024;
__global__ void __launch_bounds__(kListThreads) kCgWorkList(int cols, int target, int zMin, int capacity, int* sched) {
  const int* lo = sched;
  const int* hi = sched + cols;
  int4* items = reinterpret_cast<int4*>(sched + schedItemsOffset(cols));
  __shared__ unsigned long long total;
  __shared__ int warpTot[kListThreads / 32];
  __shared__ int carry;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) {
    total = 0;
    carry = 0;
  }
  __syncthreads();
  unsigned long long mine = 0;
  for (int c = t; c < cols; c += kListThreads)
    if (hi[c] >= lo[c]) mine += (unsigned long long)(hi[c] - lo[c] + 1);
  atomicAdd(&total, mine);
  __syncthreads();
  const long long S = (long long)total;
  const int zLen = (int)max((long long)zMin, (S + target - 1) / max(target, 1));
  for (int c0 = 0; c0 < cols; c0 += kListThreads) {
    const int c = c0 + t;
    int n = 0, l = 0;
    if (c < cols && hi[c] >= lo[c]) {
      l = lo[c];
      n = (hi[c] - l + zLen) / zLen;
    }
    int inc = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) warpTot[w] = inc;
    __syncthreads();
    if (w == 0) {
      int x = warpTot[lane], xi = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, xi, d);
        if (lane >= d) xi += y;
      }
      warpTot[lane] = xi - x;
    }
    __syncthreads();
    int k = carry + warpTot[w] + inc - n;
    for (int i = 0; i < n; ++i, ++k) {
      const int z0 = l + i * zLen;
      if (k < capacity) items[k] = make_int4(c, z0, min(z0 + zLen, hi[c] + 1), 0);
    }
    __syncthreads();
    if (t == kListThreads - 1) carry = k;
    __syncthreads();
  }
  // more items than the buffer holds cannot happen (at most target + cols);
  // if it did, a count past the grid makes the CG kernels report error 4
  if (t == 0) sched[2 * cols] = carry;
}

cudaError_t launchCgSchedule(const Dim3i& cg, const CgCode* code, int* sched, int precond, bool xDouble,
                             cudaStream_t s) {
  const int cols = cgColumns(cg);
  cudaError_t e = cudaMemsetAsync(sched, 0x7f, sizeof(int) * cols, s);  // lo: 0x7f7f7f7f, above any plane
  if (e == cudaSuccess) e = cudaMemsetAsync(sched + cols, 0xff, sizeof(int) * cols, s);  // hi: -1
  if (e != cudaSuccess) return e;
  const int zPer = 16;
  dim3 grid((cg.x + CTX - 1) / CTX, (cg.y + CTR - 1) / CTR, (cg.z + zPer - 1) / zPer);
  kFluidColumns<<<grid, dim3(CTX, CTR), 0, s>>>(cg, code, zPer, sched);
  // the shortest chunk: the tuned z-chunk length of the direction kernel, else 3 planes
  const int tuned = tunedZPer(0, cg);
  const int zMin = tuned > 0 ? tuned : std::min(3, cg.z);
  kCgWorkList<<<1, kListThreads, 0, s>>>(cols, cgScheduleTarget(precond, xDouble), zMin,
                                         (cgScheduleInts(cg) - schedItemsOffset(cols)) / 4, sched);
  return cudaGetLastError();
}

}  // namespace hfg
