// hz_ray.cuh -- device code shared by the searches (hz_trace.cu, hz_sweep.cu):
// the ray and the watertight ray/triangle test, FP64 vectors of the cell
// frames, the SVF terms and the domain lookups. Included by each translation
// unit into its own unnamed namespace.
#pragma once

#include <algorithm>

#include "hz_internal.h"

namespace hz {

namespace {

struct Ray {
  float ox, oy, oz;       // origin
  float ix, iy, iz;       // 1 / direction (IEEE)
  float oix, oiy, oiz;    // origin * inverse direction (slab test)
  float pox, poy, poz;    // origin permuted to (kx, ky, kz)
  float plx, ply, plz;    // precise mode: FP32 residual of the origin, permuted
  float Sx, Sy, Sz;       // shear constants
  // Axis order of the shear (kx, ky, kz) and the signs of the inverse
  // direction (n = 1 where negative: near plane = hi), packed in one
  // register: kx | ky << 2 | kz << 4 | nx << 6 | ny << 7 | nz << 8. The
  // persistent search then holds its state in 64 registers without spills.
  unsigned ax;
  __device__ int kx() const { return ax & 3u; }
  __device__ int ky() const { return (ax >> 2) & 3u; }
  __device__ int kz() const { return (ax >> 4) & 3u; }
  __device__ int nx() const { return (ax >> 6) & 1u; }
  __device__ int ny() const { return (ax >> 7) & 1u; }
  __device__ int nz() const { return (ax >> 8) & 1u; }
  float tfar;
};

__device__ __forceinline__ float sel3(float x, float y, float z, int k) {
  return k == 0 ? x : (k == 1 ? y : z);
}

__device__ __forceinline__ Ray make_ray(float ox, float oy, float oz, float dx, float dy,
                                        float dz, float tfar, float lx = 0.f, float ly = 0.f,
                                        float lz = 0.f) {
  Ray r;
  r.ox = ox; r.oy = oy; r.oz = oz;
  r.ix = __frcp_rn(dx); r.iy = __frcp_rn(dy); r.iz = __frcp_rn(dz);
  r.oix = __fmul_rn(ox, r.ix); r.oiy = __fmul_rn(oy, r.iy); r.oiz = __fmul_rn(oz, r.iz);
  const unsigned sx = signbit(r.ix) ? 1u : 0u, sy = signbit(r.iy) ? 1u : 0u,
                 sz = signbit(r.iz) ? 1u : 0u;
  const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  int kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  const float dkz = sel3(dx, dy, dz, kz);
  if (dkz < 0.f) { int tmp = kx; kx = ky; ky = tmp; }
  r.ax = (unsigned)kx | ((unsigned)ky << 2) | ((unsigned)kz << 4) | (sx << 6) | (sy << 7) |
         (sz << 8);
  r.Sx = __fdiv_rn(sel3(dx, dy, dz, kx), dkz);
  r.Sy = __fdiv_rn(sel3(dx, dy, dz, ky), dkz);
  r.Sz = __frcp_rn(dkz);
  r.pox = sel3(ox, oy, oz, kx);
  r.poy = sel3(ox, oy, oz, ky);
  r.poz = sel3(ox, oy, oz, kz);
  r.plx = sel3(lx, ly, lz, kx);
  r.ply = sel3(lx, ly, lz, ky);
  r.plz = sel3(lx, ly, lz, kz);
  r.tfar = tfar;
  return r;
}

// FP64 re-evaluation of the three edge functions when one of them is zero
// (rare). Kept out of line so that the common path carries no FP64 work.
__device__ __noinline__ void edge_functions_fp64(float Ax, float Ay, float Bx, float By,
                                                 float Cx, float Cy, float* U, float* V,
                                                 float* W) {
  *U = __double2float_rn(__dsub_rn(__dmul_rn((double)Cx, (double)By),
                                   __dmul_rn((double)Cy, (double)Bx)));
  *V = __double2float_rn(__dsub_rn(__dmul_rn((double)Ax, (double)Cy),
                                   __dmul_rn((double)Ay, (double)Cx)));
  *W = __double2float_rn(__dsub_rn(__dmul_rn((double)Bx, (double)Ay),
                                   __dmul_rn((double)By, (double)Ax)));
}

// Woop, Benthin & Wald 2013 on origin-relative vertices A, B, C given in the
// ray's (kx, ky, kz) order; hit iff 0 < t <= tfar. Same operation order as
// the oracle (hz_occlusion.h), every operation rounded to nearest.
__device__ __forceinline__ bool tri_hit_rel(const Ray& r, float Akx, float Aky, float Akz,
                                            float Bkx, float Bky, float Bkz, float Ckx,
                                            float Cky, float Ckz) {
  const float Ax = __fsub_rn(Akx, __fmul_rn(r.Sx, Akz));
  const float Ay = __fsub_rn(Aky, __fmul_rn(r.Sy, Akz));
  const float Bx = __fsub_rn(Bkx, __fmul_rn(r.Sx, Bkz));
  const float By = __fsub_rn(Bky, __fmul_rn(r.Sy, Bkz));
  const float Cx = __fsub_rn(Ckx, __fmul_rn(r.Sx, Ckz));
  const float Cy = __fsub_rn(Cky, __fmul_rn(r.Sy, Ckz));
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.f || V == 0.f || W == 0.f) edge_functions_fp64(Ax, Ay, Bx, By, Cx, Cy, &U, &V, &W);
  if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
  const float det = __fadd_rn(__fadd_rn(U, V), W);
  if (det == 0.f) return false;
  const float Az = __fmul_rn(r.Sz, Akz);
  const float Bz = __fmul_rn(r.Sz, Bkz);
  const float Cz = __fmul_rn(r.Sz, Ckz);
  const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
  const float tmax = __fmul_rn(r.tfar, det);
  if (det > 0.f) return T > 0.f && T <= tmax;
  return T < 0.f && T >= tmax;
}

// Reference arithmetic: FP32 vertices minus the FP32 origin in the domain's
// global ENU frame (mo_lradtopo_horayzon.cpp:403-410, 715-720). X, Y, Z are
// the triangle's (kx, ky, kz) axes: (v0, v1, v2) components of each.
__device__ __forceinline__ bool tri_hit(const Ray& r, const float4 X, const float4 Y,
                                        const float4 Z) {
  return tri_hit_rel(r, __fsub_rn(X.x, r.pox), __fsub_rn(Y.x, r.poy), __fsub_rn(Z.x, r.poz),
                     __fsub_rn(X.y, r.pox), __fsub_rn(Y.y, r.poy), __fsub_rn(Z.y, r.poz),
                     __fsub_rn(X.z, r.pox), __fsub_rn(Y.z, r.poy), __fsub_rn(Z.z, r.poz));
}

// Precise arithmetic: vertices and origin as FP32 hi + lo pairs (~48-bit
// FP64 values); the origin-relative vector (hi - o_hi) + (lo - o_lo) is
// accurate to FP32 relative to its own length, i.e. centimetres become
// micrometres for the triangles next to the cell. LX, LY, LZ: the residuals.
__device__ __forceinline__ float rel(float vh, float vl, float oh, float ol) {
  return __fadd_rn(__fsub_rn(vh, oh), __fsub_rn(vl, ol));
}
__device__ __forceinline__ bool tri_hit_hl(const Ray& r, const float4 X, const float4 Y,
                                           const float4 Z, const float4 LX, const float4 LY,
                                           const float4 LZ) {
  return tri_hit_rel(r, rel(X.x, LX.x, r.pox, r.plx), rel(Y.x, LY.x, r.poy, r.ply),
                     rel(Z.x, LZ.x, r.poz, r.plz), rel(X.y, LX.y, r.pox, r.plx),
                     rel(Y.y, LY.y, r.poy, r.ply), rel(Z.y, LZ.y, r.poz, r.plz),
                     rel(X.z, LX.z, r.pox, r.plx), rel(Y.z, LY.z, r.poy, r.ply),
                     rel(Z.z, LZ.z, r.poz, r.plz));
}

// Triangle k's axes in the ray's (kx, ky, kz) order (Tri: one float4 per
// axis), and the same for the precise residuals.
__device__ __forceinline__ void load_tri(const Tri* __restrict__ tris, const Ray& r, int k,
                                         float4& X, float4& Y, float4& Z) {
  const float4* t = reinterpret_cast<const float4*>(tris + k);
  X = __ldg(t + r.kx());
  Y = __ldg(t + r.ky());
  Z = __ldg(t + r.kz());
}

// Conservative slab test: the boxes carry a margin far above the rounding of
// these multiply-adds, so no triangle the watertight test would hit is culled.
// Each axis' near and far plane is chosen by the sign of the inverse
// direction (near = lo where it is positive). For a finite inverse direction
// the entry / exit distances equal the min / max of the two planes'; for an
// infinite one (a zero direction component) they are NaN or infinite, and the
// NaN-skipping fminf / fmaxf then leave the axis unconstrained unless the
// parallel ray lies outside the slab.
__device__ __forceinline__ bool box_hit_nf(const Ray& r, float nx, float fx, float ny, float fy,
                                           float nz, float fz, float& tentry) {
  const float tn = fmaxf(fmaxf(__fmaf_rn(nx, r.ix, -r.oix), __fmaf_rn(ny, r.iy, -r.oiy)),
                         fmaxf(__fmaf_rn(nz, r.iz, -r.oiz), 0.f));
  float tf = fminf(fminf(__fmaf_rn(fx, r.ix, -r.oix), __fmaf_rn(fy, r.iy, -r.oiy)),
                   __fmaf_rn(fz, r.iz, -r.oiz));
  tf = fminf(__fmul_rn(tf, 1.00000072f), r.tfar);
  tentry = tn;
  return tn <= tf;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

struct V3 {
  double x, y, z;
};

__device__ __forceinline__ double dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross3(V3 a, V3 b) {
  return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ void unit3(V3& a) {
  const double m = sqrt(a.x * a.x + a.y * a.y + a.z * a.z);
  a.x /= m;
  a.y /= m;
  a.z /= m;
}
// mo_lradtopo_horayzon.cpp:119-130
__device__ __forceinline__ V3 rotate3(V3 v, V3 k, double s, double c) {
  const double term = dot3(k, v) * (1.0 - c);
  V3 r;
  r.x = v.x * c + (k.y * v.z - k.z * v.y) * s + k.x * term;
  r.y = v.y * c + (k.z * v.x - k.x * v.z) * s + k.y * term;
  r.z = v.z * c + (k.x * v.y - k.y * v.x) * s + k.z * term;
  return r;
}

#ifndef HZ_CHECKED
#define HZ_CHECKED 0  // 1: the search checks its indices and records violations (kErrBounds)
#endif
// What a checked build checks. Tree search: a node reference against the tree's
// nodes, a leaf's triangle range against its triangles; both: an output row / cell.
// Profile sweep: a triangle's number, a list (its start and its entries), a grid or
// pyramid cell, a lattice elevation against its table, a slot of the warp's
// triangle queue, a cell's work position, a result code's slot; and that the error
// bound of a cell's triangles covers each of their vertices.
enum : int { kCheckNode = 1, kCheckLeaf = 2, kCheckOutput = 3, kCheckTriangle = 4, kCheckList = 5,
             kCheckGrid = 6, kCheckElevation = 7, kCheckQueue = 8, kCheckPosition = 9,
             kCheckSlot = 10, kCheckBound = 11 };

// In checked builds: records the first failed check (code, index) in err[1],
// err[2] and raises kErrBounds; the caller then skips the access. err[3] holds a
// bit for every kind of check made. Without HZ_CHECKED every check passes and
// compiles away.
__device__ __forceinline__ bool check_ok(bool ok, int code, long long index, int* err) {
#if HZ_CHECKED
  if (!(*(volatile int*)(err + 3) >> code & 1)) atomicOr(err + 3, 1 << code);
  if (!ok) {
    if (atomicCAS(err + 1, 0, code) == 0) err[2] = (int)index;
    atomicOr(err, kErrBounds);
  }
  return ok;
#else
  (void)code;
  (void)index;
  (void)err;
  return true;
#endif
}

// One ray/triangle test of triangle k (kPrecise: hi + lo vertices).
template <bool kPrecise>
__device__ __forceinline__ bool test_tri(const Tri* __restrict__ tris,
                                         const float4* __restrict__ tri_lo, const Ray& r, int k) {
  float4 X, Y, Z;
  load_tri(tris, r, k, X, Y, Z);
  if (kPrecise) {
    const float4* l = tri_lo + 3LL * k;
    return tri_hit_hl(r, X, Y, Z, __ldg(l + r.kx()), __ldg(l + r.ky()), __ldg(l + r.kz()));
  }
  return tri_hit(r, X, Y, Z);
}

// One azimuth's SVF term for sin(h) = s (cpp:333-358).
__device__ __forceinline__ double svf_term(double s, int svf_type) {
  if (svf_type == 0) return 1.0 - s;
  if (svf_type == 1) return 1.0 - (s * s);
  return 1.0 - (s * s * s);
}

// SVF term of a clipped horizon h ~ j * hori_acc: 1 for h = 0 (sin 0 = 0),
// the tabulated term of the lattice value, or computed off the table.
__device__ __forceinline__ double lattice_svf_term(const DomainDesc& D, double h, int j) {
  if (!(h > 0.0)) return 1.0;
  if (j > 0 && j < kSvfTable) return __ldg(&D.svf_lattice[j]);
  return svf_term(sin(h), D.svf_type);
}

// RN(v / pi) without a division, by Markstein's correction for a divisor
// known in advance (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990): y =
// RN(1 / pi) lies within 0.131 ulp of 1 / pi, so for a normal v >= 0
// q0 = RN(v * y) is within 0.206 + 0.5 ulp of v / pi, a faithful quotient;
// its remainder r = v - q0 * pi is then exact in one FMA, and RN(q0 + r * y)
// is the correctly rounded quotient, the value of v / pi. The search's sums
// are 0 or at least 0.25 deg, far from the subnormal range.
__device__ __forceinline__ double div_pi_rn(double v) {
  const double q0 = __dmul_rn(v, kInvPi);
  const double r = __fma_rn(-q0, kPi, v);
  return __fma_rn(r, kInvPi, q0);
}

// The epilogue's SVF term of a clipped horizon v (0, or at least 0.25 deg on
// the lattice v ~ j * hori_acc, j < kSvfTable in practice), with integer and
// FP32 operations where the search's form uses FP64 ones: v > 0 from the
// exponent bits, and j from an FP32 copy of v truncated to its top 20
// mantissa bits (relative error < 2^-20, so |f / hori_acc - j| < 0.01).
__device__ __forceinline__ double finish_svf_term(const DomainDesc& D, double v, float inv_ha) {
  const int hi = __double2hiint(v);
  const int e = (hi >> 20) & 0x7ff;
  if (hi < 0 || e == 0) return 1.0;  // v == 0 (the clip leaves no negatives)
  const int fe = e - 1023 + 127;
  if (fe <= 0 || fe >= 255) return svf_term(sin(v), D.svf_type);
  const float f = __int_as_float((fe << 23) | ((hi & 0xfffff) << 3));
  const int j = __float2int_rn(f * inv_ha);
  if (j > 0 && j < kSvfTable) return __ldg(&D.svf_lattice[j]);
  return svf_term(sin(v), D.svf_type);
}

// Domain of work id g (doms sorted by cell_offset).
__device__ __forceinline__ int domain_of(const DomainDesc* __restrict__ doms, int ndom,
                                         long long g) {
  int lo = 0, hi = ndom - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (doms[mid].cell_offset <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A warm-start lattice index within [-85, +90] deg.
__device__ __forceinline__ int clamp_start(int m) {
  return m < kMlpStartMin ? kMlpStartMin : (m > kMlpStartMax ? kMlpStartMax : m);
}

// Domain of search item k (doms sorted by item_begin).
__device__ __forceinline__ int domain_of_item(const DomainDesc* __restrict__ doms, int ndom,
                                              long long k) {
  int lo = 0, hi = ndom - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (doms[mid].item_begin <= k) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

#ifndef HZ_CARVEOUT
#define HZ_CARVEOUT 1  // 1: ask for the smallest shared-memory carveout that holds the blocks
#endif

// Shared memory is carved out of the SM's 256 KB of L1: ask for just what
// `resident` blocks need, so the rest caches the tree.
template <typename K>
inline void prefer_l1(K kernel, int resident) {
#if HZ_CARVEOUT
  cudaFuncAttributes fa;
  int dev = 0, smem_sm = 0, reserved = 0;
  if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) !=
          cudaSuccess ||
      cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) !=
          cudaSuccess ||
      smem_sm <= 0) {
    (void)cudaGetLastError();
    return;
  }
  const long long need = (long long)resident * ((long long)fa.sharedSizeBytes + reserved);
  const int pct = (int)std::min<long long>(100, (need * 100 + smem_sm - 1) / smem_sm);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct) !=
      cudaSuccess)
    (void)cudaGetLastError();
#else
  (void)kernel;
  (void)resident;
  (void)dynamic;
#endif
}

}  // namespace

}  // namespace hz
