// hz_sweep.cu -- the horizon search as one profile sweep per (cell, azimuth).
//
// The reference tests the horizon of an azimuth with one ray per elevation
// step (mo_lradtopo_horayzon.cpp:490-555). All rays of one (cell, azimuth)
// lie in the plane through the ray origin, the azimuth's horizontal direction
// and the cell's normal, and the normal points away from the Earth's centre:
// the plane contains the centre. In the gnomonic projection from the centre
// (X = R x / z, Y = R y / z in the domain's ENU axes, origin at the centre)
// such a plane is one straight line, the same for every elevation. So the
// rays of an azimuth share one track over a regular X/Y grid, and terrain
// hides a ray exactly where its height above the sphere exceeds the ray's.
//
//   * grid build: the triangles of each grid cell (counting, scan, fill) with
//     upper and lower bounds of their heights inside the cell, and a pyramid
//     of the cells' bounds (every second level, 4 x 4 children), the upper ones
//     as planes too;
//   * k_sweep: walks the track front to back at the elevation of the lowest
//     ray not yet known to be hidden, skipping every pyramid cell that lies
//     below it. A triangle that hides the ray raises the elevation, and the
//     walk goes on from there: what was skipped or passed lies below every
//     higher ray of the plane, so nothing is walked twice. It ends with the
//     lowest lattice elevation m that misses, every lattice ray from the
//     sweep's start up to m - 1 known to hit, every one from m up known to
//     miss: the hit pattern that the reference's bracketing search asks for,
//     whatever elevation it starts from;
//   * k_sweep_repair: azimuths whose hits are not one run of elevations (a
//     cell that looks under the edge of the mesh, a ray that ends in mid-air
//     at dist_search) are searched ray by ray as the reference does, a warp
//     per cell and 32 elevations at a time;
//   * k_sweep_finish: replays the reference's search of every cell on the hit
//     patterns (its carried elevation, its accumulation of 0.5 deg steps, its
//     ray count) and writes degrees and sky view factors.
//
// Exactness: hit decisions are those of the watertight FP32 test of the same
// FP32 rays. The sweep's own classification of a triangle (below the ray,
// beside the plane, hit) uses FP32 distances from the plane with error bounds
// and decides only what lies outside them; anything nearer is put to the
// watertight test itself (exact_hit), and a triangle that stays above an
// unhidden ray hands the azimuth to k_sweep_repair.
//
// Against the tree search (GB300, whole call): one traversal of a bounding
// volume tree per ray took 2.5 to 4 rays, 63 to 126 four-wide node visits and 38
// to 76 triangle tests per evaluation; the sweep takes 40 to 66 eight-byte steps and
// 15 to 23 tests. 500 m, 3.1M cells 132 -> 60.7 ms; 100 m, 1.2M cells 117 -> 39.2 ms; 2.5 km,
// 57k cells 7.7 -> 1.38 ms; 500 cells 5.2 -> 0.64 ms; 360 azimuths, 21k cells 56.0 -> 10.0 ms.
// The small domains gain most: a sweep from a low start needs no other azimuth's
// result, so a cell's azimuths run side by side.
//
// What bounds it: instruction issue (63 % of the cycles at 18.0 of 32 lanes, 640 warp
// instructions per evaluation) and L1/L2 latency with 24 resident warps per SM; DRAM
// is idle (0.7 %).
#include <cuda_fp16.h>

#include <algorithm>

#include "hz_internal.h"
#include "hz_ray.cuh"

namespace hz {

namespace {

constexpr int kSweepBlock = 128;
// Resident blocks per SM: 6 of 80 registers (1.2M cells at 100 m: 70.6 ms with 5, 67.4
// with 6, spills from 7 on: 31 ms against 26 of a 300 km domain); 5 of 96 for the
// FP64 ray mode (10.0 ms, 11.6 with 6).
#ifndef HZ_SWEEP_MIN_BLOCKS
#define HZ_SWEEP_MIN_BLOCKS 6
#endif
#ifndef HZ_SWEEP_MIN_BLOCKS_EXACT
#define HZ_SWEEP_MIN_BLOCKS_EXACT 5
#endif
// Pyramid steps per lane in one walk pass (6: +0.7 %, 11: the same); of 32 live
// lanes, those that must still walk for the pass to go on (9: +0.6 %, 15: the same)
// and those that must wait before azimuths are set up (57k cells: 3 1.08 ms, 5 1.06, 7
// 1.03, 8 1.03; 1.2M cells 39.1, 38.7, 38.8, 39.0); a grid cell's area in mean triangle
// areas (0.8 and 1.25 within 1 %, 2.2 +5 %).
#ifndef HZ_WALK_STEPS
#define HZ_WALK_STEPS 8
#endif
#ifndef HZ_WALK_MIN
#define HZ_WALK_MIN 14
#endif
#ifndef HZ_SWEEP_ADVANCE
#define HZ_SWEEP_ADVANCE 7
#endif
#ifndef HZ_CELL_TRIS
#define HZ_CELL_TRIS 1.0f
#endif

constexpr float kRf = 6371229.0f;         // kEarthRadius, exact in FP32
// Bound of the error of a vertex's FP32 distances from the plane and over the
// ray, over its distance (1-norm) from the origin: with u = 2^-24, 12 u of the
// sweep's own (axes 5 u a component, coordinates u, sums 3 u) and 7 u of the
// watertight test (sheared coordinates 6 u, direction 1 u).
constexpr float kEps = 1.28e-6f;
// The same over a bound of the distance: the 1-norm is up to sqrt(3) times the
// length in the domain's axes. A vertex of a triangle in a cell that the walk
// leaves at the horizontal distance x lies within (1 + tan(psi / 2)) x <= 1.04 x
// (the axes turn by psi <= 0.08) and GridDesc::dadd + the longest edge.
constexpr float kEpsCell = 1.7321f * kEps, kDropCell = 1.04f;
constexpr float kMagic = 8388608.0f;      // 2^23: float(2^23 | n) = 2^23 + n
constexpr int kTanRange = 180;            // lattice elevations with a tangent: |m| < 180
constexpr int kMaxM = 177;                // sweeps stop below 89 deg
// A sweep that nothing met starts over kLower steps lower, then twice that, then
// from the floor; a run's first azimuth, whose start is well below any horizon
// of its neighbourhood, from the floor at once: it looks over the mesh's edge.
// Against the floor after one lower start (there every elevation up to the
// horizon is a raise): 1.2M cells at 100 m 49.4 -> 45.0 ms, 500 cells 0.98 -> 0.70;
// with the two lower starts for first azimuths too 0.76. Third lower starts: no gain.
constexpr int kLower = 4, kLowerTries = 2;
constexpr int kRunStart = -14;            // start of a run's first azimuth (-7 deg)

// Codes of a (cell, azimuth): the lowest missing lattice elevation, or
constexpr int kCodeAllMiss = -20000;      // no lattice ray meets the terrain
constexpr int kCodeGap = -20001;          // left to k_sweep_repair
constexpr int kCodeStop = 10000;          // + ((m + 2000) << 1 | up): the search's stop itself
constexpr int kMaxStop = (32767 - kCodeStop) / 2 - 2000;  // highest m that 16 bits hold

__device__ __forceinline__ float height_magic(unsigned h16) {
  return __uint_as_float(0x4B000000u | h16);
}

// ---------------------------------------------------------------------------
// Grid build
// ---------------------------------------------------------------------------
// 9.4M triangles, ms: k_gnomonic 0.15, k_grid_count 0.47, k_grid_fill 0.63 (a scattered
// atomic and an 8-byte store per list entry, 4.8 a triangle), k_grid_heights 0.55
// (scattered vertex reads), k_grid_up 0.13; the tree build that this replaces
// took 2.4 in all.

// Gnomonic X, Y and height above the sphere of every mesh vertex, and their
// bounds (ordered keys): min X, Y, H, z; max X, Y, H. The height is (r^2 -
// R^2) / (r + R) with the numerator in FP64 (it cancels), good to 1e-3 m.
__global__ void k_gnomonic(const float* __restrict__ vert, int n, float4* __restrict__ gv,
                           unsigned* __restrict__ bounds) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  float X = 0.f, Y = 0.f, H = 0.f, z = 0.f;
  if (valid) {
    const float x = vert[3LL * i], y = vert[3LL * i + 1], zz = vert[3LL * i + 2];
    const double dx = x, dy = y, dz = zz;
    const double r2 = dx * dx + dy * dy + dz * (dz + 2.0 * kEarthRadius);
    z = (float)(dz + kEarthRadius);
    const float f = __fdiv_rn(kRf, z);
    X = x * f;
    Y = y * f;
    const float num = (float)r2;
    H = __fdiv_rn(num, sqrtf((float)(kEarthRadius * kEarthRadius + r2)) + kRf);
    gv[i] = make_float4(X, Y, H, 0.f);
  }
  const unsigned no = 0xFFFFFFFFu;
  unsigned b[7] = {valid ? f2ord(X) : no, valid ? f2ord(Y) : no, valid ? f2ord(H) : no,
                   valid ? f2ord(z) : no, valid ? f2ord(X) : 0u, valid ? f2ord(Y) : 0u,
                   valid ? f2ord(H) : 0u};
  block_bounds_atomic<4, 3>(b, bounds);
}

__global__ void k_grid_init(unsigned* b) {
  for (int k = 0; k < 4; k++) b[k] = 0xFFFFFFFFu;
  for (int k = 4; k < 8; k++) b[k] = 0u;
}

// Holes: a cell beside an ICON vertex without its triangles looks under the
// mesh's edge in half of its azimuths, and the repair searches those ray by ray, a
// warp per cell. A domain without holes has few such cells, at its border. A vertex
// missing inside costs 0.15 us (10 km spacing) to 2.3 us (0.2 km) at 24 azimuths; the
// tree search takes 20 to 60 ns per cell more than the sweep and some 5 to 10 ms per
// call. Times of the tree over those of the sweep, radius 40 km, vertices missing: 0.2 km,
// 141k cells 1.7 at 2,100, 0.94 at 7,000, 0.5 at 21,000; 1.4M cells 1.5 at 7,100, 0.93 at
// 21,000, 0.4 at 70,000; 1 km, 423k cells 1.65 at 6,300, 0.91 at 21,000; 1.4M cells 2.1 at
// 21,000, 1.2 at 71,000; 2.5 km and more: 1.6 and more with a tenth of them missing. So the
// tree search takes over where the missing vertices of a call are more than
// kHolesCall and its cells over kHolesCells, those times the size of the grid's
// cells over kHolesSize metres where that is larger. They are counted from the
// triangles that the cells lack, at most a quarter of the cells at an edge of the
// mesh (a hole has six, a third of all vertices missing four each): parts of a domain
// without any triangles cost little.
constexpr float kHolesCall = 6000.f, kHolesCells = 90.f, kHolesSize = 190.f;
// Holes of the domains of a call, in err: their sum over what the cells allow, the
// domains summed.
enum : int { kErrHoles = 4, kErrHolesDomains = 5 };

// ICON vertices of each cell with all their cells.
__global__ void k_full_vertices(const int* __restrict__ cov, int nvert,
                                uint32_t* __restrict__ full) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nvert) return;
  int c[6];
  for (int k = 0; k < 6; k++) c[k] = cov[(long long)k * nvert + v];
  for (int k = 0; k < 6; k++)
    if (c[k] < 0) return;
  for (int k = 0; k < 6; k++) atomicAdd(&full[c[k]], 1u);
}
__global__ void k_edge_cells(const uint32_t* __restrict__ full, int begin, int count,
                             int* __restrict__ edge) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const bool at = k < count && full[begin + k] > 0u && full[begin + k] < 3u;
  const unsigned n = __popc(__ballot_sync(0xffffffffu, at));
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(edge, (int)n);
}

// Grid geometry: cells of HZ_CELL_TRIS times the mean triangle area. missing:
// vertices missing beside the cells that are searched.
__global__ void k_grid_setup(const unsigned* __restrict__ b, int n_tri, long long cap0, float tfar,
                             float org_elev, float cells, float missing,
                             const int* __restrict__ edge, int ndom, GridDesc* __restrict__ g, int* __restrict__ err) {
  GridDesc q;
  const float x0 = ord2f(b[0]), y0 = ord2f(b[1]), h0 = ord2f(b[2]), z0 = ord2f(b[3]);
  const float x1 = ord2f(b[4]), y1 = ord2f(b[5]), h1 = ord2f(b[6]);
  const float ex = fmaxf(x1 - x0, 1.f), ey = fmaxf(y1 - y0, 1.f);
  const float big = fmaxf(fmaxf(fabsf(x0), fabsf(x1)), fmaxf(fabsf(y0), fabsf(y1)));
  float c = sqrtf(ex * ey * HZ_CELL_TRIS / (float)(n_tri > 0 ? n_tri : 1));
  // (Sums of 65,535 domains stay within 32 bits.)
  if (edge) missing = fminf(missing, (float)*edge * 0.25f);
  const float holes = missing - cells / kHolesCells * fmaxf(1.f, c / kHolesSize);
  atomicAdd(&err[kErrHoles], (int)fminf(fmaxf(holes, -30000.f), 30000.f));
  __threadfence();
  if (atomicAdd(&err[kErrHolesDomains], 1) == ndom - 1 &&
      (float)atomicAdd(&err[kErrHoles], 0) > kHolesCall)
    atomicOr(err, kErrGrid);
  c = fminf(fmaxf(c, fmaxf(ex, ey) * 6e-5f), 1e6f);  // at most ~16,000 cells a side
  // Domains the projection cannot hold (a vertex 60 deg or more from the
  // centre's axis) or inputs that are not finite.
  bool ok = z0 > 0.5f * kRf && isfinite(ex) && isfinite(ey) && isfinite(h0) && isfinite(h1) &&
            h1 - h0 < 2e5f && h0 > -1e5f && isfinite(c);
  int W = 1, H = 1, L = 0;
  float pad = 0.f;
  for (int it = 0; ok; it++) {
    pad = 3e-6f * big + 1e-6f * tfar + 2e-3f * c + 0.02f;
    const int nx = (int)((ex + 3.f * pad) / c) + 2, ny = (int)((ey + 3.f * pad) / c) + 2;
    L = 0;
    while (L < 8 && (min(nx, ny) >> (L + 2)) >= 2) L += 2;
    const int r = (4 << L) - 1;  // whole bricks at every level
    W = (nx + r) & ~r;
    H = (ny + r) & ~r;
    if ((long long)W * H <= cap0) break;
    c *= 1.1f;
    if (it > 200) ok = false;
  }
  q.c = c;
  q.inv_c = 1.f / c;
  q.pad = pad;
  q.x0 = x0 - 1.5f * pad;
  q.y0 = y0 - 1.5f * pad;
  q.hlo = h0;
  q.iq = 65000.f / (h1 - h0 + 1.f);
  q.unit = (h1 - h0 + 1.f) / 65000.f;
  q.hpad = 0.05f + 2e-6f * tfar;
  q.dadd = 2.f * c + 4.f * pad + (h1 - h0) + org_elev + 1.f;
  q.rlo = kRf + h0;
  q.rhi = kRf + h1;
  q.irlo = 1.f / q.rlo;
  const float s = fminf(tfar / q.rlo, 0.5f);
  q.tau_max = s / sqrtf(1.f - s * s) * 1.0001f;
  // A ray's height over its origin's sphere gains x^2 times these over rlo.
  q.cmin = (q.rlo / q.rhi) * (1.f - 0.25f * q.tau_max * q.tau_max) * 0.5f;
  // x^2 / (r (1 + cos psi)), r >= rlo: at 500 km the cosine alone lifts a ray's
  // height by 30 m against x^2 / 2 rlo.
  q.cmax = (q.rhi / q.rlo) / (1.f + rsqrtf(1.f + 1.01f * q.tau_max * q.tau_max));
  q.W = W;
  q.H = H;
  q.L = L;
  q.lmax = 0u;
  q.heavy = 0u;
  q.boxes = 0ull;
  q.ok = ok ? 1 : 0;
  if (!ok) atomicOr(err, kErrGrid);
  *g = q;
}

// Index of cell (a, b) of level l (even; a = i >> l of level 0's i): a level is
// stored in bricks of 4 x 4 cells, the children of one cell of the level
// above, so that 16 neighbours' planes are one 128-byte line (their level bounds
// 32 bytes); level l begins at n2 - (n2 >> l / 2), n2 twice the cells of level 0.
__device__ __forceinline__ int grid_index(int W, int n2, int a, int b, int l) {
  return n2 - (n2 >> (l >> 1)) + ((((b >> 2) * (W >> (l + 2)) + (a >> 2)) << 4) | ((b & 3) << 2) |
                                  (a & 3));
}

// Calls f(cell index, upper height, lower height) for every grid cell whose
// square, grown by the grid's pad, meets triangle (a, b, c): bounding box,
// then the three edge functions. The heights bound the triangle inside the
// grown cell: its plane over the cell and the bounding box, at most the
// highest vertex. Between its vertices a plane triangle lies lower than the
// linear interpolation of their heights above the sphere, by at most
// edge^2 / 8 R.
struct CellBox {
  int i0, i1, j0, j1;
};
__device__ __forceinline__ CellBox cell_box(const GridDesc& g, float gx0, float gy0, float lx,
                                            float hx, float ly, float hy) {
  return {max(0, (int)floorf((gx0 + lx - g.pad) * g.inv_c)),
          min(g.W - 1, (int)floorf((gx0 + hx + g.pad) * g.inv_c)),
          max(0, (int)floorf((gy0 + ly - g.pad) * g.inv_c)),
          min(g.H - 1, (int)floorf((gy0 + hy + g.pad) * g.inv_c))};
}
template <class F>
__device__ __forceinline__ void for_cells(const GridDesc& g, float4 a, float4 b, float4 c, F f) {
  const float pad = g.pad;
  // Coordinates relative to the first vertex.
  const float bx = b.x - a.x, by = b.y - a.y, cx = c.x - a.x, cy = c.y - a.y;
  const float lx = fminf(0.f, fminf(bx, cx)), hx = fmaxf(0.f, fmaxf(bx, cx));
  const float ly = fminf(0.f, fminf(by, cy)), hy = fmaxf(0.f, fmaxf(by, cy));
  const float hmx = fmaxf(a.z, fmaxf(b.z, c.z)), hmn = fminf(a.z, fminf(b.z, c.z));
  const float gx0 = a.x - g.x0, gy0 = a.y - g.y0;
  const CellBox box = cell_box(g, gx0, gy0, lx, hx, ly, hy);
  const float area = bx * cy - cx * by;
  const float e2 = fmaxf(fmaxf(bx * bx + by * by, cx * cx + cy * cy),
                         (cx - bx) * (cx - bx) + (cy - by) * (cy - by));
  const float sag = e2 / (8.f * kRf) * 1.05f + 0.01f;
  const bool flat = fabsf(area) > 1e-3f * e2;  // gradient usable
  const float ia = 1.f / area;
  const float px = ((b.z - a.z) * cy - (c.z - a.z) * by) * ia;
  const float py = ((c.z - a.z) * bx - (b.z - a.z) * cx) * ia;
  const float sgn = area >= 0.f ? 1.f : -1.f;
  // Edge functions n . (P - vertex) >= 0 inside: edges a-b, b-c, c-a.
  const float n0x = -by * sgn, n0y = bx * sgn;
  const float n1x = (by - cy) * sgn, n1y = (cx - bx) * sgn;
  const float n2x = cy * sgn, n2y = -cx * sgn;
  const float hw = 0.5f * g.c + 1.05f * pad;
  const float s0 = (fabsf(n0x) + fabsf(n0y)) * hw, s1 = (fabsf(n1x) + fabsf(n1y)) * hw,
              s2 = (fabsf(n2x) + fabsf(n2y)) * hw;
  const bool sat = fabsf(area) > 1e-6f * e2;  // else a sliver: its box
  for (int j = box.j0; j <= box.j1; j++) {
    const float y = ((float)j + 0.5f) * g.c - gy0;
    for (int i = box.i0; i <= box.i1; i++) {
      const float x = ((float)i + 0.5f) * g.c - gx0;
      if (sat && (n0x * x + n0y * y + s0 < 0.f ||
                  n1x * (x - bx) + n1y * (y - by) + s1 < 0.f ||
                  n2x * x + n2y * y + s2 < 0.f))
        continue;
      float up = hmx, lo = hmn;
      if (flat) {
        const float xa = fmaxf(lx, x - hw), xb = fminf(hx, x + hw);
        const float ya = fmaxf(ly, y - hw), yb = fminf(hy, y + hw);
        const float u = a.z + px * (px > 0.f ? xb : xa) + py * (py > 0.f ? yb : ya);
        const float v = a.z + px * (px > 0.f ? xa : xb) + py * (py > 0.f ? ya : yb);
        up = fminf(up, u + 0.02f);
        lo = fmaxf(lo, v - 0.02f);
      }
      f(grid_index(g.W, 2 * g.W * g.H, i, j, 0), up, lo - sag);
    }
  }
}

// Cells in a triangle's box.
__device__ __forceinline__ unsigned box_cells(const GridDesc& g, float4 a, float4 b, float4 c) {
  const CellBox box =
      cell_box(g, a.x - g.x0, a.y - g.y0, fminf(0.f, fminf(b.x - a.x, c.x - a.x)),
               fmaxf(0.f, fmaxf(b.x - a.x, c.x - a.x)), fminf(0.f, fminf(b.y - a.y, c.y - a.y)),
               fmaxf(0.f, fmaxf(b.y - a.y, c.y - a.y)));
  return (unsigned)max(0, box.i1 - box.i0 + 1) * (unsigned)max(0, box.j1 - box.j0 + 1);
}

// Most cells in the box of one triangle (a thread goes through them), and in the
// boxes of all per triangle: a proper mesh has some ten, lists hold twelve. Beyond
// them (vertices that join cells from all over the domain) the time of the build would
// grow with the square of the triangles: the call is the tree search's.
constexpr unsigned kMaxBox = 1u << 16, kMaxBoxes = 64u;

// Triangles per cell; also the triangle records (identity order; precise:
// the FP32 residuals too) and the longest edge.
__global__ void k_grid_count(const float* __restrict__ vert, const float* __restrict__ vert_lo,
                             const int* __restrict__ vot, int n, const float4* __restrict__ gv,
                             GridDesc* __restrict__ gd, uint32_t* __restrict__ count,
                             long long cap0, Tri* __restrict__ tris, float4* __restrict__ tri_lo,
                             int* __restrict__ err) {
  __shared__ unsigned smax, boxes, skip;
  if (threadIdx.x == 0) {
    smax = 0u;
    boxes = 0u;
    skip = 0u;
  }
  __syncthreads();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool mine = t < n && gd->ok;
  if (mine) {
    const unsigned k = box_cells(*gd, gv[vot[3LL * t]], gv[vot[3LL * t + 1]], gv[vot[3LL * t + 2]]);
    if (k > kMaxBox) skip = 1u;
    atomicAdd(&boxes, min(k, kMaxBox));
  }
  __syncthreads();
  if (threadIdx.x == 0 &&
      (skip || atomicAdd(&gd->boxes, (unsigned long long)boxes) + boxes >
                   (unsigned long long)kMaxBoxes * n + kMaxBox)) {
    skip = 1u;
    gd->ok = 0;
    atomicOr(err, kErrGrid);
  }
  __syncthreads();
  if (mine && !skip) {
    const GridDesc& g = *gd;
    const int v0 = vot[3LL * t], v1 = vot[3LL * t + 1], v2 = vot[3LL * t + 2];
    const float* p0 = vert + 3LL * v0;
    const float* p1 = vert + 3LL * v1;
    const float* p2 = vert + 3LL * v2;
    Tri r;
    r.x = make_float4(p0[0], p1[0], p2[0], __int_as_float(t));
    r.y = make_float4(p0[1], p1[1], p2[1], 0.f);
    r.z = make_float4(p0[2], p1[2], p2[2], 0.f);
    tris[t] = r;
    if (tri_lo) {
      const float* q0 = vert_lo + 3LL * v0;
      const float* q1 = vert_lo + 3LL * v1;
      const float* q2 = vert_lo + 3LL * v2;
      for (int k = 0; k < 3; k++) tri_lo[3LL * t + k] = make_float4(q0[k], q1[k], q2[k], 0.f);
    }
    auto len2 = [](float x, float y, float z) { return x * x + y * y + z * z; };
    const float e = fmaxf(len2(r.x.y - r.x.x, r.y.y - r.y.x, r.z.y - r.z.x),
                          fmaxf(len2(r.x.z - r.x.x, r.y.z - r.y.x, r.z.z - r.z.x),
                                len2(r.x.z - r.x.y, r.y.z - r.y.y, r.z.z - r.z.y)));
    atomicMax(&smax, __float_as_uint(sqrtf(e)));
    for_cells(g, gv[v0], gv[v1], gv[v2], [&](int cell, float, float) {
      if (check_ok(cell >= 0 && cell < cap0, kCheckGrid, cell, err)) atomicAdd(&count[cell], 1u);
    });
  }
  __syncthreads();
  if (threadIdx.x == 0 && smax) atomicMax(&gd->lmax, smax);
}

// Meshes that fill little of their bounds (patches far apart), or with triangles far
// smaller than the mean (fine patches beside coarse ones): the grid's cells are
// coarse against them, and every visit of one is a long list. Times of the tree over
// those of the sweep by triangles per cell where the terrain is: two patches of 7,600
// cells 3 to 20 deg apart 3.8 at 12, 2.4 at 48, 1.9 at 96, 1.2 at 190, 0.69 at 380 (of 1,200
// cells 2.4 at 100, 1.2 at 210); two of
// 350,000 cells 2.0 at 10, 1.6 at 40, 1.25 at 85, 0.94 at 145; half of 22,700 cells beside
// cells 20 to 100 times as wide 1.8 at 30, 1.3 at 66, 0.94 at 115, 0.63 at 250, 0.27 at 690.
// The tree search takes over where lists longer than this hold entries for more than
// a quarter of the triangles.
constexpr unsigned kHeavyList = 160;

// (triangle, upper | lower height << 16) into each cell's list (triangles are
// numbered through the domains of a call); count runs down from the cell's number of entries.
__global__ void k_grid_fill(const int* __restrict__ vot, int n, int tri_base,
                            const float4* __restrict__ gv, GridDesc* __restrict__ gd,
                            uint32_t* __restrict__ count, const uint32_t* __restrict__ start,
                            long long cap0, uint2* __restrict__ refs, long long cap_refs,
                            int* __restrict__ err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n || !gd->ok) return;
  const GridDesc& g = *gd;
  for (long long k = t; k < (long long)g.W * g.H; k += n) {
    const unsigned length = start[k + 1] - start[k];
    if (length > kHeavyList) atomicAdd(&gd->heavy, length);
  }
  bool over = false;
  for_cells(g, gv[vot[3LL * t]], gv[vot[3LL * t + 1]], gv[vot[3LL * t + 2]],
            [&](int cell, float up, float lo) {
              if (!check_ok(cell >= 0 && cell < cap0, kCheckGrid, cell, err)) return;
              const long long pos = (long long)start[cell] + atomicSub(&count[cell], 1u) - 1;
              if (pos >= cap_refs) {
                over = true;
                return;
              }
              const float u = ceilf((up - g.hlo) * g.iq) + 1.f;
              const float l = floorf((lo - g.hlo) * g.iq);
              const unsigned hu = (unsigned)fminf(fmaxf(u, 1.f), 65535.f);
              const unsigned hl = (unsigned)fminf(fmaxf(l, 0.f), 65535.f);
              refs[pos] = make_uint2((unsigned)(tri_base + t), hu | (hl << 16));
            });
  if (over) atomicOr(err, kErrGrid);
}

// A pyramid cell: an upper bound of the terrain's height over it as a plane,
// height at the cell's centre and gradient per level-0 cell (FP16), in the
// grid's units; empty: far below. A plane lies closer than a level bound
// wherever the terrain slopes: against level bounds the sweeps take 0.79 times the
// steps and look at 0.48 times the lists (100 m, 1.2M cells: search 67.4 -> 50.1 ms;
// 300 km domain at 500 m 26.3 -> 19.1 ms, grid build 0.38 -> 0.49 ms). What it
// carries besides: the rounding of the gradient and of positions (which lie
// within the cell's pad), and the sag size^2 / 4 R of a ray's height, convex along
// the track, below its chord over the cell.
constexpr float kNothing = -1e30f;
__device__ __forceinline__ uint2 pack_plane(const GridDesc& g, int l, float h, float gx, float gy) {
  const float size = g.c * (float)(1 << l), steep = fabsf(gx) + fabsf(gy);
  const float margin = steep * (0.001f * size + 2.f * g.pad) + size * size / (3.9f * kRf) + 0.03f;
  const __half2 grad = __floats2half2_rn(gx * g.iq * g.c, gy * g.iq * g.c);
  return make_uint2(__float_as_uint((h + margin - g.hlo) * g.iq),
                    *reinterpret_cast<const unsigned*>(&grad));
}
__device__ __forceinline__ bool plane_fits(const GridDesc& g, float gx, float gy) {
  const float steep = fabsf(gx) + fabsf(gy);
  return steep < 30.f && steep * g.iq * g.c < 60000.f;  // false for NaN
}

// Level 0: per cell the bounds of its list (empty: 0 and 65535) and the plane,
// its gradient the mean of the triangles', its height the least that is above
// all of them within the cell: each is below its own plane, and below its
// vertices.
__global__ void k_grid_heights(const GridDesc* __restrict__ gd, const uint32_t* __restrict__ start,
                               const uint2* __restrict__ refs, long long cap_refs, int tri_base,
                               const int* __restrict__ vot, const float4* __restrict__ gv,
                               long long cap0, int n_tri, uint16_t* __restrict__ top,
                               uint16_t* __restrict__ low, uint2* __restrict__ planes,
                               int* __restrict__ err) {
  if (!gd->ok) return;
  const GridDesc& g = *gd;
  if (g.heavy > (unsigned)n_tri / 4u) {
    if (threadIdx.x == 0) atomicOr(err, kErrGrid);
    return;
  }
  const long long n0 = (long long)g.W * g.H;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n0 || !check_ok(k < cap0, kCheckGrid, k, err)) return;
  // Cell (i, j) of index k in the brick order.
  const int brick = (int)(k >> 4), wb = g.W >> 2;
  const int i = 4 * (brick % wb) + (int)(k & 3), j = 4 * (brick / wb) + (int)((k >> 2) & 3);
  const float ccx = g.x0 + ((float)i + 0.5f) * g.c, ccy = g.y0 + ((float)j + 0.5f) * g.c;
  const long long q0 = start[k], q1 = min((long long)start[k + 1], cap_refs);
  unsigned hi = 0u, lo = 0xFFFFu;
  float sx = 0.f, sy = 0.f;
  int n = 0;
  auto corners = [&](unsigned tri, float3 (&v)[3]) {
    const int* t = vot + 3LL * ((int)tri - tri_base);
    for (int u = 0; u < 3; u++) {
      const float4 w = gv[t[u]];
      v[u] = make_float3(w.x - ccx, w.y - ccy, w.z);
    }
  };
  auto gradient = [&](const float3 (&v)[3], float& px, float& py) {
    const float bx = v[1].x - v[0].x, by = v[1].y - v[0].y, cx = v[2].x - v[0].x,
                cy = v[2].y - v[0].y, area = bx * cy - cx * by;
    const float ia = 1.f / area;
    px = ((v[1].z - v[0].z) * cy - (v[2].z - v[0].z) * by) * ia;
    py = ((v[2].z - v[0].z) * bx - (v[1].z - v[0].z) * cx) * ia;
    return fabsf(area) > 1e-3f * (bx * bx + by * by + cx * cx + cy * cy) && plane_fits(g, px, py);
  };
  for (long long q = q0; q < q1; q++) {
    const uint2 r = refs[q];
    hi = max(hi, r.y & 0xFFFFu);
    lo = min(lo, r.y >> 16);
    float3 v[3];
    float px, py;
    corners(r.x, v);
    if (gradient(v, px, py)) {
      sx += px;
      sy += py;
      n++;
    }
  }
  if (n) {
    sx /= (float)n;
    sy /= (float)n;
  }
  const float hw = 0.5f * g.c + 1.05f * g.pad;
  float h = kNothing;
  for (long long q = q0; q < q1; q++) {
    float3 v[3];
    float px, py;
    corners(refs[q].x, v);
    float t = kNothing;
    for (int u = 0; u < 3; u++) t = fmaxf(t, v[u].z - sx * v[u].x - sy * v[u].y);
    if (gradient(v, px, py))
      t = fminf(t, v[0].z - px * v[0].x - py * v[0].y + (fabsf(px - sx) + fabsf(py - sy)) * hw);
    h = fmaxf(h, t);
  }
  top[k] = (uint16_t)hi;
  low[k] = (uint16_t)lo;
  planes[k] = q1 > q0 ? pack_plane(g, 0, h, sx, sy) : make_uint2(__float_as_uint(kNothing), 0u);
}

// Level l of the pyramid from level l - 2: a cell's children are one brick.
// Plane: gradient from the children's heights, the least height above every
// child's plane or top within the child.
__global__ void k_grid_up(const GridDesc* __restrict__ gd, int l, long long cap0,
                          uint16_t* __restrict__ top, uint16_t* __restrict__ low,
                          uint2* __restrict__ planes, int* __restrict__ err) {
  if (!gd->ok || l > gd->L) return;
  const GridDesc& g = *gd;
  const int W = g.W, n2 = 2 * W * g.H;
  const int w = W >> l, h = g.H >> l;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)w * h) return;
  const int b = (int)(k / w), a = (int)(k - (long long)b * w);
  const int from = grid_index(W, n2, 4 * a, 4 * b, l - 2), to = grid_index(W, n2, a, b, l);
  if (!check_ok(from >= 0 && from + 16 <= 2 * cap0 && to >= 0 && to < 2 * cap0, kCheckGrid, to,
                err))
    return;
  const float size = g.c * (float)(1 << (l - 2));  // of a child
  unsigned hi = 0u, lo = 0xFFFFu;
  float n = 0.f, mx = 0.f, my = 0.f, mh = 0.f, xx = 0.f, yy = 0.f, xh = 0.f, yh = 0.f;
  for (int q = 0; q < 16; q++) {
    hi = max(hi, (unsigned)top[from + q]);
    lo = min(lo, (unsigned)low[from + q]);
    const float hc = __uint_as_float(planes[from + q].x) * g.unit;
    if (top[from + q] == 0) continue;
    const float x = ((float)(q & 3) - 1.5f) * size, y = ((float)(q >> 2) - 1.5f) * size;
    n += 1.f;
    mx += x; my += y; mh += hc;
    xx += x * x; yy += y * y; xh += x * hc; yh += y * hc;
  }
  const float in = 1.f / fmaxf(n, 1.f);
  float sx = xx - mx * mx * in, sy = yy - my * my * in;
  sx = sx > 0.f ? (xh - mx * mh * in) / sx : 0.f;
  sy = sy > 0.f ? (yh - my * mh * in) / sy : 0.f;
  if (!plane_fits(g, sx, sy)) sx = sy = 0.f;
  float height = kNothing;
  const float hw = 0.5f * size + g.pad, per = g.unit / g.c;
  for (int q = 0; q < 16; q++) {
    if (top[from + q] == 0) continue;
    const uint2 p = planes[from + q];
    const float2 gr = __half22float2(*reinterpret_cast<const __half2*>(&p.y));
    const float x = ((float)(q & 3) - 1.5f) * size, y = ((float)(q >> 2) - 1.5f) * size;
    const float at = sx * x + sy * y;
    const float own = __uint_as_float(p.x) * g.unit +
                      (fabsf(gr.x * per - sx) + fabsf(gr.y * per - sy)) * hw;
    const float level = (float)top[from + q] * g.unit + (fabsf(sx) + fabsf(sy)) * hw;
    height = fmaxf(height, fminf(own, level) - at);
  }
  top[to] = (uint16_t)hi;
  low[to] = (uint16_t)lo;
  planes[to] = hi ? pack_plane(g, l, height + g.hlo, sx, sy)
                  : make_uint2(__float_as_uint(kNothing), 0u);
}

// ---------------------------------------------------------------------------
// Cell frames
// ---------------------------------------------------------------------------

// FP64 frame of a cell (mo_lradtopo_horayzon.cpp:694-720, the expressions of
// the other searches).
struct CellFrame {
  V3 normal, north, east;
  double ox, oy, oz;
};
__device__ __forceinline__ CellFrame cell_frame64(const DomainDesc& D, int cell) {
  CellFrame f;
  const V3 q{D.cell_enu[3LL * cell], D.cell_enu[3LL * cell + 1], D.cell_enu[3LL * cell + 2]};
  f.normal = V3{q.x - D.centre.x, q.y - D.centre.y, q.z - D.centre.z};
  unit3(f.normal);
  const V3 v_n{D.pole.x - q.x, D.pole.y - q.y, D.pole.z - q.z};
  const double dp = dot3(v_n, f.normal);
  f.north = V3{v_n.x - dp * f.normal.x, v_n.y - dp * f.normal.y, v_n.z - dp * f.normal.z};
  unit3(f.north);
  f.east = cross3(f.north, f.normal);
  f.ox = q.x + f.normal.x * D.ray_org_elev;
  f.oy = q.y + f.normal.y * D.ray_org_elev;
  f.oz = q.z + f.normal.z * D.ray_org_elev;
  return f;
}

// FP32 frame table by work position, quadruples of one cell together: origin
// and its height, normal, north and the origin's gnomonic X, east and Y, and
// (precise) the origin's FP32 residual. Lanes set up azimuths of scattered
// cells: four accesses, where one row after another over all cells took 14 (FP64 ray
// mode, 194k cells: 7.15 -> 6.93 ms).
enum : int { kFrameOrigin, kFrameNormal, kFrameNorth, kFrameEast, kFrameRest };
template <bool kPrecise>
__device__ __forceinline__ float4* cell_rows(const DomainDesc& D, long long p) {
  return reinterpret_cast<float4*>(D.cell_f32) + p * (kPrecise ? 5 : 4);
}

// The watertight test of one lattice ray and one triangle, for the few
// triangles the sweep's own arithmetic leaves undecided (p: work position).
// The FP64 frame comes from its table: recomputing it (two square roots and
// six divisions) took more of the FP64 pipe than the whole rest of the sweep.
template <bool kPrecise>
__device__ __forceinline__ Ray table_ray(const DomainDesc& D, int p, int a, double2 ecs) {
  const double* fr = D.cell_frame + 9ll * p;
  const float4* f32 = cell_rows<kPrecise>(D, p);
  const float4 o = __ldg(f32), q = kPrecise ? __ldg(f32 + kFrameRest) : o;
  const double2 cs = __ldg(&D.azim_cs[a]);
  const float dx = (float)(ecs.x * (cs.x * fr[3] + cs.y * fr[6]) + ecs.y * fr[0]);
  const float dy = (float)(ecs.x * (cs.x * fr[4] + cs.y * fr[7]) + ecs.y * fr[1]);
  const float dz = (float)(ecs.x * (cs.x * fr[5] + cs.y * fr[8]) + ecs.y * fr[2]);
  return kPrecise ? make_ray(o.x, o.y, o.z, dx, dy, dz, D.tfar, q.x, q.y, q.z)
                  : make_ray(o.x, o.y, o.z, dx, dy, dz, D.tfar);
}
template <bool kPrecise>
__device__ __noinline__ bool exact_hit(const DomainDesc* D, int p, int a, int m, int tri) {
  // Sweeps stay within kTanRange of the horizontal, well inside the table.
  const Ray r = table_ray<kPrecise>(*D, p, a, __ldg(&D->elev_cs[m - kElevMin]));
  return test_tri<kPrecise>(D->tris, D->tri_lo, r, tri);
}

// FP64 pipe (square roots and divisions): 3.1M cells 0.75 ms, beside the grid build.
template <bool kPrecise>
__global__ void k_sweep_frames(const DomainDesc* __restrict__ doms, int ndom,
                               const int* __restrict__ order, int total) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= total) return;
  const long long gid = order[k];
  const DomainDesc& D = doms[domain_of(doms, ndom, gid)];
  const int cell = (int)(gid - D.cell_offset);
  const long long p = k - D.k_begin;
  const CellFrame f = cell_frame64(D, cell);
  double* fr = D.cell_frame + 9 * p;
  fr[0] = f.normal.x; fr[1] = f.normal.y; fr[2] = f.normal.z;
  fr[3] = f.north.x; fr[4] = f.north.y; fr[5] = f.north.z;
  fr[6] = f.east.x; fr[7] = f.east.y; fr[8] = f.east.z;
  const float ox = (float)f.ox, oy = (float)f.oy, oz = (float)f.oz;
  const double dz = oz;
  const float fz = __fdiv_rn(kRf, (float)(dz + kEarthRadius));
  const double r2 = (double)ox * ox + (double)oy * oy + dz * (dz + 2.0 * kEarthRadius);
  const float height =
      __fdiv_rn((float)r2, sqrtf((float)(kEarthRadius * kEarthRadius + r2)) + kRf);
  float4* o = cell_rows<kPrecise>(D, p);
  o[kFrameOrigin] = make_float4(ox, oy, oz, height);
  o[kFrameNormal] =
      make_float4((float)f.normal.x, (float)f.normal.y, (float)f.normal.z, 0.f);
  o[kFrameNorth] = make_float4((float)f.north.x, (float)f.north.y, (float)f.north.z, ox * fz);
  o[kFrameEast] = make_float4((float)f.east.x, (float)f.east.y, (float)f.east.z, oy * fz);
  if (kPrecise)
    o[kFrameRest] = make_float4((float)(f.ox - (double)ox), (float)(f.oy - (double)oy),
                                (float)(f.oz - (double)oz), 0.f);
}

// Track of one (cell, azimuth) on the grid, in metres s along the gnomonic
// line: cell coordinates o + s d, the factors that turn s into lower / upper
// bounds of the distance from the origin's normal (r sin psi), and the end of
// the walk. tan(psi) = s gh / (lambda + s gu) with gh, gu the components of
// the line's direction along h and u.
struct Track {
  float ox, oy, dx, dy;
  float xlo, xhi;   // metres of horizontal distance per metre of s, times 1
  float smax;
};
__device__ __forceinline__ Track make_track(const GridDesc& g, float X0, float Y0, float hx,
                                            float hy, float hz, float ux, float uy, float uz) {
  Track t;
  const float kx = X0 * (1.f / kRf), ky = Y0 * (1.f / kRf);
  float gx = __fmaf_rn(-kx, hz, hx), gy = __fmaf_rn(-ky, hz, hy);
  const float n = rsqrtf(__fmaf_rn(gx, gx, gy * gy));
  gx *= n;
  gy *= n;
  const float gh = __fmaf_rn(gx, hx, gy * hy), gu = __fmaf_rn(gx, ux, gy * uy);
  const float lambda = __fdividef(kRf, uz);  // |(X0, Y0, R)|, along u
  t.smax = __fdividef(g.tau_max * lambda, fmaxf(__fmaf_rn(-g.tau_max, gu, gh), 1e-3f)) * 1.0001f +
           2.f * g.pad;
  // sin(psi) / s is gh over the distance of the line's point from the centre: the
  // farther end has the lowest, tan(psi) / s of either end is no less than any.
  const float a0 = __fdividef(gh, lambda), end = __fmaf_rn(t.smax, gu, lambda);
  const float a1 = __fdividef(gh, end);
  const float far = rsqrtf(__fmaf_rn(end, end, t.smax * gh * (t.smax * gh)));
  t.xlo = fminf(a0, gh * far) * (1.f - 4e-6f) * g.rlo;
  t.xhi = fmaxf(a0, a1) * (1.f + 4e-6f) * g.rhi;
  t.ox = (X0 - g.x0) * g.inv_c;
  t.oy = (Y0 - g.y0) * g.inv_c;
  t.dx = gx * g.inv_c;
  t.dy = gy * g.inv_c;
  // Never 0: the distance to the next column or row stays finite.
  if (fabsf(t.dx) < 1e-12f) t.dx = t.dx < 0.f ? -1e-12f : 1e-12f;
  if (fabsf(t.dy) < 1e-12f) t.dy = t.dy < 0.f ? -1e-12f : 1e-12f;
  return t;
}

// A sweep starts this many elevations below the previous azimuth's lowest miss:
// one is the least (the search comes from the hit below it) and leaves less to
// raise, two spares more second sweeps where the horizon falls from one azimuth
// to the next. From kDenseAzimuths on one is no slower on any terrain (per search
// with two / with one, rough 500 m terrain: 24 azimuths 5.56 / 5.66 ms, 120 20.6 /
// 21.2, 180 30.1 / 29.8; smooth 1 km: 24 3.24 / 3.35, 96 9.71 / 9.74, 180 17.7 / 16.5;
// 240 azimuths at 500 m 40.2 / 38.7).
constexpr int kDenseAzimuths = 160;
// Azimuths whose last result a warp keeps, for starts where the horizon falls
// (1.2M cells at 100 m: second sweeps in half of the evaluations, 41.8 -> 38.7 ms;
// 300 km domain at 500 m 17.5 -> 17.2; for every azimuth of every cell a smooth 1 km
// domain lost 2 %).
constexpr int kGuesses = 64;
__device__ __forceinline__ int start_drop(const DomainDesc& D) {
  return D.L >= kDenseAzimuths ? 1 : 2;
}

// First azimuth of a run of azimuths (of run D.runs: L) of the cell at position p;
// the first `extra` runs hold one more than the others.
__device__ __forceinline__ int run_start(const DomainDesc& D, int p, int run) {
  const bool tail = p >= D.tail_begin;
  return run * (tail ? D.tail_run_len : D.run_len) + min(run, tail ? D.tail_run_extra : D.run_extra);
}

// ---------------------------------------------------------------------------
// The sweep
// ---------------------------------------------------------------------------
enum : int { kLaneAdvance = 0, kLaneWalk = 1, kLaneList = 2 };
// Lane flags; kFlagAbove and kFlagRedo also come back from the triangle pass.
enum : int { kFlagAny = 1, kFlagAbove = 2, kFlagRedo = 4, kFlagGap = 8, kFlagTested = 16,
             kFlagRough = 32,  // a sweep of the item has started lower
             kFlagRetry = 64 };  // and up: lower starts so far

// What the triangle pass needs of a thread's azimuth and cell, in shared
// memory: any lane of the warp tests triangles for any other. Quadruples, read
// in one access each:
//   kRowOrigin   ray origin; error bound of the distances of the cell's triangles
//   kRowSide     lateral axis h x u; height below which list entries do not reach the ray
//   kRowRay      u - tan(e) h; tan(e) at the current elevation
//   kRowAlong    horizontal direction h of the azimuth; bound of the distance at the cell's exit
//   kRowUp       cell normal u; search radius
//   kRowTrack    track: origin and direction in grid cells
//   kRowHeight   a ray's height at s: T s (y if T >= 0 else z) + w, T = s x + tan(e)
//   kRowRest     precise: FP32 residual of the origin
// The walk reads its own thread's track anew in each pass: kept in registers
// through the triangle pass they cost a quarter of the resident warps.
enum : int { kRowOrigin, kRowSide, kRowRay, kRowAlong, kRowUp, kRowTrack, kRowHeight, kRowRest };
constexpr int kWarps = kSweepBlock / 32;

// Triangle records, list entries, list starts and pyramids of all domains of
// the call, one after another (DomainDesc::cell_base and ref_base).
struct SweepScene {
  const Tri* tris;
  const float4* tri_lo;
  const uint2* refs;
  const uint32_t* gstart;
  const uint2* planes;
  long long n_tri, n_cells, n_refs;
};

// Grid cell at of a thread's domain and the one after it lie in the call's list starts.
__device__ __forceinline__ bool size_ok(const int4 size, int at, const SweepScene& sc) {
  return at >= 0 && at < size.x * size.y && size.w + (long long)at + 1 < sc.n_cells;
}

template <bool kPrecise>
struct SweepShared {
  // Odd numbers of quadruples: threads' rows fall on different banks.
  float4 v[kSweepBlock][kPrecise ? 9 : 7];
  float4 grid[kSweepBlock];            // of the thread's domain: unit, 2 pad, error distance
  int4 size[kSweepBlock];              // its columns, rows, highest level, first cell
  float smax[kSweepBlock];             // end of the walk
  int mstop[kSweepBlock];              // elevation known to miss
  // Domain, cell, work position, azimuth, end azimuth, previous result,
  // elevation; elevation and flags from the triangle pass.
  int dom[kSweepBlock], cell[kSweepBlock], pos[kSweepBlock], az[kSweepBlock], az_end[kSweepBlock],
      prev[kSweepBlock], m[kSweepBlock], m_new[kSweepBlock], flags[kSweepBlock];
  int2 entry[kSweepBlock];             // per list in order: thread, first entry - its number
  int2 queue[kWarps][64];              // (thread, triangle) to be cut with the plane
  float tan_m[kTanTable];
  short guess[kWarps][kGuesses];         // the warp's last results of the first azimuths
  int wq[2][kWarps];                   // next and end of the warp's chunk of items
};

// A triangle's vertices relative to the ray origin of thread o.
template <bool kPrecise>
__device__ __forceinline__ void load_relative(const SweepShared<kPrecise>& sh, int o,
                                              const float4 org, const SweepScene& sc, int tri,
                                              float3& a, float3& b, float3& c) {
  const float4* tp = reinterpret_cast<const float4*>(sc.tris + tri);
  const float4 X = __ldg(tp), Y = __ldg(tp + 1), Z = __ldg(tp + 2);
  if (kPrecise) {
    const float4* lo = sc.tri_lo + 3LL * tri;
    const float4 LX = __ldg(lo), LY = __ldg(lo + 1), LZ = __ldg(lo + 2);
    const float4 q = sh.v[o][kPrecise ? kRowRest : 0];
    a = make_float3(rel(X.x, LX.x, org.x, q.x), rel(Y.x, LY.x, org.y, q.y),
                    rel(Z.x, LZ.x, org.z, q.z));
    b = make_float3(rel(X.y, LX.y, org.x, q.x), rel(Y.y, LY.y, org.y, q.y),
                    rel(Z.y, LZ.y, org.z, q.z));
    c = make_float3(rel(X.z, LX.z, org.x, q.x), rel(Y.z, LY.z, org.y, q.y),
                    rel(Z.z, LZ.z, org.z, q.z));
  } else {
    a = make_float3(X.x - org.x, Y.x - org.y, Z.x - org.z);
    b = make_float3(X.y - org.x, Y.y - org.y, Z.y - org.z);
    c = make_float3(X.z - org.x, Y.z - org.y, Z.z - org.z);
  }
}
__device__ __forceinline__ float dot3f(const float3 a, const float4 b) {
  return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, a.z * b.z));
}

// Whether triangle tri may hide the current ray of thread o or a higher one:
// not when its vertices lie on one side of the plane of the rays, nor all
// below the ray, nor when both edges that cross the plane (those at the vertex
// alone on its side) cross it below the ray, each by more than the bound of
// the errors. An edge from (q0, h0) to (q1, h1) crosses at the height (h0 |q1| +
// h1 |q0|) / (|q0| + |q1|).
template <bool kPrecise>
__device__ __forceinline__ bool may_hide(const SweepShared<kPrecise>& sh, int o,
                                         const float4 side, const SweepScene& sc, int tri,
                                         int* err) {
  float3 a, b, c;
  const float4 org = sh.v[o][kRowOrigin];
  load_relative(sh, o, org, sc, tri, a, b, c);
  const auto norm1 = [](float3 v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); };
  if (!check_ok(org.w >= kEps * fmaxf(norm1(a), fmaxf(norm1(b), norm1(c))), kCheckBound, tri, err))
    return true;
  const float q0 = dot3f(a, side), q1 = dot3f(b, side), q2 = dot3f(c, side);
  const float mu = org.w;
  if (fminf(q0, fminf(q1, q2)) > mu || fmaxf(q0, fmaxf(q1, q2)) < -mu) return false;
  const float4 ray = sh.v[o][kRowRay];
  const float h0 = dot3f(a, ray), h1 = dot3f(b, ray), h2 = dot3f(c, ray);
  const float mh = -mu * (1.f + fabsf(ray.w));
  if (fmaxf(h0, fmaxf(h1, h2)) < mh) return false;
  const bool p0 = q0 > 0.f, p1 = q1 > 0.f, p2 = q2 > 0.f;
  if (p0 == p1 && p1 == p2) return true;  // touches the plane
  const bool odd0 = p1 == p2, odd2 = p0 == p1;
  const float qo = fabsf(odd0 ? q0 : (odd2 ? q2 : q1)), ho = odd0 ? h0 : (odd2 ? h2 : h1);
  const float qa = fabsf(odd0 ? q1 : q0), ha = odd0 ? h1 : h0;
  const float qb = fabsf(odd2 ? q1 : q2), hb = odd2 ? h1 : h2;
  return !(__fmaf_rn(ho, qa, ha * qo) < 2.f * mh * (qo + qa + fabsf(ho - ha)) &&
           __fmaf_rn(ho, qb, hb * qo) < 2.f * mh * (qo + qb + fabsf(ho - hb)));
}

// Cuts triangle tri with the plane of thread o's rays and compares the segment
// with its current ray: nothing to do (below, beside, behind, out of reach or
// past the cell), kFlagAbove (it stays above the ray), or a raise: m_new, the
// lowest elevation it is not known to hide, with kFlagRedo when it may hide
// that one too. Distances in the plane: x along h, heights over the ray times
// 1 / cos(e), each with a bound of its error.
template <bool kPrecise>
__device__ __forceinline__ int cut_triangle(const SweepShared<kPrecise>& sh, int o,
                                            const SweepScene& sc, const DomainDesc* doms,
                                            int tri, int& m_new, int* err) {
  float3 a, b, c;
  const float4 org = sh.v[o][kRowOrigin], side = sh.v[o][kRowSide], ray = sh.v[o][kRowRay],
               along = sh.v[o][kRowAlong];
  load_relative(sh, o, org, sc, tri, a, b, c);
  const float q0 = dot3f(a, side), q1 = dot3f(b, side), q2 = dot3f(c, side);
  const float h0 = dot3f(a, ray), h1 = dot3f(b, ray), h2 = dot3f(c, ray);
  const float x0 = dot3f(a, along), x1 = dot3f(b, along), x2 = dot3f(c, along);
  const float e0 = kEps * (fabsf(a.x) + fabsf(a.y) + fabsf(a.z)),
              e1 = kEps * (fabsf(b.x) + fabsf(b.y) + fabsf(b.z)),
              e2 = kEps * (fabsf(c.x) + fabsf(c.y) + fabsf(c.z));
  const float ta = ray.w, ts = 1.f + fabsf(ta), xexit = along.w, tfar = sh.v[o][kRowUp].w,
              reach = tfar * rsqrtf(__fmaf_rn(ta, ta, 1.f));  // the search radius along x
  const float* tm = sh.tan_m + kTanRange;
  const int m = sh.m[o];
  if (!check_ok(m >= -kTanRange && m <= kMaxM, kCheckElevation, m, err)) return kFlagAbove;
  // Vertices in the plane within rounding: one of them is an end point of the
  // segment whichever side it is taken to be on (the cell's own vertex, under
  // the ray origin, always is); two leave the segment open.
  const bool n0 = fabsf(q0) <= e0, n1 = fabsf(q1) <= e1, n2 = fabsf(q2) <= e2;
  const bool p0 = q0 > 0.f, p1 = q1 > 0.f, p2 = q2 > 0.f;
  const bool beside = p0 == p1 && p1 == p2;
  const bool edge = beside || (n0 && n1) || (n0 && n2) || (n1 && n2);
  float ah = 0.f, bh = 0.f, ax = 0.f, bx = 0.f, ea = 0.f, eb = 0.f;
  bool decided = false;  // above for certain; else the watertight test is asked
  const auto all = [&](auto f) {
    return (!n0 || f(h0, x0, e0)) && (!n1 || f(h1, x1, e1)) && (!n2 || f(h2, x2, e2));
  };
  if (edge) {
    // It meets the plane in an edge or in one vertex, if at all: nowhere but
    // at the vertices in the plane and between them. Which of the triangles at
    // such an edge a ray hits is the watertight test's to say.
    if ((beside && !(n0 || n1 || n2)) ||
        all([&](float h, float, float e) { return h < -ts * e; }) ||
        all([&](float, float x, float e) { return x < -e; }) ||
        all([&](float, float x, float e) { return x - e > xexit; }))
      return 0;
  } else {
    // End points on the two edges at the vertex that lies alone on its side.
    const bool odd0 = p1 == p2, odd2 = p0 == p1;
    const float qo = fabsf(odd0 ? q0 : (odd2 ? q2 : q1));
    const float qa = fabsf(odd0 ? q1 : q0), qb = fabsf(odd2 ? q1 : q2);
    const float ho = odd0 ? h0 : (odd2 ? h2 : h1);
    const float ha = odd0 ? h1 : h0, hb = odd2 ? h1 : h2;
    const float xo = odd0 ? x0 : (odd2 ? x2 : x1);
    const float xa = odd0 ? x1 : x0, xb = odd2 ? x1 : x2;
    const float eo = odd0 ? e0 : (odd2 ? e2 : e1);
    const float va = odd0 ? e1 : e0, vb = odd2 ? e1 : e2;
    const float ra = __fdividef(1.f, qo + qa), rb = __fdividef(1.f, qo + qb);
    ah = __fmaf_rn(ho, qa, ha * qo) * ra;
    bh = __fmaf_rn(ho, qb, hb * qo) * rb;
    ax = __fmaf_rn(xo, qa, xa * qo) * ra;
    bx = __fmaf_rn(xo, qb, xb * qo) * rb;
    const float fa = ra * __fmaf_rn(eo, qa, va * qo), fb = rb * __fmaf_rn(eo, qb, vb * qo);
    const float ga = __fmaf_rn(fa * ra, fabsf(ho - ha), fa),
                gb = __fmaf_rn(fb * rb, fabsf(ho - hb), fb);
    ea = ts * ga;
    eb = ts * gb;
    const float xea = __fmaf_rn(fa * ra, fabsf(xo - xa), fa),
                xeb = __fmaf_rn(fb * rb, fabsf(xo - xb), fb);
    const float xem = fmaxf(xea, xeb), xmin = fminf(ax, bx) - xem;
    // Below, behind, past the cell (its own cell follows), out of reach. (The
    // reach along x is that of the ray for rising ones, whose higher
    // neighbours reach less far, and the radius itself for falling ones.)
    if ((ah < -ea && bh < -eb) || fmaxf(ax, bx) < -xem || xmin > xexit ||
        xmin > 1.00001f * (ta > 0.f ? reach : tfar))
      return 0;
    decided = ah > ea && bh > eb;
    if ((ah > ea && bh < -eb) || (ah < -ea && bh > eb)) {
      // It crosses the ray's line, in front of the origin or behind it.
      const float fh = fabsf(ah), gh = fabsf(bh), r2 = __fdividef(1.f, fh + gh);
      const float xc = __fmaf_rn(ax, gh, bx * fh) * r2;
      const float xe = 2.f * r2 * (__fmaf_rn(xea, gh, xeb * fh) +
                                   fabsf(ax - bx) * r2 * __fmaf_rn(ea, gh, eb * fh));
      if (xc < -xe) {
        if ((ax > bx ? ah : bh) < 0.f) return 0;
        decided = true;
      } else if (xc > xe && xc < reach * 0.99999f - xe) {
        // Hidden, and with it every ray up to the segment's higher end.
        const bool top = ah > 0.f;
        const float th = top ? ah : bh, tx = top ? ax : bx, tg = top ? ga : gb;
        m_new = m + 1;
        if (!(tx > 0.f)) return kFlagRedo;
        // Ray k is hidden where it passes the higher end below it by more than
        // the error te and within the radius (so do all between m and k then):
        // it meets the segment between ray m's crossing and that end.
        const float far2 = 0.999f * tfar * tfar;
        const float tx2 = fmaxf(tx, xc) * fmaxf(tx, xc);
        float v = 0.f, te = 0.f;
        const auto hides = [&](int k) {
          const float tk = tm[k];
          v = __fmaf_rn(ta - tk, tx, th);
          te = tg * (1.f + fabsf(ta) + fabsf(tk));
          return v > te && __fmaf_rn(tx2 * tk, tk, tx2) < far2;
        };
        int k = m;
        if (__fmaf_rn(ta - tm[min(m + 4, kMaxM)], tx, th) > 0.f) {  // far up: near the end at once
          k = max(m, min((int)floorf(atanf(__fmaf_rn(th, __fdividef(1.f, tx), ta)) * 114.591559f),
                         kMaxM) - 1);
          if (k > m && !hides(k)) return kFlagRedo;
        }
        while (hides(k + 1) && k < kMaxM) k++;
        m_new = k + 1;
        return v < -te ? kFlagAny : kFlagRedo;
      }
    }
  }
  if (!decided) {
    // Undecided: the watertight test (along an edge, as many rays as it hides);
    // and, where it does not hide this one, whether it is below the next.
    int k = m;
    while (k <= kMaxM && (edge || k == m) &&
           exact_hit<kPrecise>(doms + sh.dom[o], sh.pos[o], sh.az[o], k, tri))
      k++;
    if (k > m) {
      m_new = k;
      return kFlagRedo;
    }
    const float tn = tm[m + 1], d = ta - tn;
    if (edge ? all([&](float h, float x, float e) {
          return __fmaf_rn(d, x, h) < -(1.f + fabsf(tn)) * e;
        })
             : __fmaf_rn(d, ax, ah) < -ea && __fmaf_rn(d, bx, bh) < -eb)
      return 0;
    if (edge) return kFlagAbove;
  }
  // Above the ray: unless it begins past this cell (by the angle at the
  // Earth's centre), where the walk meets it again.
  const GridDesc& g = *doms[sh.dom[o]].grid;
  const bool first = ax < bx;
  const float xm = first ? ax : bx, ym = __fmaf_rn(ta, xm, first ? ah : bh);
  const float ro = dot3f(make_float3(org.x, org.y, org.z + kRf), sh.v[o][kRowUp]);
  return __fdividef(xm, ro + ym) * g.rhi > __fmaf_rn(1e-5f, xexit, xexit) ? 0 : kFlagAbove;
}

template <bool kPrecise>
__global__ void __launch_bounds__(kSweepBlock, kPrecise ? HZ_SWEEP_MIN_BLOCKS_EXACT
                                                      : HZ_SWEEP_MIN_BLOCKS)
    k_sweep(const DomainDesc* __restrict__ doms, int ndom, const int* __restrict__ order,
            int total, int* __restrict__ work, int s_full, int* __restrict__ list,
            int* __restrict__ list_n, unsigned* __restrict__ listed, const SweepScene sc,
            int lanes, int* __restrict__ err) {
  __shared__ SweepShared<kPrecise> sh;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kUnknown = -30000, kFirst = -30001;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const unsigned below_me = (1u << lane) - 1u;
  if (*err & kErrGrid) return;  // set by the grid build: the caller searches with the tree
  for (int k = t; k < kTanTable; k += kSweepBlock) sh.tan_m[k] = __ldg(&doms[0].tan_m[k]);
  if (lane == 0) {
    sh.wq[0][wid] = 0;
    sh.wq[1][wid] = 0;
  }
  for (int k = lane; k < kGuesses; k += 32) sh.guess[wid][k] = 1000;
  sh.az[t] = 0;
  sh.az_end[t] = 0;
  sh.dom[t] = 0;
  __syncthreads();

  bool alive = lane < lanes;
  int st = kLaneAdvance, fl = 0;
  int m = 0;
  int i = 0, j = 0, l = 0;
  float s = 0.f, s1 = 0.f, ta = 0.f;        // walk position, exit of the current cell, tan(e)
  int at = 0;

  // Slope and plane normal of the ray at lattice elevation m.
  auto set_elevation = [&]() {
    if (!check_ok(m > -kTanRange && m <= kMaxM + 1, kCheckElevation, m, err)) m = 0;
    ta = sh.tan_m[m + kTanRange];
    const float4 h = sh.v[t][kRowAlong], u = sh.v[t][kRowUp];
    sh.v[t][kRowRay] = make_float4(__fmaf_rn(-ta, h.x, u.x), __fmaf_rn(-ta, h.y, u.y),
                                   __fmaf_rn(-ta, h.z, u.z), ta);
    sh.m[t] = m;
  };
  // Height (as encoded in the lists) below which terrain between sa and sb
  // does not reach the ray: at distance x a ray of slope tan(e) is x (tan(e) +
  // x / 2r) above its origin's sphere at least, lowest at the near end when
  // that rises and at the far end when it falls.
  auto threshold = [&](const float4 hc, float sa, float sb) {
    const float T = __fmaf_rn(sa, hc.x, ta);
    return __fmaf_rn(T, T >= 0.f ? sa * hc.y : sb * hc.z, hc.w);
  };
  // Its height at one position.
  auto height = [&](const float4 hc, float sa) {
    const float T = __fmaf_rn(sa, hc.x, ta);
    return __fmaf_rn(T, sa * (T >= 0.f ? hc.y : hc.z), hc.w);
  };

  for (;;) {
    const unsigned live = __ballot_sync(kFull, alive);
    if (live == 0u) break;
    // Shares of the lanes at work: few in small domains and at the queue's end.
    const int walk_min = max(1, __popc(live) * HZ_WALK_MIN >> 5),
              adv_min = max(1, __popc(live) * HZ_SWEEP_ADVANCE >> 5);
    const unsigned waiting = __ballot_sync(kFull, alive && st == kLaneAdvance);
    if (waiting != 0u && (__popc(waiting) >= adv_min || waiting == live)) {
      const bool mine = alive && st == kLaneAdvance;
      bool again = false;
      if (mine && sh.az[t] < sh.az_end[t]) {
        // An azimuth has ended.
        const DomainDesc& D = doms[sh.dom[t]];
        const int a = sh.az[t];
        int code;
        if (fl & kFlagGap) {
          code = kCodeGap;
        } else if (fl & kFlagAny) {
          code = m;
        } else if (m > s_full) {
          // Nothing met the start's ray or any above it: start lower.
          again = true;
          sh.mstop[t] = m;
          const int tries = fl / kFlagRetry;
          m = tries < kLowerTries ? max(s_full, m - (kLower << tries)) : s_full;
          fl = (tries + 1) * kFlagRetry | kFlagRough;
        } else {
          code = kCodeAllMiss;
        }
        if (!again) {
          if (check_ok(a >= 0 && a < D.L && sh.cell[t] >= 0 && sh.cell[t] < D.ncell, kCheckSlot,
                       (long long)a * D.ncell + sh.cell[t], err))
            D.codes[(long long)a * D.ncell + sh.cell[t]] = (int16_t)code;
          if (code == kCodeGap) {
            const long long q = D.k_begin + sh.pos[t];
            const unsigned bit = 1u << (q & 31);
            if (!(atomicOr(&listed[q >> 5], bit) & bit)) list[atomicAdd(list_n, 1)] = (int)q;
          }
          sh.prev[t] = code > kCodeAllMiss ? code : kUnknown;
          if (code > kCodeAllMiss && a < kGuesses) sh.guess[wid][a] = (short)code;
          sh.az[t] = a + 1;
        }
      }
      // New items for the lanes whose azimuths are done.
      const unsigned starting = __ballot_sync(kFull, mine && sh.az[t] >= sh.az_end[t]);
      if (starting != 0u) {
        const int nreq = __popc(starting);
        int first = 0, take = 0, nb = 0;
        if (lane == 0) {
          take = min(sh.wq[1][wid] - sh.wq[0][wid], nreq);
          first = sh.wq[0][wid];
          sh.wq[0][wid] += take;
          if (take < nreq) {
            // Near the end of the queue a warp takes only what it needs.
            const int left = total - *(volatile int*)work;
            const bool tail = left < (int)min(2147483647ll, (long long)gridDim.x * kWarps * lanes);
            const int grab = tail ? nreq - take : max(32, nreq - take);
            nb = atomicAdd(work, grab);
            sh.wq[0][wid] = nb + (nreq - take);
            sh.wq[1][wid] = nb + grab;
          }
        }
        first = __shfl_sync(kFull, first, 0);
        take = __shfl_sync(kFull, take, 0);
        nb = __shfl_sync(kFull, nb, 0);
        if (starting >> lane & 1u) {
          const int rank = __popc(starting & below_me);
          const int item = rank < take ? first + rank : nb + (rank - take);
          if (item >= total) {
            alive = false;
          } else {
            const int dom = domain_of_item(doms, ndom, item);
            const DomainDesc& D = doms[dom];
            const unsigned local = (unsigned)(item - D.item_begin);
            // Run by run over the cells; then over those of the tail.
            const unsigned whole = (unsigned)D.tail_begin * (unsigned)D.runs;
            const bool tail = local >= whole;
            const unsigned rest = tail ? local - whole : local;
            const unsigned cells = (unsigned)(tail ? D.ncell_traced - D.tail_begin : D.tail_begin);
            unsigned run = rest / cells;
            int p = (int)(rest - run * cells) + (tail ? D.tail_begin : 0);
            if (!check_ok(p >= 0 && p < D.ncell_traced && run_start(D, p, (int)run + 1) <= D.L,
                          kCheckPosition, item, err))
              p = run = 0;
            const float4* fr = cell_rows<kPrecise>(D, p);
            const float4 fo = __ldg(fr + kFrameOrigin), fu = __ldg(fr + kFrameNormal);
            sh.v[t][kRowOrigin] = make_float4(fo.x, fo.y, fo.z, 0.f);
            sh.v[t][kRowUp] = make_float4(fu.x, fu.y, fu.z, D.tfar);
            if (kPrecise) sh.v[t][kPrecise ? kRowRest : 0] = __ldg(fr + kFrameRest);
            const GridDesc& g = *D.grid;
            sh.v[t][kRowHeight].w = (fo.w - g.hpad - g.hlo) * g.iq;
            sh.grid[t] = make_float4(g.unit, 2.f * g.pad, g.dadd + 2.f * __uint_as_float(g.lmax),
                                     __uint_as_float(D.ref_base));
            sh.size[t] = make_int4(g.W, g.H, g.L, D.cell_base);
            sh.dom[t] = dom;
            sh.cell[t] = (int)(order[D.k_begin + p] - D.cell_offset);
            sh.pos[t] = p;
            sh.az[t] = run_start(D, p, (int)run);
            sh.az_end[t] = run_start(D, p, (int)run + 1);
            fl = 0;
            sh.prev[t] = sh.az[t] == 0 ? start_drop(D) : kFirst;  // the search starts at 0 (cpp:511)
          }
        }
      }
      if (mine && alive) {
        const DomainDesc& D = doms[sh.dom[t]];
        const GridDesc& g = *D.grid;
        if (!again) {
          const int a = sh.az[t];
          const int prev = sh.prev[t];
          sh.mstop[t] = 1 << 20;
          fl = (fl & kFlagRough) | (prev == kFirst ? kLowerTries * kFlagRetry : 0);
          // Below the previous azimuth's result (start_drop); a run's first azimuth
          // well below any horizon of its neighbourhood (k_sweep_runs checks
          // that the search came from no lower); else from the floor.
          m = prev == kUnknown
                  ? s_full
                  : max(s_full, prev == kFirst ? kRunStart : prev - start_drop(D));
          // Where a sweep of this item has started over, from no higher than just
          // below what the warp found last in this azimuth: its cells are
          // neighbours, and a fall of the horizon that one has met costs the others
          // no second sweep.
          if (a < kGuesses && (fl & kFlagRough))
            m = max(s_full, max(m - 8, min(m, sh.guess[wid][a] - 1)));
          if (D.start_m && (D.start_all || a % (D.L / D.groups) == 0)) {
            const int m0 = clamp_start(D.start_m[(long long)a * D.ncell + sh.cell[t]]);
            m = max(min(m, m0 - 1), 1 - kTanRange);
            if (m0 > kMaxM) fl = kFlagGap;  // a start at the zenith: ray by ray
          }
          const double2 cs64 = __ldg(&D.azim_cs[a]);
          const float c = (float)cs64.x, n = (float)cs64.y;
          const float4* fr = cell_rows<kPrecise>(D, sh.pos[t]);
          const float4 fn = __ldg(fr + kFrameNorth), fe = __ldg(fr + kFrameEast);
          const float hx = __fmaf_rn(c, fn.x, n * fe.x);
          const float hy = __fmaf_rn(c, fn.y, n * fe.y);
          const float hz = __fmaf_rn(c, fn.z, n * fe.z);
          const float4 u = sh.v[t][kRowUp];
          const float ux = u.x, uy = u.y, uz = u.z;
          sh.v[t][kRowAlong] = make_float4(hx, hy, hz, 0.f);
          sh.v[t][kRowSide] = make_float4(__fmaf_rn(hy, uz, -hz * uy), __fmaf_rn(hz, ux, -hx * uz),
                                          __fmaf_rn(hx, uy, -hy * ux), 0.f);
          const Track tr = make_track(g, fn.w, fe.w, hx, hy, hz, ux, uy, uz);
          sh.v[t][kRowTrack] = make_float4(tr.ox, tr.oy, tr.dx, tr.dy);
          sh.v[t][kRowHeight].x = tr.xlo * g.cmin * g.irlo;
          sh.v[t][kRowHeight].y = tr.xlo * g.iq;
          sh.v[t][kRowHeight].z = tr.xhi * g.iq;
          sh.smax[t] = tr.smax;
        }
        i = min(max((int)floorf(sh.v[t][kRowTrack].x), 0), sh.size[t].x - 1);
        j = min(max((int)floorf(sh.v[t][kRowTrack].y), 0), sh.size[t].y - 1);
        l = 0;
        s = 0.f;
        st = (fl & kFlagGap) ? kLaneAdvance : kLaneWalk;
        set_elevation();
      }
    }

    // Walk pass: pyramid steps while enough lanes walk. A step looks at the
    // cell of level l at the walk's position: visible, it goes down (to the
    // cell's list from level 0), else on to the next cell, and up a level where
    // that one begins a cell of it.
    {
    const float4 tr = sh.v[t][kRowTrack], hc = sh.v[t][kRowHeight];
    const int4 size = sh.size[t];
    const float smax = sh.smax[t];
    const int W = size.x, n2 = 2 * size.x * size.y;
    const uint2* planes = sc.planes + 2 * (long long)size.w;
    const int nx = (int)(__float_as_uint(tr.z) >> 31), ny = (int)(__float_as_uint(tr.w) >> 31);
    const float ix = __fdividef(1.f, tr.z), iy = __fdividef(1.f, tr.w);
    const float back_x = nx ? 1.f : -1.f, back_y = ny ? 1.f : -1.f;
    // Track position (cells) and the ray's height at s.
    float x0 = __fmaf_rn(s, tr.z, tr.x), y0 = __fmaf_rn(s, tr.w, tr.y), r0 = height(hc, s);
#pragma unroll 1
    for (int q = 0; q < HZ_WALK_STEPS; q++) {
      if (st == kLaneWalk) {
        const int a = i >> l, b = j >> l;
        at = grid_index(W, n2, a, b, l);
        if (!check_ok(at >= 0 && at < n2 && 2 * (long long)size.w + at < 2 * sc.n_cells, kCheckGrid,
                      at, err))
          at = 0;
        const uint2 pl = __ldg(planes + at);
        const int bx = (a + 1 - nx) << l, by = (b + 1 - ny) << l;
        const float fx = (float)bx, fy = (float)by;
        const float tx = (fx - tr.x) * ix, ty = (fy - tr.y) * iy;
        s1 = fmaxf(s, fminf(fminf(tx, ty), smax));
        const float x1 = __fmaf_rn(s1, tr.z, tr.x), y1 = __fmaf_rn(s1, tr.w, tr.y);
        const float r1 = height(hc, s1);
        // The plane over entry and exit against the ray.
        const float half = __int_as_float((126 + l) << 23);  // half a cell of level l
        const float cx = __fmaf_rn(back_x, half, fx), cy = __fmaf_rn(back_y, half, fy);
        const float2 gr = __half22float2(*reinterpret_cast<const __half2*>(&pl.y));
        const float hp = __uint_as_float(pl.x);
        const bool over = __fmaf_rn(gr.x, x0 - cx, __fmaf_rn(gr.y, y0 - cy, hp)) >= r0 ||
                          __fmaf_rn(gr.x, x1 - cx, __fmaf_rn(gr.y, y1 - cy, hp)) >= r1;
        if (over && !(fl & kFlagTested)) {
          if (l == 0) st = kLaneList;
          l = max(l - 2, 0);
        } else {
          fl &= ~kFlagTested;
          s = s1;
          x0 = x1;
          y0 = y1;
          r0 = r1;
          const bool xx = tx < ty;
          const int last = (1 << l) - 1;
          const int fi = min(max((int)floorf(x1), a << l), (a << l) + last);
          const int fj = min(max((int)floorf(y1), b << l), (b << l) + last);
          i = xx ? bx - nx : fi;
          j = xx ? fj : by - ny;
          if (((xx ? bx : by) & (3 << l)) == 0 && l < size.z) l += 2;
          if (s >= smax || (unsigned)i >= (unsigned)W || (unsigned)j >= (unsigned)size.y)
            st = kLaneAdvance;
        }
      }
      if (__popc(__ballot_sync(kFull, st == kLaneWalk)) < walk_min) break;
    }
    }

    // Triangle pass: the lists of all lanes that reached a cell, their
    // entries spread over the warp.
    const unsigned lists = __ballot_sync(kFull, st == kLaneList);
    if (lists == 0u) continue;
    int n = 0;
    unsigned k0 = 0;
    if (st == kLaneList) {
      const uint32_t* gs = sc.gstart + (sh.size[t].w + at);
      const uint32_t k = __ldg(gs);
      n = (int)(__ldg(gs + 1) - k);
      const float4 g = sh.grid[t];
      const float4 hc = sh.v[t][kRowHeight];
      const float xexit = s1 * hc.z * g.x;
      k0 = __float_as_uint(g.w) + k;
      if (!check_ok(size_ok(sh.size[t], at, sc) && n >= 0 && (long long)k0 + n <= sc.n_refs,
                    kCheckList, k0, err))
        n = 0;
      sh.v[t][kRowOrigin].w = kEpsCell * __fmaf_rn(kDropCell, xexit, g.z);
      sh.v[t][kRowSide].w = threshold(hc, s, s1) + kMagic;
      sh.v[t][kRowAlong].w = xexit + g.y;
      sh.m_new[t] = m;
      sh.flags[t] = 0;
    }
    int off = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(kFull, off, d);
      if (lane >= d) off += v;
    }
    const int entries = __shfl_sync(kFull, off, 31);
    off -= n;
    const unsigned filled = __ballot_sync(kFull, n > 0);
    if (n > 0) sh.entry[wid * 32 + __popc(filled & below_me)] = make_int2(t, (int)k0 - off);
    __syncwarp();
    int queued = 0;
    auto cut = [&](int count) {
      if (lane < count) {
        const int2 e = sh.queue[wid][lane];
        int m_new = 0;
        const int r = cut_triangle<kPrecise>(sh, e.x, sc, doms, e.y, m_new, err);
        if (r == kFlagAbove) atomicOr(&sh.flags[e.x], kFlagAbove);
        else if (r != 0) {
          atomicMax(&sh.m_new[e.x], m_new);
          if (r == kFlagRedo) atomicOr(&sh.flags[e.x], kFlagRedo);
        }
      }
      __syncwarp();
    };
    for (int base = 0; base < entries; base += 32) {
      // Lists that begin in this stretch mark their first entry; the rank of
      // a list among all gives its owner.
      const int rel0 = off - base;
      const unsigned marks = __reduce_or_sync(
          kFull, n > 0 && rel0 >= 0 && rel0 < 32 ? 1u << rel0 : 0u);
      const int before = __popc(__ballot_sync(kFull, n > 0 && off < base));
      const int x = base + lane;
      bool want = false;
      int o = 0, tri = 0;
      if (x < entries) {
        const int2 e = sh.entry[wid * 32 + before + __popc(marks & ((2u << lane) - 1u)) - 1];
        o = e.x;
        const uint2 rf = __ldg(sc.refs + (unsigned)(e.y + x));
        const float4 side = sh.v[o][kRowSide];
        if (height_magic(rf.y & 0xFFFFu) >= side.w &&
            check_ok((int)rf.x >= 0 && (int)rf.x < sc.n_tri, kCheckTriangle, (int)rf.x, err)) {
          tri = (int)rf.x;
          want = may_hide<kPrecise>(sh, o, side, sc, tri, err);
        }
      }
      const unsigned wants = __ballot_sync(kFull, want);
      if (want && check_ok(queued + __popc(wants & below_me) < 64, kCheckQueue, queued, err))
        sh.queue[wid][queued + __popc(wants & below_me)] = make_int2(o, tri);
      queued += __popc(wants);
      __syncwarp();
      if (queued >= 32) {
        cut(32);
        queued -= 32;
        const int2 e = sh.queue[wid][32 + lane];
        __syncwarp();
        if (lane < queued) sh.queue[wid][lane] = e;
        __syncwarp();
      }
    }
    if (queued > 0) cut(queued);
    if (st == kLaneList) {
      const int f = sh.flags[t], mn = sh.m_new[t];
      if (mn > m) {
        fl |= kFlagAny;
        if (mn >= sh.mstop[t]) {
          m = sh.mstop[t];  // known to miss from the sweep above
          st = kLaneAdvance;
        } else if (mn > kMaxM) {
          fl |= kFlagGap;
          st = kLaneAdvance;
        } else {
          m = mn;
          set_elevation();
          // Triangles that were above the ray, or may hide the new one too:
          // the list again.
          if (!(f & (kFlagAbove | kFlagRedo))) {
            fl |= kFlagTested;
            st = kLaneWalk;
          }
        }
      } else if (f & kFlagAbove) {
        // A triangle stays above with nothing hiding the ray: the hits of this
        // azimuth are not one run of elevations.
        fl |= kFlagGap;
        st = kLaneAdvance;
      } else {
        fl |= kFlagTested;
        st = kLaneWalk;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Ray by ray
// ---------------------------------------------------------------------------

// Any-hit query of one lattice ray on the grid.
template <bool kPrecise>
__device__ bool grid_ray(const DomainDesc& D, const GridDesc& g, const Ray& r, const Track& tr,
                         float ho, float slope, int* err) {
  const int W = g.W, H = g.H, n2 = 2 * W * H;
  const float kl = tr.xlo * g.cmin / g.rlo, kh = tr.xhi * g.cmax / g.rlo;
  const float cl = (ho - g.hpad - g.hlo) * g.iq, ch = __fmaf_rn(ho + g.hpad - g.hlo, g.iq, 2.f);
  const float xlo = tr.xlo * g.iq, xhi = tr.xhi * g.iq;
  int i = min(max((int)floorf(tr.ox), 0), W - 1);
  int j = min(max((int)floorf(tr.oy), 0), H - 1);
  int l = 0;
  float s = 0.f;
  bool tested = false;
  for (;;) {
    const int a = i >> l, b = j >> l;
    const int at = grid_index(W, n2, a, b, l);
    if (!check_ok(at >= 0 && at < n2, kCheckGrid, at, err)) return false;
    const uint2 pl = __ldg(D.planes + at);
    const unsigned lo = __ldg(D.low + at);
    const bool sx = tr.dx > 0.f, sy = tr.dy > 0.f;
    const float tx = __fdividef((float)((sx ? a + 1 : a) << l) - tr.ox, tr.dx);
    const float ty = __fdividef((float)((sy ? b + 1 : b) << l) - tr.oy, tr.dy);
    const float s1 = fmaxf(s, fminf(fminf(tx, ty), tr.smax));
    // Lowest and highest height of the ray over [s, s1].
    const float T0 = __fmaf_rn(s, kl, slope), T1 = __fmaf_rn(s1, kh, slope);
    const float tlo = __fmaf_rn(T0, T0 >= 0.f ? s * xlo : s1 * xhi, cl);
    const float thi = __fmaf_rn(T1, T1 >= 0.f ? s1 * xhi : s * xlo, ch);
    const float half = 0.5f * (float)(1 << l);
    const float cx = (float)(a << l) + half, cy = (float)(b << l) + half;
    const float2 gr = __half22float2(*reinterpret_cast<const __half2*>(&pl.y));
    const float hp = __uint_as_float(pl.x);
    const auto over = [&](float q) {
      const float T = __fmaf_rn(q, kl, slope);
      return __fmaf_rn(gr.x, __fmaf_rn(q, tr.dx, tr.ox) - cx,
                       __fmaf_rn(gr.y, __fmaf_rn(q, tr.dy, tr.oy) - cy, hp)) >=
             __fmaf_rn(T, q * (T >= 0.f ? xlo : xhi), cl);
    };
    const bool vis = !tested && (float)lo <= thi && (over(s) || over(s1));
    if (vis && l > 0) {
      l -= 2;
      continue;
    }
    if (vis) {
      const unsigned e = D.gstart[at + 1];
      for (unsigned k = D.gstart[at]; k < e; k++) {
        const uint2 rf = __ldg(D.refs + k);
        if ((float)(rf.y & 0xFFFFu) < tlo || (float)(rf.y >> 16) > thi) continue;
        if (check_ok((int)rf.x >= D.tri_base && (int)rf.x < D.tri_base + D.n_tri, kCheckTriangle,
                     (int)rf.x, err) &&
            test_tri<kPrecise>(D.tris, D.tri_lo, r, (int)rf.x))
          return true;
      }
      tested = true;
      continue;
    }
    tested = false;
    s = s1;
    const bool xx = tx < ty;
    int cross;
    if (xx) {
      cross = sx ? a + 1 : a;
      i = sx ? cross << l : (cross << l) - 1;
      j = min(max((int)floorf(__fmaf_rn(s, tr.dy, tr.oy)), b << l), ((b + 1) << l) - 1);
    } else {
      cross = sy ? b + 1 : b;
      j = sy ? cross << l : (cross << l) - 1;
      i = min(max((int)floorf(__fmaf_rn(s, tr.dx, tr.ox)), a << l), ((a + 1) << l) - 1);
    }
    if ((cross & 3) == 0 && l < g.L) l += 2;
    if (s >= tr.smax || (unsigned)i >= (unsigned)W || (unsigned)j >= (unsigned)H) return false;
  }
}

// Cosine and sine of lattice elevation m. Under a roof (a mesh folded over
// itself) every ray of a turn hits, and each azimuth carries the search a turn
// further, past the table.
__device__ __forceinline__ double2 elevation(const DomainDesc& D, int m) {
  if (m >= kElevMin && m < kElevMin + kElevTable) return __ldg(&D.elev_cs[m - kElevMin]);
  const double e = (double)m * D.two_ha;
  return make_double2(cos(e), sin(e));
}

// The first azimuth of every run but a cell's first was swept from kRunStart:
// where the search can come to it from below that (the azimuth before has no
// hits from there up, or is open), the cell goes to the repair.
__global__ void k_sweep_runs(const DomainDesc* __restrict__ doms, int ndom, int first, int total,
                             int* __restrict__ list, int* __restrict__ list_n,
                             unsigned* __restrict__ listed, const int* __restrict__ order,
                             const int* __restrict__ err) {
  const int k = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= first + total || (*err & kErrGrid)) return;
  const long long gid = order[k];
  const DomainDesc& D = doms[domain_of(doms, ndom, gid)];
  const int cell = (int)(gid - D.cell_offset);
  bool open = false;
  const int p = (int)(k - D.k_begin), runs = p >= D.tail_begin ? D.tail_runs : D.runs;
  for (int r = 1; r < runs; r++) {
    const int a = run_start(D, p, r);
    const int16_t* c = D.codes + (long long)a * D.ncell + cell;
    open |= *c > kCodeAllMiss && c[-(long long)D.ncell] <= kRunStart + 1;
  }
  if (open) {
    const unsigned bit = 1u << (k & 31);
    if (!(atomicOr(&listed[k >> 5], bit) & bit)) list[atomicAdd(list_n, 1)] = k;
  }
}

// n additions of c (+-two_ha) to elev, each rounded, as the reference carries
// its elevation. While the sum stays in one binade an addition moves it by the
// same number of its last places, c rounded to them (unless c lies half way
// between two): one integer addition for all steps, where each FP64 addition
// holds the SM's pipe for 16 cycles. The step that leaves a binade is an FP64
// addition; so is one that would reach its lower end, below which the places
// are finer.
__device__ __forceinline__ void add_steps(double& elev, double c, int n) {
  const long long cb = __double_as_longlong(c);
  const unsigned long long mant = (1ull << 52) - 1;
  const unsigned long long mc = ((unsigned long long)cb & mant) | (mant + 1);
  const int ec = (int)((unsigned long long)cb >> 52) & 0x7ff;
#pragma unroll 1
  while (n > 0) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(elev);
    const int sh = ((int)(x >> 52) & 0x7ff) - ec;
    if (sh > 0 && sh < 20) {
      const unsigned long long half = 1ull << (sh - 1), rest = mc & (2 * half - 1);
      const unsigned long long k = (mc >> sh) + (rest > half ? 1ull : 0ull);
      const bool grows = (long long)x >= 0 == (cb >= 0);
      // Steps to the binade's end, rounded down.
      const unsigned long long room = grows ? mant - (x & mant) : x & mant;
      const int t = min(n, (int)(__fdividef((float)(unsigned)(room >> 20),
                                            (float)(unsigned)(k >> 20)) * 0.9999f));
      const unsigned long long y = grows ? x + (unsigned)t * k : x - (unsigned)t * k;
      if (rest != half && (y >> 52) == (x >> 52) && (grows || (y & mant) != 0ull)) {
        elev = __longlong_as_double((long long)y);
        n -= t;
      }
    }
    if (n > 0) {
      elev += c;
      n--;
    }
  }
}

// Lattice elevations from here up are more than the rounding of any carried
// elevation above the floor of the downward search.
__device__ __forceinline__ int above_floor(const DomainDesc& D) {
  return (int)floorf((float)D.elev_floor / (float)D.two_ha) + 2;
}

// The reference's search of one azimuth from (m, elev), given a lattice hit
// pattern that ends at the lowest miss M (kCodeAllMiss: no hits) or, for a
// code of k_sweep_repair, its stop. Returns true when it went up; n counts
// the steps (one ray each after the first).
__device__ __forceinline__ bool replay(int code, const DomainDesc& D, int safe, int& m,
                                       double& elev, int& n) {
  const int from = m;
  bool up = m < code;
  int stop = up ? code : min(m, max(code, safe) - 1);
  if (code >= kCodeStop) {
    stop = ((code - kCodeStop) >> 1) - 2000;
    up = (code - kCodeStop) & 1;
    if (up ? stop < m : stop > m) stop = m;
  }
  add_steps(elev, up ? D.two_ha : -D.two_ha, abs(stop - m));
  m = stop;
  if (code < kCodeStop && !up) {
    while (m >= code && elev > D.elev_floor) {
      m--;
      elev -= D.two_ha;
    }
  }
  n = abs(m - from);
  return up;
}

// First elevation of azimuth a: carried, or given (DomainDesc::start_m; 0 for
// the first azimuth, cpp:511).
__device__ __forceinline__ void chain_start(const DomainDesc& D, int cell, int a, int& m,
                                            double& elev) {
  if (a == 0) {
    m = 0;
    elev = 0.0;
  }
  if (D.start_m && (D.start_all || a % (D.L / D.groups) == 0)) {
    m = clamp_start(D.start_m[(long long)a * D.ncell + cell]);
    elev = (double)m * D.two_ha;
  }
}

// A warp per listed cell: replays the cell's azimuths and searches the ones
// left open by rays, 32 elevations at a time. Latency of a few border cells: 20,000
// to 70,000 cycles per round of 32 rays, whose grazing ones walk the whole track, 2.1
// rounds per open azimuth (57k cells 0.18 ms, 1.2M cells at 100 m 1.3). Neither five to
// eight blocks per SM nor list entries four at a time changed it.
template <bool kPrecise>
__global__ void __launch_bounds__(128)
    k_sweep_repair(const DomainDesc* __restrict__ doms, int ndom, const int* __restrict__ order,
                   const int* __restrict__ list, const int* __restrict__ list_n,
                   int* __restrict__ next, int s_full, int* __restrict__ err) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (*err & kErrGrid) return;
  const int n = *list_n;
  for (;;) {
    int w = 0;
    if (lane == 0) w = *(volatile int*)err & kErrGrid ? n : atomicAdd(next, 1);
    w = __shfl_sync(kFull, w, 0);
    if (w >= n) return;
    const long long gid = order[list[w]];
    const DomainDesc& D = doms[domain_of(doms, ndom, gid)];
    const GridDesc& g = *D.grid;
    const int cell = (int)(gid - D.cell_offset);
    const int p = list[w] - (int)D.k_begin;
    if (!check_ok(p >= 0 && p < D.ncell_traced && cell >= 0 && cell < D.ncell, kCheckPosition,
                  list[w], err))
      continue;
    const long long nc = D.ncell;
    const float4* fr = cell_rows<kPrecise>(D, p);
    const float4 fu = __ldg(fr + kFrameNormal), fn = __ldg(fr + kFrameNorth),
                 fe = __ldg(fr + kFrameEast);
    const float ho = __ldg(&fr[kFrameOrigin].w);
    const int safe = above_floor(D);
    int codes = 0;
    int m = 0, run = 0, before = 0;
    double elev = 0.0;
    for (int a = 0; a < D.L; a++) {
      chain_start(D, cell, a, m, elev);
      int16_t* slot = D.codes + (long long)a * D.ncell + cell;
      if ((a & 31) == 0 && a + lane < D.L) codes = slot[(long long)lane * nc];
      const int code = __shfl_sync(kFull, codes, a & 31);
      int steps;
      // Where this azimuth's sweep began: the hits below that are not known.
      int from = s_full;
      if (run_start(D, p, run) == a) {
        from = a == 0 ? 0 : max(s_full, kRunStart);
        run++;
      } else if (before > kCodeAllMiss) {
        from = max(s_full, before - start_drop(D));
      }
      before = code;
      if (code != kCodeGap && (m >= from || code == kCodeAllMiss)) {
        replay(code, D, safe, m, elev, steps);
        continue;
      }
      const double2 cs = __ldg(&D.azim_cs[a]);
      const float c = (float)cs.x, e = (float)cs.y;
      const float hx = __fmaf_rn(c, fn.x, e * fe.x);
      const float hy = __fmaf_rn(c, fn.y, e * fe.y);
      const float hz = __fmaf_rn(c, fn.z, e * fe.z);
      auto ray_hits = [&](int mm) {
        const double2 ecs = elevation(D, mm);
        const Ray r = table_ray<kPrecise>(D, p, a, ecs);
        // Beyond the zenith the ray runs along the opposite azimuth.
        const float sg = ecs.x < 0.0 ? -1.f : 1.f;
        const Track tr = make_track(g, fn.w, fe.w, sg * hx, sg * hy, sg * hz, fu.x,
                                    fu.y, fu.z);
        const float c = fmaxf(fabsf((float)ecs.x), 1e-7f);
        return grid_ray<kPrecise>(D, g, r, tr, ho, __fdiv_rn((float)ecs.y, c), err);
      };
      // Lanes 0-15: m .. m + 15; lanes 16-31: m - 1 .. m - 16.
      unsigned hits = __ballot_sync(kFull, ray_hits(lane < 16 ? m + lane : m - (lane - 15)));
      bool up = hits & 1u;
      if (up) {
        int base = m, have = 16, left = kMaxUpSteps;
        for (;;) {
          const unsigned miss = ~hits & (have == 32 ? kFull : 0xFFFFu);
          const int reach = miss ? __ffs(miss) - 1 : have;  // first miss at base + reach
          const int to = min(base + reach, m + left);       // up to there
          add_steps(elev, D.two_ha, to - m);
          left -= to - m;
          m = to;
          if (miss || left == 0) break;
          base += have;
          have = 32;
          hits = __ballot_sync(kFull, ray_hits(base + lane));
        }
      } else {
        int base = m - 1, have = 16;
        unsigned below = hits >> 16;
        for (;;) {
          // Down to the first hit, the last of the rays at hand, or near the floor.
          const int hit_at = below ? __ffs(below) - 1 : 64;
          int q = max(0, min(min(have, hit_at + 1), m - safe + 1));
          add_steps(elev, -D.two_ha, q);
          m -= q;
          bool hit = q == hit_at + 1;
          for (; q < have && elev > D.elev_floor && !hit; q++) {
            m--;
            elev -= D.two_ha;
            hit = below >> q & 1u;
          }
          if (hit || !(elev > D.elev_floor)) break;
          base -= have;
          have = 32;
          below = __ballot_sync(kFull, ray_hits(base - lane));
        }
      }
      if (m > kMaxStop) {  // many turns under a roof: the tree search carries on
        if (lane == 0) atomicOr(err, kErrGrid);
        break;
      }
      if (lane == 0) *slot = (int16_t)(kCodeStop + (((m + 2000) << 1) | (up ? 1 : 0)));
    }
  }
}

// ---------------------------------------------------------------------------
// Outputs
// ---------------------------------------------------------------------------

// The reference's search of every traced cell on its hit patterns: carried
// elevations, clip, sector means, SVF sums, ray count (cpp:490-555, 736-754).
// Bound by the FP64 pipe (60 % busy) and by what the lanes of a warp do not
// share of the walk up and down: with an FP64 addition per elevation step 1.2M cells
// took 2.05 ms and 500 cells 0.157 (border cells step down to the floor), with
// add_steps 0.76 and 0.051. Codes come four azimuths at a time, packed, and the
// loop over them is not unrolled: eight times over it ran out of the
// instruction cache.
template <bool kRefine1>
__device__ __forceinline__ unsigned finish_sweep(const DomainDesc& D, int cell, int* err) {
  const long long nc = D.ncell;
  const float inv_ha = (float)(1.0 / D.hori_acc);
  const double ha = D.hori_acc, refine = (double)D.refine;
  const int span = D.L / D.groups, safe = above_floor(D);
  int m = 0;
  double elev = 0.0, sector = 0.0, svf = 0.0, part = 0.0;
  unsigned rays = 0;
  int in_sector = 0, row = 0, in_group = 0;
#pragma unroll 1
  for (int a0 = 0; a0 < D.L; a0 += 4) {
    unsigned long long codes = 0;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (a0 + u < D.L)
        codes |= (unsigned long long)(uint16_t)D.codes[(long long)(a0 + u) * nc + cell] << (16 * u);
    const int end = min(a0 + 4, D.L);
#pragma unroll 1
    for (int a = a0; a < end; a++, codes >>= 16) {
      chain_start(D, cell, a, m, elev);
      int steps;
      const bool up = replay((int16_t)codes, D, safe, m, elev, steps);
      rays += 1u + (unsigned)steps;
      double h = up ? elev - ha : elev + ha;
      const int j = up ? 2 * m - 1 : 2 * m + 1;
      if (D.raw_j) D.raw_j[(long long)a * nc + cell] = (int16_t)j;
      if (h < 0.0) h = 0.0;
      if (kRefine1) {
        svf = svf + finish_svf_term(D, h, inv_ha);
        if (check_ok(cell >= 0 && cell < nc && a < D.nhori, kCheckOutput, a * nc + cell, err))
          D.horizon[(long long)a * nc + cell] = __dmul_rn(div_pi_rn(h), 180.0);
      } else {
        part = part + lattice_svf_term(D, h, j);
        sector = sector + h;
        if (++in_sector == D.refine) {
          if (check_ok(cell >= 0 && cell < nc && row < D.nhori, kCheckOutput, row * nc + cell, err))
            D.horizon[(long long)row * nc + cell] = __dmul_rn(div_pi_rn(sector), 180.0) / refine;
          sector = 0.0;
          in_sector = 0;
          row++;
        }
        if (++in_group == span) {
          svf = a + 1 == span ? part : svf + part;
          part = 0.0;
          in_group = 0;
        }
      }
    }
  }
  D.skyview[cell] = svf / (double)D.L;
  return rays;
}

// With D.done (a batch): the cells done of each domain, and the time of its last one.
__global__ void k_sweep_finish(const DomainDesc* __restrict__ doms, int ndom, int first, int total,
                               unsigned long long* __restrict__ counters,
                               int* __restrict__ err) {
  const int k = first + blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long rays = 0;
  const bool mine = k < first + total && !(*err & kErrGrid);
  int lo = 0;
  if (mine) {
    int hi = ndom - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (doms[mid].k_begin <= k) lo = mid;
      else hi = mid - 1;
    }
    const DomainDesc& D = doms[lo];
    const int cell = D.cell_begin + (int)(k - D.k_begin);
    rays = D.refine == 1 ? finish_sweep<true>(D, cell, err) : finish_sweep<false>(D, cell, err);
  }
  if (doms[0].done) {
    __threadfence();  // the outputs before the count
    const unsigned peers = __match_any_sync(0xffffffffu, mine ? lo : -1);
    if (mine && (int)(threadIdx.x & 31) == __ffs(peers) - 1) {
      const DomainDesc& D = doms[lo];
      const unsigned long long n = __popc(peers);
      if (atomicAdd(&D.done[0], n) + n == (unsigned long long)D.ncell_traced) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        D.done[1] = now;
      }
    }
  }
  rays = warp_sum_u64(rays);
  if ((threadIdx.x & 31) == 0 && rays) atomicAdd(&counters[0], rays);
}

}  // namespace

long long sweep_cells_cap(long long n_tri) { return std::max(4096ll, 5 * n_tri / 2); }
long long sweep_refs_cap(long long n_tri) { return 12 * n_tri + 4096; }
size_t sweep_frame_floats(bool precise) { return precise ? 20 : 16; }
float sweep_holes_allowed(float cells) { return kHolesCall + cells / kHolesCells; }

cudaError_t sweep_edge_cells(const int* cov, int nvert, int ncell, int begin, int count,
                             uint32_t* scratch, int* edge, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * (size_t)ncell, s);
  if (e != cudaSuccess || nvert <= 0) return e;
  k_full_vertices<<<grid_for(nvert, 256), 256, 0, s>>>(cov, nvert, scratch);
  k_edge_cells<<<grid_for(count, 256), 256, 0, s>>>(scratch, begin, count, edge);
  note_launches(2);
  return cudaGetLastError();
}

cudaError_t sweep_grid(const float* vert32, const float* vert_lo, const int* vot, int n_tri,
                       int n_vert, int tri_base, float tfar, float org_elev, float cells,
                       float missing, const int* edge, int ndom, const SweepBuffers& b, Tri* tris,
                       float4* tri_lo, int* err, cudaStream_t s) {
  const long long cap0 = sweep_cells_cap(n_tri);
  cudaError_t e = cudaMemsetAsync(b.count, 0, sizeof(uint32_t) * (size_t)(cap0 + 1), s);
  if (e != cudaSuccess) return e;
  k_grid_init<<<1, 1, 0, s>>>(b.bounds);
  k_gnomonic<<<grid_for(n_vert, 256), 256, 0, s>>>(vert32, n_vert, b.gv, b.bounds);
  k_grid_setup<<<1, 1, 0, s>>>(b.bounds, n_tri, cap0, tfar, org_elev, cells, missing, edge, ndom,
                               b.grid, err);
  note_launches(3);
  if (n_tri > 0) {
    k_grid_count<<<grid_for(n_tri, 256), 256, 0, s>>>(vert32, vert_lo, vot, n_tri, b.gv, b.grid,
                                                      b.count, cap0, tris, vert_lo ? tri_lo : nullptr, err);
    note_launches(1);
  }
  e = scan_exclusive_u32(b.count, b.start, cap0 + 1, b.total, b.partials, s);
  if (e != cudaSuccess) return e;
  if (n_tri > 0) {
    k_grid_fill<<<grid_for(n_tri, 256), 256, 0, s>>>(vot, n_tri, tri_base, b.gv, b.grid, b.count, b.start,
                                                     cap0, b.refs, sweep_refs_cap(n_tri), err);
    note_launches(1);
  }
  k_grid_heights<<<grid_for(cap0, 256), 256, 0, s>>>(b.grid, b.start, b.refs,
                                                     sweep_refs_cap(n_tri), tri_base, vot, b.gv,
                                                     cap0, n_tri, b.top, b.low, b.planes, err);
  note_launches(1);
  for (int l = 2; l <= 8; l += 2) {
    k_grid_up<<<grid_for(cap0 >> (2 * l), 128), 128, 0, s>>>(b.grid, l, cap0, b.top, b.low,
                                                             b.planes, err);
    note_launches(1);
  }
  return cudaGetLastError();
}

// Blocks of a kernel that are resident on the device at once; `wanted` per SM, for
// which shared memory is set aside and the rest left to L1 (FP64 ray mode with the
// share of six blocks where five run: 7.7 ms, with theirs 7.15).
template <typename K>
static long long resident_blocks(K kernel, int block, int wanted) {
  int dev = 0, sms = 0, per_sm = 0;
  prefer_l1(kernel, wanted);
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0);
  return (long long)sms * (per_sm > 0 ? per_sm : 1);
}

template <bool kPrecise>
static cudaError_t launch_search(const DomainDesc* doms, int ndom, const int32_t* order, int first,
                                 int total, int total_items, int s_full, int* work, int* list,
                                 unsigned* listed, const SweepScene& sc, int* err,
                                 cudaStream_t s) {
  // Fewer items than resident threads go to all warps, a few lanes each: the
  // lanes of a warp wait for one another's triangles and azimuths (500 cells x 24
  // azimuths: 288 us in full warps, 187 with four lanes per warp).
  const long long resident = resident_blocks(
      k_sweep<kPrecise>, kSweepBlock, kPrecise ? HZ_SWEEP_MIN_BLOCKS_EXACT : HZ_SWEEP_MIN_BLOCKS);
  const long long lanes = std::min(
      32ll, std::max(1ll, ((long long)total_items + resident * kWarps - 1) / (resident * kWarps)));
  const long long most = ((long long)total_items + lanes * kWarps - 1) / (lanes * kWarps);
  k_sweep<kPrecise><<<(unsigned)std::min(resident, most), kSweepBlock, 0, s>>>(
      doms, ndom, order, total_items, work, s_full, list, work + 1, listed, sc, (int)lanes, err);
  note_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (total_items > total) {
    k_sweep_runs<<<grid_for(total, 128), 128, 0, s>>>(doms, ndom, first, total, list, work + 1, listed,
                                                      order, err);
    note_launches(1);
  }
  const long long blocks = std::min(resident_blocks(k_sweep_repair<kPrecise>, 128, 4),
                                    ((long long)total + 3) / 4);
  k_sweep_repair<kPrecise><<<(unsigned)blocks, 128, 0, s>>>(doms, ndom, order, list, work + 1,
                                                            work + 2, s_full, err);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t sweep_frames(const DomainDesc* doms, int ndom, const int32_t* order, int total,
                         bool precise, cudaStream_t s) {
  if (total <= 0 || ndom <= 0) return cudaSuccess;
  if (precise) k_sweep_frames<true><<<grid_for(total, 128), 128, 0, s>>>(doms, ndom, order, total);
  else k_sweep_frames<false><<<grid_for(total, 128), 128, 0, s>>>(doms, ndom, order, total);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t sweep_search(const DomainDesc* doms, const SweepGroup& group, const int32_t* order,
                         int s_full, int* work, int* list, unsigned* listed, const SweepAll& all,
                         unsigned long long* counters, int* err, bool precise, cudaStream_t s) {
  if (group.total <= 0 || group.ndom <= 0) return cudaSuccess;
  doms += group.first;
  list += group.k_begin;
  const SweepScene sc{all.tris,   all.tri_lo, all.refs,    all.start,
                      all.planes, all.n_tri,  all.n_cells, all.n_refs};
  // work[0]: taken items, work[1]: listed cells, work[2]: taken by the repair.
  const cudaError_t e =
      precise ? launch_search<true>(doms, group.ndom, order, group.k_begin, group.total,
                                    (int)group.items, s_full, work, list, listed, sc, err, s)
              : launch_search<false>(doms, group.ndom, order, group.k_begin, group.total,
                                     (int)group.items, s_full, work, list, listed, sc, err, s);
  if (e != cudaSuccess) return e;
  k_sweep_finish<<<grid_for(group.total, 128), 128, 0, s>>>(doms, group.ndom, group.k_begin,
                                                            group.total, counters, err);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace hz
