// ws_grid.cu — grid-side kernels of the substep (js/solver.js:865-1636, 2629-2653).
//
// Each kernel cites the reference lines it restates. Grid kernels are
// HBM-bound streaming passes; their algorithmic bytes per element are listed
// next to each launcher and used for the roofline report.
#include "ws_kernels.cuh"
#include <algorithm>
#include <cub/cub.cuh>

// ------------------------------------------------------------ face decoding
struct FaceIJK { int comp, i, j, k; long long local; };
// 32-bit index arithmetic: face counts stay below 2^32 for grids up to 1000^3
__device__ __forceinline__ FaceIJK decode_face(const Dims& d, long long f64) {
  FaceIJK r;
  unsigned f = (unsigned)f64, nx = d.nx, ny = d.ny, uN = (unsigned)d.uN, vN = (unsigned)d.vN;
  if (f < uN) {
    r.comp = 0; r.local = f;
    unsigned t = fastdiv(f, d.dnx1); r.i = (int)(f - t * (nx + 1));
    unsigned k = fastdiv(t, d.dny); r.j = (int)(t - k * ny); r.k = (int)k;
  } else if (f < uN + vN) {
    unsigned g = f - uN; r.comp = 1; r.local = g;
    unsigned t = fastdiv(g, d.dnx); r.i = (int)(g - t * nx);
    unsigned k = fastdiv(t, d.dny1); r.j = (int)(t - k * (ny + 1)); r.k = (int)k;
  } else {
    unsigned g = f - uN - vN; r.comp = 2; r.local = g;
    unsigned t = fastdiv(g, d.dnx); r.i = (int)(g - t * nx);
    unsigned k = fastdiv(t, d.dny); r.j = (int)(t - k * ny); r.k = (int)k;
  }
  return r;
}
__device__ __forceinline__ void decode_cell(const Dims& d, long long c64, int& i, int& j, int& k) {
  unsigned c = (unsigned)c64, nx = d.nx, ny = d.ny;
  unsigned t = fastdiv(c, d.dnx); i = (int)(c - t * nx);
  unsigned kk = fastdiv(t, d.dny); j = (int)(t - kk * ny); k = (int)kk;
}
// the two cells a face separates; boundary=true for the domain planes
__device__ __forceinline__ bool face_cells(const Dims& d, const FaceIJK& F, long long& cL, long long& cR) {
  long long nx = d.nx, ny = d.ny;
  if (F.comp == 0) {
    if (F.i == 0 || F.i == d.nx) return true;
    cR = ((long long)F.k * ny + F.j) * nx + F.i; cL = cR - 1;
  } else if (F.comp == 1) {
    if (F.j == 0 || F.j == d.ny) return true;
    cR = ((long long)F.k * ny + F.j) * nx + F.i; cL = cR - nx;
  } else {
    if (F.k == 0 || F.k == d.nz) return true;
    cR = ((long long)F.k * ny + F.j) * nx + F.i; cL = cR - nx * ny;
  }
  return false;
}

// ------------------------------------------------------------ static types
// _rasterizeStatic static part, js/solver.js:872-900: terrain voxel at the
// cell centre, plus the closed domain shell.
__global__ void k_static_types(Dims d, TerrainDev t, double coreR, uint8_t* __restrict__ st) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells) return;
  int i, j, k; decode_cell(d, c, i, j, k);
  bool shell = (j == 0 || j == d.ny - 1 || k == 0 || k == d.nz - 1 || i == 0 || i == d.nx - 1);
  bool rock;
  if (t.has) {
    int vx = jtrunc((i + 0.5) * d.dx / t.dv), vy = jtrunc((j + 0.5) * d.dx / t.dv), vz = jtrunc((k + 0.5) * d.dx / t.dv);
    if (vx < 0) vx = 0; else if (vx >= t.n) vx = t.n - 1;
    if (vy < 0) vy = 0; else if (vy >= t.n) vy = t.n - 1;
    if (vz < 0) vz = 0; else if (vz >= t.n) vz = t.n - 1;
    rock = t.solid[((long long)vz * t.n + vy) * t.n + vx] == 1;
  } else {
    double dx2 = (i + 0.5) * d.dx - d.cx, dy2 = (j + 0.5) * d.dx - d.cy, dz2 = (k + 0.5) * d.dx - d.cz;
    rock = dx2 * dx2 + dy2 * dy2 + dz2 * dz2 < coreR * coreR;
  }
  st[c] = (shell || rock) ? WS_SOLID : WS_AIR;
}
// rock within one cell of each interior cell (the shell's own solid cells do
// not count: rock_cell_at clamps to the interior)
__global__ void k_near_rock(Dims d, const uint8_t* __restrict__ st, uint8_t* __restrict__ near) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells) return;
  int i, j, k; decode_cell(d, c, i, j, k);
  bool rock = false;
  for (int z = max(k - 1, 1); z <= min(k + 1, d.nz - 2); z++)
    for (int y = max(j - 1, 1); y <= min(j + 1, d.ny - 2); y++)
      for (int x = max(i - 1, 1); x <= min(i + 1, d.nx - 2); x++)
        rock |= st[((long long)z * d.ny + y) * d.nx + x] == WS_SOLID;
  near[c] = rock ? WS_SOLID : WS_AIR;
}
void launch_static_types(const Dims& d, const TerrainDev& t, double coreR, uint8_t* st, uint8_t* nearRock, cudaStream_t s) {
  k_static_types<<<grid_for(d.nCells, 256), 256, 0, s>>>(d, t, coreR, st);
  k_near_rock<<<grid_for(d.nCells, 256), 256, 0, s>>>(d, st, nearRock);
}

// _buildPlanetGravity, js/solver.js:1177-1210: unit-g radial geometry per face
__global__ void k_gravity_geometry(Dims d, double oceanR, float* __restrict__ g) {
  long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (f >= d.F) return;
  FaceIJK F = decode_face(d, f);
  double g0 = oceanR * oceanR, ex, ey, ez, e;
  if (F.comp == 0) { ex = F.i * d.dx - d.cx; ey = (F.j + 0.5) * d.dx - d.cy; ez = (F.k + 0.5) * d.dx - d.cz; e = ex; }
  else if (F.comp == 1) { ex = (F.i + 0.5) * d.dx - d.cx; ey = F.j * d.dx - d.cy; ez = (F.k + 0.5) * d.dx - d.cz; e = ey; }
  else { ex = (F.i + 0.5) * d.dx - d.cx; ey = (F.j + 0.5) * d.dx - d.cy; ez = F.k * d.dx - d.cz; e = ez; }
  double r3 = pow(ex * ex + ey * ey + ez * ez, 1.5);
  if (r3 == 0) r3 = 1e-9;
  g[f] = (float)(-g0 * e / r3);
}
void launch_gravity_geometry(const Dims& d, double oceanR, float* g, cudaStream_t s) {
  k_gravity_geometry<<<grid_for(d.F, 256), 256, 0, s>>>(d, oceanR, g);
}

// ------------------------------------------------------------ 1. clear + raster
// u..wW.fill(0) (js/solver.js:2569-2570) and cellType <- static types
// (:865-871). Bytes: 8F (acc) + 2N.
// 16-byte stores: two faces of the accumulator, sixteen cell types per
// thread (both buffers are separate allocations, 256-byte aligned). In a
// substep (bricks) only the accumulator of the last substep's work list is
// cleared, unless a forced full pass follows; the list's counter starts anew.
__device__ __forceinline__ unsigned cell_faces(const Dims& d, int i, int j, int k, unsigned (&f)[3]) {
  const unsigned nx = (unsigned)d.nx, ny = (unsigned)d.ny, row = (unsigned)k * ny + (unsigned)j;
  const unsigned c = row * nx + (unsigned)i;
  f[0] = c + row;                                       // u: rows of nx + 1
  f[1] = (unsigned)d.uN + c + (unsigned)k * nx;         // v: planes of ny + 1 rows
  f[2] = (unsigned)(d.uN + d.vN) + c;
  return c;
}
// A block of 256 threads on four bricks of the work list: the list holds
// x-neighbours side by side, so a warp takes two y rows of all four (32 cells
// along x by 2 lie in 2 to 4 lines) rather than half of one brick (8 rows of
// 16 bytes). The brick's number among the four, and the cell in the brick.
__device__ __forceinline__ void quad_cell(int& q, int& li, int& lj, int& lk) {
  const int t = threadIdx.x;
  li = t & 3; q = (t >> 2) & 3; lj = ((t >> 4) & 1) | ((t >> 4) & 2); lk = t >> 6;
}
__global__ void __launch_bounds__(256) k_clear_raster(Dims d, GridDev g, DevStatus* st, BrickSet B, int bricks) {
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const long long F2 = d.F >> 1, n16 = d.nCells >> 4;
  for (long long t = t0; t < n16; t += step)
    reinterpret_cast<uint4*>(g.type)[t] = reinterpret_cast<const uint4*>(g.staticTypes)[t];
  if (t0 < (d.nCells & 15)) { const long long c = (n16 << 4) + t0; g.type[c] = g.staticTypes[c]; }
  if (t0 == 0) {
    st->umaxBits = 0u; st->airborne = 0; st->nFluid = 0; st->oddFluid = 0;
    if (bricks) B.count[0] = 0;
  }
  if (!bricks || *B.forceAll) {
    for (long long t = t0; t < F2; t += step) reinterpret_cast<float4*>(g.acc)[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t0 == 0 && (d.F & 1)) g.acc[d.F - 1] = make_float2(0.f, 0.f);
    return;
  }
  const int n = B.count[1];                             // the last substep's list
  int q, li, lj, lk;
  quad_cell(q, li, lj, lk);
  for (int it = blockIdx.x * 4 + q; it < n; it += gridDim.x * 4) {
    int bx, by, bz;
    brick_coords(B, B.list[it], bx, by, bz);
    const int i = bx * 4 + li, j = by * 4 + lj, k = bz * 4 + lk;
    if (i >= d.nx || j >= d.ny || k >= d.nz) continue;
    unsigned f[3];
    cell_faces(d, i, j, k, f);
#pragma unroll
    for (int a = 0; a < 3; a++) g.acc[f[a]] = make_float2(0.f, 0.f);
    if (i == d.nx - 1) g.acc[f[0] + 1] = make_float2(0.f, 0.f);
    if (j == d.ny - 1) g.acc[f[1] + d.nx] = make_float2(0.f, 0.f);
    if (k == d.nz - 1) g.acc[f[2] + d.nx * d.ny] = make_float2(0.f, 0.f);
  }
}
void launch_clear_raster(const Dims& d, const GridDev& g, DevStatus* st, const BrickSet& B, bool bricks, cudaStream_t s) {
  const unsigned need = grid_for(bricks ? (d.nCells >> 4) + 16 : (d.F >> 1) + 16, 256);
  k_clear_raster<<<std::min(std::max(need, 148u * 2u), 148u * 8u), 256, 0, s>>>(d, g, st, B, bricks ? 1 : 0);
}

// ------------------------------------------------------------ 2. mark fluid
// _markFluidCells, js/solver.js:945-1000 (sphere). Bytes: 13P + N.
// The range and NaN latch of the marking on the stored float position: a
// float exceeds the double bound exactly when it exceeds the largest float
// not above it.
__device__ __forceinline__ bool mark_sound_f(const Dims& d, float x, float y, float z, int* err) {
  if (!(isfinite(x) && isfinite(y) && isfinite(z))) { atomicOr(err, WS_DERR_NAN); return false; }
  if (x < 0.f || y < 0.f || z < 0.f || x > __double2float_rd(d.W) || y > __double2float_rd(d.H) ||
      z > __double2float_rd(d.D)) atomicOr(err, WS_DERR_RANGE);
  return true;
}
// whether a float position may pass the sky test's radius or row condition:
// the float radius is within 1e-6 of the double one, so below the bound less
// 1e-5 of it the double test cannot pass
__device__ __forceinline__ bool mark_high_f(const Dims& d, double oceanR, float x, float y, float z, int j) {
  const float rx = x - (float)d.cx, ry = y - (float)d.cy, rz = z - (float)d.cz;
  const float bound = (float)((oceanR + 0.3) * (oceanR + 0.3) * (1 - 1e-5));
  return !(rx * rx + ry * ry + rz * rz < bound) || j >= d.ny - 2;
}
// whether a grid-coupled particle in grid row j turns airborne
__device__ __forceinline__ bool mark_airborne(const Dims& d, const GridDev& g, const TerrainDev& t, double oceanR,
                                              double coreR, int j, double X, double Y, double Z) {
  double rx = X - d.cx, ry = Y - d.cy, rz = Z - d.cz;
  double radius2 = rx * rx + ry * ry + rz * rz;
  double skyAlt = 2 * d.dx > 0.3 ? 2 * d.dx : 0.3;
  if (radius2 > (oceanR + 0.3) * (oceanR + 0.3) &&
      sqrt(radius2) - terrain_radius_at(t, coreR, X, Y, Z) > skyAlt &&
      !(t.has && rock_cell_at(d, g.staticTypes, X, Y, Z))) return true;
  return j >= d.ny - 2 && sqrt(radius2) - terrain_radius_at(t, coreR, X, Y, Z) > 0.3;
}
// the cell a grid-coupled particle marks, or -1 (not coupled, or it turns airborne: pflag 1)
__device__ __forceinline__ long long mark_cell(const Dims& d, const GridDev& g, PartsDev& P, const TerrainDev& t,
                                               double oceanR, double coreR, int p, int fl, double X, double Y,
                                               double Z) {
  if (fl != 0) return -1;
  int i = jfloor_clamp(over_dx(d, X), 0, d.nx - 1);
  int j = jfloor_clamp(over_dx(d, Y), 0, d.ny - 1);
  int k = jfloor_clamp(over_dx(d, Z), 0, d.nz - 1);
  if (mark_airborne(d, g, t, oceanR, coreR, j, X, Y, Z)) { P.pflag[p] = 1; return -1; }
  return ((long long)k * d.ny + j) * d.nx + i;
}
// Warp-aggregated increment of count[key] for every lane with key >= 0: the
// lanes holding one key share a single atomic; each gets its own rank. All
// 32 lanes of the warp call it (lanes without work pass -1).
__device__ __forceinline__ int warp_rank_inc(int* count, int key) {
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader && key >= 0) base = atomicAdd(&count[key], __popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}
// the sort key of cell (i, j, k): its 4^3 brick times 64 plus its place in the brick
__device__ __forceinline__ int brick_key(const GridDev& g, int i, int j, int k) {
  return ((((k >> 2) * g.nby + (j >> 2)) * g.nbx + (i >> 2)) << 6) | ((k & 3) << 4) | ((j & 3) << 2) | (i & 3);
}
// Two particles per thread: both particles' loads, then both cells' type
// loads, then the (idempotent) stores, so the two chains overlap. With a
// cell sort (cs.count set) every particle that P2G will scatter (marked, with
// a finite velocity) is also counted in its cell, and its rank recorded.
__global__ void k_mark_fluid(Dims d, GridDev g, PartsDev P, TerrainDev t, double oceanR, double coreR, CellSort cs,
                             int* err) {
  const int p0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x), p1 = p0 + 1;
  const bool has0 = p0 < P.nP, has1 = p1 < P.nP;
  long long c0 = -1, c1 = -1;
  bool fin0 = false, fin1 = false;
  if (has0) {
    const int fl0 = P.pflag[p0], fl1 = has1 ? P.pflag[p1] : 1;
    const double X0 = P.px[p0], Y0 = P.py[p0], Z0 = P.pz[p0];
    const double X1 = has1 ? P.px[p1] : 0.0, Y1 = has1 ? P.py[p1] : 0.0, Z1 = has1 ? P.pz[p1] : 0.0;
    if (cs.count) {
      fin0 = isfinite(P.pvx[p0]) && isfinite(P.pvy[p0]) && isfinite(P.pvz[p0]);
      fin1 = has1 && isfinite(P.pvx[p1]) && isfinite(P.pvy[p1]) && isfinite(P.pvz[p1]);
    }
    // the first pass of a substep to read the positions: every particle must
    // be finite and inside the domain box (the reference's passes keep it there)
    particle_sound(d, X0, Y0, Z0, 0.0, 0.0, 0.0, err, true);
    if (has1) particle_sound(d, X1, Y1, Z1, 0.0, 0.0, 0.0, err, true);
    // the brick of every particle's cell seeds this substep's active bricks
    seed_cell(g, jfloor_clamp(over_dx(d, X0), 0, d.nx - 1), jfloor_clamp(over_dx(d, Y0), 0, d.ny - 1),
              jfloor_clamp(over_dx(d, Z0), 0, d.nz - 1));
    if (has1)
      seed_cell(g, jfloor_clamp(over_dx(d, X1), 0, d.nx - 1), jfloor_clamp(over_dx(d, Y1), 0, d.ny - 1),
                jfloor_clamp(over_dx(d, Z1), 0, d.nz - 1));
    c0 = mark_cell(d, g, P, t, oceanR, coreR, p0, fl0, X0, Y0, Z0);
    c1 = mark_cell(d, g, P, t, oceanR, coreR, p1, fl1, X1, Y1, Z1);
    const uint8_t t0 = c0 >= 0 ? g.type[c0] : (uint8_t)WS_SOLID, t1 = c1 >= 0 ? g.type[c1] : (uint8_t)WS_SOLID;
    if (t0 == WS_AIR) g.type[c0] = WS_FLUID;
    if (t1 == WS_AIR) g.type[c1] = WS_FLUID;
  }
  if (!cs.count) return;                                // uniform over the launch
  // a marked particle with a non-finite velocity stays off the grid and is latched
  if ((c0 >= 0 && !fin0) || (c1 >= 0 && !fin1)) atomicOr(err, WS_DERR_NAN);
  auto key_of = [&](long long c) { int i, j, k; cell_ijk(d, c, i, j, k); return brick_key(g, i, j, k); };
  const int k0 = c0 >= 0 && fin0 ? key_of(c0) : -1, k1 = c1 >= 0 && fin1 ? key_of(c1) : -1;
  const int r0 = warp_rank_inc(cs.count, k0), r1 = warp_rank_inc(cs.count, k1);
  if (has0) { cs.pcell[p0] = k0; cs.pslot[p0] = r0; }
  if (has1) { cs.pcell[p1] = k1; cs.pslot[p1] = r1; }
}
// Without the cell sort: four consecutive particles per thread (float4 and
// uchar4 loads), the seed brick stored once per run of particles in one
// brick, the cell types of all four loaded before any store, and a store
// once per run of particles in one cell. Same marks as k_mark_fluid.
__global__ void __launch_bounds__(256) k_mark_fluid_runs(Dims d, GridDev g, PartsDev P, TerrainDev t, double oceanR,
                                                         double coreR, int* err) {
  const int p0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (p0 >= P.nP) return;
  float xs[4], ys[4], zs[4];
  int fl[4];
  int nHave = 4;
  if (p0 + 3 < P.nP) {                                // the arrays are 16-byte aligned and p0 % 4 == 0
    const float4 X = *reinterpret_cast<const float4*>(P.px + p0), Y = *reinterpret_cast<const float4*>(P.py + p0);
    const float4 Z = *reinterpret_cast<const float4*>(P.pz + p0);
    const uchar4 F = *reinterpret_cast<const uchar4*>(P.pflag + p0);
    xs[0] = X.x; xs[1] = X.y; xs[2] = X.z; xs[3] = X.w; ys[0] = Y.x; ys[1] = Y.y; ys[2] = Y.z; ys[3] = Y.w;
    zs[0] = Z.x; zs[1] = Z.y; zs[2] = Z.z; zs[3] = Z.w; fl[0] = F.x; fl[1] = F.y; fl[2] = F.z; fl[3] = F.w;
  } else {
    nHave = P.nP - p0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const bool has = r < nHave;
      xs[r] = has ? P.px[p0 + r] : 0.f; ys[r] = has ? P.py[p0 + r] : 0.f; zs[r] = has ? P.pz[p0 + r] : 0.f;
      fl[r] = has ? P.pflag[p0 + r] : 1;
    }
  }
  long long c[4];
  int lastBrick = -1;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    c[r] = -1;
    if (r >= nHave) continue;
    const double X = xs[r], Y = ys[r], Z = zs[r];
    // the first pass of a substep to read the positions: every particle must
    // be finite and inside the domain box (the reference's passes keep it there)
    particle_sound(d, X, Y, Z, 0.0, 0.0, 0.0, err, true);
    // the brick of every particle's cell seeds this substep's active bricks
    const int i = jfloor_clamp(over_dx(d, X), 0, d.nx - 1), j = jfloor_clamp(over_dx(d, Y), 0, d.ny - 1);
    const int k = jfloor_clamp(over_dx(d, Z), 0, d.nz - 1);
    const int sb = ((k >> 2) * g.nby + (j >> 2)) * g.nbx + (i >> 2);
    if (g.seed && sb != lastBrick) { g.seed[sb] = 1; lastBrick = sb; }
    c[r] = mark_cell(d, g, P, t, oceanR, coreR, p0 + r, fl[r], X, Y, Z);
  }
  uint8_t ty[4];
#pragma unroll
  for (int r = 0; r < 4; r++) ty[r] = c[r] >= 0 ? g.type[c[r]] : (uint8_t)WS_SOLID;
#pragma unroll
  for (int r = 0; r < 4; r++)
    if (ty[r] == WS_AIR && (r == 0 || c[r] != c[r - 1])) g.type[c[r]] = WS_FLUID;
}
void launch_mark_fluid(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t,
                       double oceanR, double coreR, const CellSort* cs, DevStatus* st, cudaStream_t s) {
  if (P.nP <= 0) return;
  if (!cs) {
    k_mark_fluid_runs<<<grid_for((P.nP + 3) / 4, 256), 256, 0, s>>>(d, g, P, t, oceanR, coreR, &st->err);
    return;
  }
  k_mark_fluid<<<grid_for((P.nP + 1) / 2, 256), 256, 0, s>>>(d, g, P, t, oceanR, coreR, *cs, &st->err);
}

// ------------------------------------------------------------ 3. P2G scatter
// _p2gInto, js/solver.js:1035-1105: trilinear momentum + weight per face,
// one float2 vector atomic per face (momentum, weight). FP32 arithmetic: the
// face indices and fractions are exact (face_coords_f), the weights and
// terms carry FP32 rounding (a few 1e-8 relative against the double sums).
//
// Runs of consecutive particles: each thread scatters R (2 or 4) consecutive
// particles (the fill's lattice runs along x about a third of a cell apart).
// Per component it holds the eight (momentum, weight) sums of one stencil in
// registers. A particle whose stencil starts at the same face adds to them;
// one whose stencil starts one face further along x sends the four faces of
// the column left behind and keeps the other four as its own first column;
// any other sends all eight.
//
// In a whole substep without balls the fluid marking (section 2) rides along:
// it needs the same positions, its arithmetic runs while the load/store units
// are full of reductions, and P2G reads nothing that it writes.
//
// What bounds it: the reductions (lanes sent to L2). Before, with four
// particles a thread, all eight faces sent at each new stencil, and the
// marking as its own kernel: 106.6 + 22.3 us for 1.86M particles at 128^3,
// 789 + 152 us for 15.3M at 256^3, 43.1 + 12.5 us for 0.7M at 97^3; now 90,
// 612 and 34.5 us. Eight particles a thread hold too many registers (103, 660
// and 47 us).
template <int COMP, int R>
__device__ __forceinline__ void p2g_run_comp(const Dims& d, float2* __restrict__ acc, const float (&x)[R],
                                             const float (&y)[R], const float (&z)[R], const float (&v)[R],
                                             unsigned okMask) {
  unsigned sj, sk;
  face_strides32(d, COMP, sj, sk);
  const unsigned nx = (unsigned)d.nx, ny = (unsigned)d.ny, uN = (unsigned)d.uN, vN = (unsigned)d.vN;
  float m8[8], w8[8];                                 // corner q: x + 2 y + 4 z
  unsigned cur = 0xffffffffu;
  auto send = [&](int col) {                          // the four faces of column col (0: lower x)
    float2* p = acc + cur + col;
    atomicAdd(p, make_float2(m8[col], w8[col]));
    atomicAdd(p + sj, make_float2(m8[2 + col], w8[2 + col]));
    atomicAdd(p + sk, make_float2(m8[4 + col], w8[4 + col]));
    atomicAdd(p + sk + sj, make_float2(m8[6 + col], w8[6 + col]));
  };
#pragma unroll
  for (int r = 0; r < R; r++) {
    if (!((okMask >> r) & 1u)) continue;
    int i0, j0, k0; float tx, ty, tz;
    face_coords_f(d, COMP, x[r], y[r], z[r], i0, j0, k0, tx, ty, tz);
    const unsigned idx = COMP == 0 ? ((unsigned)k0 * ny + (unsigned)j0) * (nx + 1) + (unsigned)i0
                       : COMP == 1 ? uN + ((unsigned)k0 * (ny + 1) + (unsigned)j0) * nx + (unsigned)i0
                                   : uN + vN + ((unsigned)k0 * ny + (unsigned)j0) * nx + (unsigned)i0;
    if (idx != cur) {
      const bool next = idx == cur + 1u && cur != 0xffffffffu;
      if (cur != 0xffffffffu) {
        send(0);
        if (!next) send(1);
      }
#pragma unroll
      for (int q = 0; q < 8; q += 2) {                // column 1 becomes column 0, or both start anew
        m8[q] = next ? m8[q + 1] : 0.f; w8[q] = next ? w8[q + 1] : 0.f;
        m8[q + 1] = 0.f; w8[q + 1] = 0.f;
      }
      cur = idx;
    }
    const float s0 = 1.f - tx, s1 = tx, t0 = 1.f - ty, t1 = ty, r0 = 1.f - tz, r1 = tz;
    const float wA = s0 * t0, wB = s1 * t0, wC = s0 * t1, wD = s1 * t1;
    const float w[8] = { wA * r0, wB * r0, wC * r0, wD * r0, wA * r1, wB * r1, wC * r1, wD * r1 };
#pragma unroll
    for (int q = 0; q < 8; q++) { m8[q] = fmaf(w[q], v[r], m8[q]); w8[q] += w[q]; }
  }
  if (cur != 0xffffffffu) { send(0); send(1); }
}
// R consecutive values of a 16-byte aligned array (p0 a multiple of R), 0 past the end
template <int R>
__device__ __forceinline__ void load_run(const float* __restrict__ a, int p0, int n, float (&v)[R]) {
  if (p0 + R <= n) {
    if constexpr (R == 2) {
      const float2 l = *reinterpret_cast<const float2*>(a + p0);
      v[0] = l.x; v[1] = l.y;
    } else {
#pragma unroll
      for (int q = 0; q < R; q += 4) {
        const float4 l = *reinterpret_cast<const float4*>(a + p0 + q);
        v[q] = l.x; v[q + 1] = l.y; v[q + 2] = l.z; v[q + 3] = l.w;
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = p0 + r < n ? a[p0 + r] : 0.f;
  }
}
// The marking of one thread's R particles (as k_mark_fluid): range and
// NaN latch, seed bricks, the sky test, fluid cells. The cell types of this
// substep are the static ones and what this pass marks (no balls), so a cell
// is marked when its static type is air. Particles that turn airborne leave
// fl.
template <int R>
__device__ __forceinline__ void mark_run(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, double oceanR,
                                      double coreR, int p0, const float (&x)[R], const float (&y)[R],
                                      const float (&z)[R], int (&fl)[R], int* err) {
  int lastBrick = -1;
  long long lastCell = -1;
#pragma unroll
  for (int r = 0; r < R; r++) {
    if (p0 + r >= P.nP) continue;
    mark_sound_f(d, x[r], y[r], z[r], err);
    int i, j, k;
    cell_of_f(d, x[r], y[r], z[r], i, j, k);
    const int sb = ((k >> 2) * g.nby + (j >> 2)) * g.nbx + (i >> 2);
    if (sb != lastBrick) { g.seed[sb] = 1; lastBrick = sb; }
    if (fl[r] != 0) continue;
    if (mark_high_f(d, oceanR, x[r], y[r], z[r], j) &&
        mark_airborne(d, g, t, oceanR, coreR, j, x[r], y[r], z[r])) { P.pflag[p0 + r] = 1; fl[r] = 1; continue; }
    const long long c = ((long long)k * d.ny + j) * d.nx + i;
    if (c != lastCell) { lastCell = c; if (g.staticTypes[c] == WS_AIR) g.type[c] = WS_FLUID; }
  }
}
template <bool MARK, int R>
__global__ void __launch_bounds__(128, 8) k_p2g_runs(Dims d, GridDev g, PartsDev P, TerrainDev t, double oceanR,
                                                     double coreR, int* err) {
  const int p0 = R * (blockIdx.x * blockDim.x + threadIdx.x);
  if (p0 >= P.nP) return;
  float x[R], y[R], z[R], v[R];
  int fl[R];
  load_run<R>(P.px, p0, P.nP, x); load_run<R>(P.py, p0, P.nP, y); load_run<R>(P.pz, p0, P.nP, z);
  if (R == 4 && p0 + R <= P.nP) {
    const unsigned F = *reinterpret_cast<const unsigned*>(P.pflag + p0);
#pragma unroll
    for (int r = 0; r < R; r++) fl[r] = (int)((F >> (8 * r)) & 0xffu);
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) fl[r] = p0 + r < P.nP ? P.pflag[p0 + r] : 1;
  }
  if (MARK) mark_run<R>(d, g, P, t, oceanR, coreR, p0, x, y, z, fl, err);
  // a fluid particle with a non-finite state is left out of the grid and latched
  unsigned ok = 0;
#pragma unroll
  for (int r = 0; r < R; r++)
    if (fl[r] == 0) ok |= 1u << r;
  if (!ok) return;
  {
    float vy[R], vz[R];
    load_run<R>(P.pvx, p0, P.nP, v); load_run<R>(P.pvy, p0, P.nP, vy); load_run<R>(P.pvz, p0, P.nP, vz);
#pragma unroll
    for (int r = 0; r < R; r++)
      if (((ok >> r) & 1u) && !particle_sound_f(x[r], y[r], z[r], v[r], vy[r], vz[r], err)) ok &= ~(1u << r);
  }
  p2g_run_comp<0, R>(d, g.acc, x, y, z, v, ok);
  load_run<R>(P.pvy, p0, P.nP, v);                          // from L1: fewer registers than keeping all three
  p2g_run_comp<1, R>(d, g.acc, x, y, z, v, ok);
  load_run<R>(P.pvz, p0, P.nP, v);
  p2g_run_comp<2, R>(d, g.acc, x, y, z, v, ok);
}
template <bool MARK>
static void launch_p2g_runs(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, double oceanR,
                            double coreR, int* err, cudaStream_t s) {
  if (P.nP <= 0) return;
  // four particles a thread send fewer reductions, two leave more threads and
  // shorter chains (R = 4 against 2 in us: 10k particles 11.6/6.1, 0.7M
  // 37.5/34.5, 1.86M 90.1/90.4, 15.3M 612/647)
  if (P.nP < (3 << 19)) k_p2g_runs<MARK, 2><<<grid_for((P.nP + 1LL) / 2, 128), 128, 0, s>>>(d, g, P, t, oceanR, coreR, err);
  else k_p2g_runs<MARK, 4><<<grid_for((P.nP + 3LL) / 4, 128), 128, 0, s>>>(d, g, P, t, oceanR, coreR, err);
}
void launch_p2g(const Dims& d, const GridDev& g, const PartsDev& P, DevStatus* st, cudaStream_t s) {
  launch_p2g_runs<false>(d, g, P, TerrainDev{}, 0, 0, &st->err, s);
}
void launch_mark_p2g(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, double oceanR, double coreR,
                     DevStatus* st, cudaStream_t s) {
  launch_p2g_runs<true>(d, g, P, t, oceanR, coreR, &st->err, s);
}

// ------------------------------------------------------------ 3b. P2G in cell order
// The same scatter (_p2gInto, js/solver.js:1035-1105) over the particles
// sorted by cell, brick-major: the key of cell (i, j, k) is its 4^3 brick
// times 64 plus its place in the brick, so a brick's particles are one range
// of the permutation. One block per brick adds every particle's eight FP32
// (momentum, weight) terms per component into a shared-memory copy of the
// faces the brick's particles can reach (red.shared.add.f32), then sends one
// float2 atomic per touched face. Every FP32 term is the one k_p2g_runs adds;
// only the order of the FP32 sums differs. A particle whose stencil leaves
// the brick's faces (a ball pushed it after the binning) adds its terms to
// global memory directly.

// The stage-wise P2G, without a mark pass that counted: the particles P2G
// scatters (pflag 0, finite state) counted per cell, each with its rank.
__global__ void k_bin_cells(Dims d, GridDev g, PartsDev P, CellSort cs, int* err) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int key = -1;
  if (p < P.nP && P.pflag[p] == 0) {
    const double x = P.px[p], y = P.py[p], z = P.pz[p];
    if (particle_sound(d, x, y, z, P.pvx[p], P.pvy[p], P.pvz[p], err, false))
      key = brick_key(g, jfloor_clamp(over_dx(d, x), 0, d.nx - 1), jfloor_clamp(over_dx(d, y), 0, d.ny - 1),
                      jfloor_clamp(over_dx(d, z), 0, d.nz - 1));
  }
  const int r = warp_rank_inc(cs.count, key);          // every lane of the warp takes part
  if (p < P.nP) { cs.pcell[p] = key; cs.pslot[p] = r; }
}
// particle ids into their cells' ranges
__global__ void k_cell_scatter(int nP, CellSort cs, int* err) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nP) return;
  const int c = cs.pcell[p];
  if (c < 0) return;
  const int at = cs.start[c] + cs.pslot[p];
  if (at >= 0 && at < cs.cap) cs.perm[at] = p;
  else atomicOr(err, WS_DERR_RANGE);
}

// Shared-memory faces of one brick: per component the faces of the brick's
// cells widened by one along the two tangential axes (5 x 6 x 6 = 180), the
// component's own axis keeping its upper face. Momentum sums first, then
// the weights.
constexpr int kBrickFaces = 180;
// origin offset of component comp's face box from the brick's first cell, and its x and y extents
__device__ __forceinline__ void brick_face_box(int comp, int& oi, int& oj, int& ok, int& ex, int& ey) {
  oi = comp == 0 ? 0 : -1; oj = comp == 1 ? 0 : -1; ok = comp == 2 ? 0 : -1;
  ex = comp == 0 ? 5 : 6; ey = comp == 1 ? 5 : 6;
}
// one particle's eight terms of component comp: into the brick's faces when
// the whole stencil lies inside them, else straight to global memory
__device__ __forceinline__ void p2g_brick_comp(const Dims& d, float2* __restrict__ acc, float* sm, int comp,
                                               int fx, int fy, int fz, float x, float y, float z, float vel) {
  int i0, j0, k0; float tx, ty, tz;
  face_coords_f(d, comp, x, y, z, i0, j0, k0, tx, ty, tz);
  const float s0 = 1.f - tx, s1 = tx, t0 = 1.f - ty, t1 = ty, r0 = 1.f - tz, r1 = tz;
  const float wA = s0 * t0, wB = s1 * t0, wC = s0 * t1, wD = s1 * t1;
  const float w8[8] = { wA * r0, wB * r0, wC * r0, wD * r0, wA * r1, wB * r1, wC * r1, wD * r1 };
  int oi, oj, ok, ex, ey;
  brick_face_box(comp, oi, oj, ok, ex, ey);
  const int ez = comp == 2 ? 5 : 6;
  const int li = i0 - (fx + oi), lj = j0 - (fy + oj), lk = k0 - (fz + ok);
  if ((unsigned)li < (unsigned)(ex - 1) && (unsigned)lj < (unsigned)(ey - 1) && (unsigned)lk < (unsigned)(ez - 1)) {
    float* m = sm + comp * kBrickFaces;
    float* w = m + 3 * kBrickFaces;
    const int o = (lk * ey + lj) * ex + li, sj = ex, sk = ex * ey;
    const int o8[8] = { o, o + 1, o + sj, o + sj + 1, o + sk, o + sk + 1, o + sk + sj, o + sk + sj + 1 };
#pragma unroll
    for (int q = 0; q < 8; q++) {
      atomicAdd(&m[o8[q]], w8[q] * vel);
      atomicAdd(&w[o8[q]], w8[q]);
    }
  } else {
    long long idx, sj, sk;
    face_strides(d, comp, i0, j0, k0, idx, sj, sk);
    const long long o8[8] = { idx, idx + 1, idx + sj, idx + sj + 1, idx + sk, idx + sk + 1, idx + sk + sj,
                              idx + sk + sj + 1 };
#pragma unroll
    for (int q = 0; q < 8; q++) atomicAdd(&acc[o8[q]], make_float2(w8[q] * vel, w8[q]));
  }
}
// One block per brick (the brick list, or every brick when allBricks). The
// brick's particle range is cut into 32 lane chunks, so the 32 lanes of a
// warp work on particles about a 32nd of the range apart, mostly in
// different cells, and their shared-memory adds rarely meet on one address.
__global__ void __launch_bounds__(256) k_p2g_bricks(Dims d, GridDev g, PartsDev P, CellSort cs, BrickSet B,
                                                    int allBricks, int* err) {
  __shared__ float sm[6 * kBrickFaces];
  const int nB = allBricks ? B.nbx * B.nby * B.nbz : *B.count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = blockIdx.x; e < nB; e += gridDim.x) {
    const int b = allBricks ? e : B.list[e];
    const int s0 = cs.start[b << 6], n = cs.start[(b << 6) + 64] - s0;
    if (n <= 0) continue;                              // uniform over the block
    if (threadIdx.x < 64) cs.count[(b << 6) + threadIdx.x] = 0;   // zero again for the next binning
    if (s0 < 0 || s0 + n > cs.cap) { if (threadIdx.x == 0) atomicOr(err, WS_DERR_RANGE); continue; }
    int bx, by, bz;
    brick_coords(B, b, bx, by, bz);
    const int fx = bx * 4, fy = by * 4, fz = bz * 4;
    for (int t = threadIdx.x; t < 6 * kBrickFaces; t += blockDim.x) sm[t] = 0.f;
    __syncthreads();
    const int L = (n + 31) >> 5;                       // lane chunk
    for (int a = warp; a < L; a += 8) {
      const int at = lane * L + a;
      if (at >= n) continue;
      const int p = cs.perm[s0 + at];
      const float x = P.px[p], y = P.py[p], z = P.pz[p];
      const float u = P.pvx[p], v = P.pvy[p], w = P.pvz[p];
      p2g_brick_comp(d, g.acc, sm, 0, fx, fy, fz, x, y, z, u);
      p2g_brick_comp(d, g.acc, sm, 1, fx, fy, fz, x, y, z, v);
      p2g_brick_comp(d, g.acc, sm, 2, fx, fy, fz, x, y, z, w);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 3 * kBrickFaces; t += blockDim.x) {
      const float m = sm[t], wt = sm[t + 3 * kBrickFaces];
      if (wt == 0.f && m == 0.f) continue;            // a face no stencil reached
      const int comp = t / kBrickFaces, f = t - comp * kBrickFaces;
      int oi, oj, ok, ex, ey;
      brick_face_box(comp, oi, oj, ok, ex, ey);
      const int li = f % ex, lj = (f / ex) % ey, lk = f / (ex * ey);
      long long idx, sj, sk;
      face_strides(d, comp, fx + oi + li, fy + oj + lj, fz + ok + lk, idx, sj, sk);
      atomicAdd(&g.acc[idx], make_float2(m, wt));
    }
    __syncthreads();                                   // sm is cleared for the next brick
  }
}
size_t cell_sort_scratch_bytes(long long nKeys) {
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const int*)nullptr, (int*)nullptr, (int)(nKeys + 1));
  return bytes;
}
// P2G in cell order. binned: the mark pass of this substep counted the
// particles (k_mark_fluid with the cell sort) and the brick list is current;
// otherwise the particles are counted here and every brick is visited.
// Returns the number of kernel launches made (-1 on a launch error).
int launch_p2g_sorted(const Dims& d, const GridDev& g, const PartsDev& P, const CellSort& cs, const BrickSet& B,
                      bool binned, void* scratch, size_t scratchBytes, DevStatus* st, cudaStream_t s) {
  if (P.nP <= 0) return 0;
  const long long nKeys = 64LL * B.nbx * B.nby * B.nbz;
  int launches = 0;
  if (!binned) {
    if (cudaMemsetAsync(cs.count, 0, sizeof(int) * (size_t)(nKeys + 1), s) != cudaSuccess) return -1;
    k_bin_cells<<<grid_for(P.nP, 256), 256, 0, s>>>(d, g, P, cs, &st->err);
    launches++;
  }
  // prefix sum over the keys (CUB's device scan, a CUDA toolkit library)
  if (cub::DeviceScan::ExclusiveSum(scratch, scratchBytes, cs.count, cs.start, (int)(nKeys + 1), s) != cudaSuccess)
    return -1;
  launches += 2;
  k_cell_scatter<<<grid_for(P.nP, 256), 256, 0, s>>>(P.nP, cs, &st->err);
  // A block takes a brick at a time; up to 16 rounds of them are evened out, as a
  // ragged last round shows there (64^3 with 193k particles 97.5 -> 94.5 us, 97^3 with
  // 0.7M 198 -> 190), beyond them all blocks run (128^3: 401, evened 433). The face
  // passes' grid of four bricks a block took 64 us for 32^3 with 10k particles, this 42.
  const int nB = B.nbx * B.nby * B.nbz, most = 148 * 8, rounds = (nB + most - 1) / most;
  k_p2g_bricks<<<rounds <= 16 ? (nB + rounds - 1) / rounds : most, 256, 0, s>>>(d, g, P, cs, B, binned ? 0 : 1, &st->err);
  return launches + 2;
}

// ------------------------------------------------------------ 6. pressure setup
// _pressureSolve passes 1-2, js/solver.js:1321-1366: q = 0 off the fluid,
// diag = Nf + Na, rhs = -dx^2 div, relaxation weight pw = omega/diag
// (float32, as the reference's pW). pw < 0 marks a non-fluid cell. The pass
// (k_pressure_setup, below the brick list) also leaves each 4^3 brick's mask
// of interior fluid cells, from which the solve builds its plan.
// one cell of the setup: returns whether it is fluid and its SOR colour (-1 off the lists)
__device__ __forceinline__ bool cell_pressure_setup(const Dims& d, const GridDev& g, uint8_t* __restrict__ diag8,
                                                    double omega, unsigned c, int i, int j, int k, int& col) {
  col = -1;
  // every load in one round trip: most cells of a listed brick are not fluid,
  // but their loads share lines with those that are
  const unsigned nx = (unsigned)d.nx, nxy = nx * (unsigned)d.ny;
  const bool in[6] = { i > 0, i < d.nx - 1, j > 0, j < d.ny - 1, k > 0, k < d.nz - 1 };
  const unsigned o[6] = { c - 1u, c + 1u, c - nx, c + nx, c - nxy, c + nxy };
  const int tc = g.type[c];
  int tn[6];
#pragma unroll
  for (int q = 0; q < 6; q++) tn[q] = in[q] ? g.type[o[q]] : WS_SOLID;
  unsigned f[3];
  cell_faces(d, i, j, k, f);
  const float u0 = g.vel[f[0]], u1 = g.vel[f[0] + 1u], v0 = g.vel[f[1]], v1 = g.vel[f[1] + nx];
  const float w0 = g.vel[f[2]], w1 = g.vel[f[2] + nxy];
  if (tc != WS_FLUID) { g.q[c] = 0.f; g.pw[c] = -1.f; diag8[c] = 0; return false; }
  int cnt = 0;
#pragma unroll
  for (int q = 0; q < 6; q++) cnt += tn[q] != WS_SOLID;
  const double div = over_dx(d, (double)u1 - (double)u0 + (double)v1 - (double)v0 + (double)w1 - (double)w0);
  g.rhs[c] = (float)(-d.dx * d.dx * div);
  g.pw[c] = (float)(cnt > 0 ? omega / (double)cnt : 0.0);
  diag8[c] = (uint8_t)cnt;
  // membership of the SOR colour lists: interior fluid cells (sor_colour)
  if (in[0] && in[1] && in[2] && in[3] && in[4] && in[5]) col = (i + j + k) & 1;
  return true;
}
// ------------------------------------------------------------ 7. red-black SOR
// One colour of the SOR sweep, js/solver.js:1397-1404 in red-black order:
// q <- q (1 - omega) + pw (rhs + sum of the six neighbour q), FP64 arithmetic
// rounded to float32 as the reference's Float32Array store. q is zero on
// every non-fluid cell, so summing all six neighbours in the reference's
// order (-x, +x, -y, +y, -z, +z) equals its sum over fluid neighbours.
// The thread layout packs the cells of one colour: thread t -> row r, slot s,
// i = 2 s + ((j + k + colour) & 1). Bytes per full iteration: 13 per cell.
__global__ void k_sor_color(Dims d, float* __restrict__ q, const float* __restrict__ rhs,
                            const float* __restrict__ pw, int color, double om1) {
  int nx = d.nx, ny = d.ny, nz = d.nz;
  int half = (nx + 1) >> 1;
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long rows = (long long)ny * nz;
  if (t >= rows * half) return;
  int sl = (int)(t % half); long long r = t / half;
  int j = (int)(r % ny), k = (int)(r / ny);
  int i = 2 * sl + ((j + k + color) & 1);
  if (i >= nx) return;
  long long c = r * nx + i;
  float w = pw[c];
  if (w < 0.f) return;
  if (i < 1 || i > nx - 2 || j < 1 || j > ny - 2 || k < 1 || k > nz - 2) return;
  long long nxy = (long long)nx * ny;
  q[c] = sor_update(q[c], w, rhs[c], q[c - 1], q[c + 1], q[c - nx], q[c + nx], q[c - nxy], q[c + nxy], om1);
}
void launch_sor_color(const Dims& d, const GridDev& g, int color, double om1, cudaStream_t s) {
  long long n = (long long)d.ny * d.nz * ((d.nx + 1) >> 1);
  k_sor_color<<<grid_for(n, 256), 256, 0, s>>>(d, g.q, g.rhs, g.pw, color, om1);
}

// ------------------------------------------------------------ 8. FP64 residual
// ||b - A q||_2 / ||b||_2 over fluid cells with A, b the reference assembly
// (js/solver.js:1361-1365): r = rhs + sum_fluid q_n - diag q. Block partials
// in FP64, combined in a fixed order by k_residual_final (deterministic).
__global__ void k_residual_partial(Dims d, const float* __restrict__ q, const float* __restrict__ rhs,
                                   const float* __restrict__ pw, const uint8_t* __restrict__ diag8,
                                   double2* __restrict__ partials) {
  __shared__ double srr[32], sbb[32];
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double rr = 0, bb = 0;
  bool interior = false;
  if (c < d.nCells) {
    int i, j, k; decode_cell(d, c, i, j, k);
    interior = i > 0 && i < d.nx - 1 && j > 0 && j < d.ny - 1 && k > 0 && k < d.nz - 1;
  }
  if (interior && pw[c] >= 0.f) {
    int nx = d.nx; long long nxy = (long long)nx * d.ny;
    double sum = (double)q[c - 1];
    sum += (double)q[c + 1]; sum += (double)q[c - nx]; sum += (double)q[c + nx];
    sum += (double)q[c - nxy]; sum += (double)q[c + nxy];
    double b = rhs[c];
    double r = b + sum - (double)diag8[c] * (double)q[c];
    rr = r * r; bb = b * b;
  }
  rr = warp_sum(rr); bb = warp_sum(bb);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { srr[wid] = rr; sbb[wid] = bb; }
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    rr = lane < nw ? srr[lane] : 0; bb = lane < nw ? sbb[lane] : 0;
    rr = warp_sum(rr); bb = warp_sum(bb);
    if (lane == 0) partials[blockIdx.x] = make_double2(rr, bb);
  }
}
__global__ void k_residual_final(const double2* __restrict__ partials, int n, DevStatus* st, double* hostMirror) {
  __shared__ double srr[32], sbb[32];
  double rr = 0, bb = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) { rr += partials[i].x; bb += partials[i].y; }
  rr = warp_sum(rr); bb = warp_sum(bb);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { srr[wid] = rr; sbb[wid] = bb; }
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    rr = lane < nw ? srr[lane] : 0; bb = lane < nw ? sbb[lane] : 0;
    rr = warp_sum(rr); bb = warp_sum(bb);
    if (lane == 0) {
      double rel = bb > 0 ? sqrt(rr) / sqrt(bb) : sqrt(rr);
      st->rr = rr; st->bb = bb; st->relres = rel;
      if (hostMirror) *hostMirror = rel;
    }
  }
}
int residual_blocks(const Dims& d) { return (int)grid_for(d.nCells, 256); }
void launch_residual(const Dims& d, const GridDev& g, const uint8_t* diag8, double2* partials,
                     DevStatus* st, double* hostMirror, cudaStream_t s) {
  int nb = residual_blocks(d);
  k_residual_partial<<<nb, 256, 0, s>>>(d, g.q, g.rhs, g.pw, diag8, partials);
  k_residual_final<<<1, 1024, 0, s>>>(partials, nb, st, hostMirror);
}

// ------------------------------------------------------------ 9. clamp and max |u|
// _clampUmSlice (:2629-2653) with the max |u| reduction (exact: max of
// non-negative float bit patterns); in the projection pass when vorticity is off.
// block-level max, then one atomic per block (every thread of the block must call)
__device__ __forceinline__ void umax_reduce(float a, DevStatus* st) {
  __shared__ unsigned sm[32];
  unsigned bits = __float_as_uint(fabsf(a));
  bits = warp_max_u(bits);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sm[wid] = bits;
  __syncthreads();
  if (wid == 0) {
    bits = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0u;
    bits = warp_max_u(bits);
    if (lane == 0 && bits) atomicMax(&st->umaxBits, bits);
  }
}
__global__ void k_clamp_umax(Dims d, float* __restrict__ vel, float vcap, DevStatus* st) {
  long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  float u = 0.f;
  if (f < d.F) {
    u = vel[f];
    if (u > vcap) { u = vcap; vel[f] = u; } else if (u < -vcap) { u = -vcap; vel[f] = u; }
  }
  umax_reduce(u, st);
}
void launch_clamp_umax(const Dims& d, const GridDev& g, double maxSpeed, DevStatus* st, cudaStream_t s) {
  k_clamp_umax<<<grid_for(d.F, 256), 256, 0, s>>>(d, g.vel, (float)(maxSpeed * 1.1), st);
}

// ------------------------------------------------------------ 10. vorticity
// _vorticityConfinement, js/solver.js:1454-1559. (a) omega per cell from the
// float32 cell-centred velocities (recomputed from the faces, rounded as the
// reference stores them), (b) the gated confinement force per fluid cell,
// (c) the splat onto faces between two fluid cells.
// cell-centred velocities of cell (i, j, k), as the reference's _vcx/_vcy/_vcz
// (float stores of the two-face means)
__device__ __forceinline__ float ccx(const Dims& d, const float* u, int i, int j, int k) {
  const long long ui = ((long long)k * d.ny + j) * (d.nx + 1) + i;
  return (float)(0.5 * ((double)u[ui] + (double)u[ui + 1]));
}
__device__ __forceinline__ float ccy(const Dims& d, const float* v, int i, int j, int k) {
  const long long vi = ((long long)k * (d.ny + 1) + j) * d.nx + i;
  return (float)(0.5 * ((double)v[vi] + (double)v[vi + d.nx]));
}
__device__ __forceinline__ float ccz(const Dims& d, const float* w, int i, int j, int k) {
  const long long c = ((long long)k * d.ny + j) * d.nx + i, nxy = (long long)d.nx * d.ny;
  return (float)(0.5 * ((double)w[c] + (double)w[c + nxy]));
}
// Omega is read only at fluid cells: k_vort_force reads omg and om* at a fluid
// cell, and omg at its six neighbours only when all six are fluid.
__global__ void k_vort_omega(Dims d, GridDev g) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells || g.type[c] != WS_FLUID) return;
  int nx = d.nx, ny = d.ny, nz = d.nz;
  int i, j, k; decode_cell(d, c, i, j, k);
  const float* u = g.vel; const float* v = g.vel + d.uN; const float* w = g.vel + d.uN + d.vN;
  // the clamped neighbours of the reference's central differences (a boundary cell uses itself)
  const int im = i > 0 ? i - 1 : i, ip = i < nx - 1 ? i + 1 : i;
  const int jm = j > 0 ? j - 1 : j, jp = j < ny - 1 ? j + 1 : j;
  const int km = k > 0 ? k - 1 : k, kp = k < nz - 1 ? k + 1 : k;
  double inv2 = 0.5 / d.dx;
  double wx = ((double)ccz(d, w, i, jp, k) - (double)ccz(d, w, i, jm, k) -
               ((double)ccy(d, v, i, j, kp) - (double)ccy(d, v, i, j, km))) * inv2;
  double wy = ((double)ccx(d, u, i, j, kp) - (double)ccx(d, u, i, j, km) -
               ((double)ccz(d, w, ip, j, k) - (double)ccz(d, w, im, j, k))) * inv2;
  double wz = ((double)ccy(d, v, ip, j, k) - (double)ccy(d, v, im, j, k) -
               ((double)ccx(d, u, i, jp, k) - (double)ccx(d, u, i, jm, k))) * inv2;
  g.omx[c] = (float)wx; g.omy[c] = (float)wy; g.omz[c] = (float)wz;
  g.omg[c] = (float)sqrt(wx * wx + wy * wy + wz * wz);
}
__global__ void k_vort_force(Dims d, GridDev g, double eps, double dt) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells) return;
  const uint8_t* type = g.type;
  if (type[c] != WS_FLUID) return;
  int nx = d.nx, ny = d.ny, nz = d.nz; long long nxy = (long long)nx * ny;
  int i, j, k; decode_cell(d, c, i, j, k);
  const float* omg = g.omg;
  if (omg[c] < 0.35f ||
      (i > 0 && type[c - 1] != WS_FLUID) || (i < nx - 1 && type[c + 1] != WS_FLUID) ||
      (j > 0 && type[c - nx] != WS_FLUID) || (j < ny - 1 && type[c + nx] != WS_FLUID) ||
      (k > 0 && type[c - nxy] != WS_FLUID) || (k < nz - 1 && type[c + nxy] != WS_FLUID)) {
    g.vfx[c] = 0.f; g.vfy[c] = 0.f; g.vfz[c] = 0.f; return;
  }
  double gx = (double)omg[i < nx - 1 ? c + 1 : c] - (double)omg[i > 0 ? c - 1 : c];
  double gy = (double)omg[j < ny - 1 ? c + nx : c] - (double)omg[j > 0 ? c - nx : c];
  double gz = (double)omg[k < nz - 1 ? c + nxy : c] - (double)omg[k > 0 ? c - nxy : c];
  double g2 = gx * gx + gy * gy + gz * gz;
  if (g2 < 1e-12) { g.vfx[c] = 0.f; g.vfy[c] = 0.f; g.vfz[c] = 0.f; return; }
  double inv = 1 / sqrt(g2);
  double Nx = gx * inv, Ny = gy * inv, Nz = gz * inv;
  double ox = g.omx[c], oy = g.omy[c], oz = g.omz[c];
  double fx = eps * (Ny * oz - Nz * oy), fy = eps * (Nz * ox - Nx * oz), fz = eps * (Nx * oy - Ny * ox);
  double f2 = fx * fx + fy * fy + fz * fz, fCap = 6.0;
  if (f2 > fCap * fCap) { double fs = fCap / sqrt(f2); fx *= fs; fy *= fs; fz *= fs; }
  g.vfx[c] = (float)(fx * dt); g.vfy[c] = (float)(fy * dt); g.vfz[c] = (float)(fz * dt);
}
__global__ void k_vort_splat(Dims d, GridDev g) {
  long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (f >= d.F) return;
  FaceIJK F = decode_face(d, f);
  long long cL = 0, cR = 0;
  if (face_cells(d, F, cL, cR)) return;
  if (g.type[cL] != WS_FLUID || g.type[cR] != WS_FLUID) return;
  const float* fv = F.comp == 0 ? g.vfx : (F.comp == 1 ? g.vfy : g.vfz);
  g.vel[f] = (float)((double)g.vel[f] + 0.5 * ((double)fv[cL] + (double)fv[cR]));
}
void launch_vorticity(const Dims& d, const GridDev& g, double eps, double dt, cudaStream_t s) {
  k_vort_omega<<<grid_for(d.nCells, 256), 256, 0, s>>>(d, g);
  k_vort_force<<<grid_for(d.nCells, 256), 256, 0, s>>>(d, g, eps, dt);
  k_vort_splat<<<grid_for(d.F, 256), 256, 0, s>>>(d, g);
}

// ------------------------------------------------------------ active bricks
// Faces and cells far from every particle and moving solid hold fixed values
// (zero velocity, the static valid flags, q = 0 and pw = -1 off the fluid), so
// a full pass over them rewrites what is already there. The substep therefore
// runs its face and cell passes over a list of 4^3 bricks: those within one
// brick of a particle's or moving solid's cell this substep (the reach of
// P2G's stencils, the extrapolation layer and G2P's midpoint sample is under
// four cells), plus those active in the previous substep, so a brick that
// empties is rewritten once to the fixed values. A forced full pass (after a
// caller wrote grid fields) processes every brick; after a write of q alone,
// which only the pressure setup turns back to the fixed value, that pass does.
__global__ void __launch_bounds__(256) k_brick_activity(BrickSet B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  const int nB = B.nbx * B.nby * B.nbz;
  int p = 0;
  if (b < nB) {
    int bx, by, bz;
    brick_coords(B, b, bx, by, bz);
    int a = 0;
    // all 27 seeds in flight at once (a clamped neighbour only repeats a seed of the block)
#pragma unroll
    for (int dz = -1; dz <= 1; dz++) {
      const int z = min(max(bz + dz, 0), B.nbz - 1);
#pragma unroll
      for (int dy = -1; dy <= 1; dy++) {
        const uint8_t* row = B.seed + (z * B.nby + min(max(by + dy, 0), B.nby - 1)) * B.nbx;
        a |= row[max(bx - 1, 0)] | row[bx] | row[min(bx + 1, B.nbx - 1)];
      }
    }
    p = a | B.act[b] | (*B.forceAll != 0);
    B.act[b] = (uint8_t)a;
  }
  // the work list: one atomic per warp (the passes over it do not depend on its order)
  const unsigned m = __ballot_sync(0xffffffffu, p != 0);
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(B.count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (p) B.list[base + __popc(m & ((1u << lane) - 1u))] = b;
}
// activity and work list; the normalising pass that follows clears the seeds
// and the projection the forced-pass flags for the next substep
void launch_brick_activity(const BrickSet& B, cudaStream_t s) {
  k_brick_activity<<<grid_for((long long)B.nbx * B.nby * B.nbz, 256), 256, 0, s>>>(B);
}

// ------------------------------------------------------------ the face passes
// 4. _p2gNormalizeFace (:1109-1120) + _applyBC (:1130-1171) + FLIP snapshot
//    (:2579) + the extrapolation valid mark (:1578-1611)
// 5. forces: _viscosity (:1259-1304, Jacobi: neighbours from the snapshot,
//    which equals the post-BC field on entry), planet gravity (:1229-1256
//    with the ramp of :2656-2662 applied by the caller in gs), BC again (:2598)
// 9. _projectSlice (:1417-1443) and, fused when vorticity is off, the clamp
//    and max |u| of _clampUmSlice (:2629-2653)
// 11. _extrapolate (:1562-1636) in Jacobi order: an invalid face takes the
//    mean of the neighbours (same component grid) that were valid before the
//    pass, summed in the reference's order -i, +i, -j, +j, -k, +k. Filled
//    faces are marked 2 so no thread reads a value written in this pass.
//
// One thread per cell of a 4^3 brick handles the cell's three lower faces
// (and the domain's upper plane where the cell is the last along the axis):
// its loads are issued together and its type is shared by the three faces.
// Bytes per face: normalise 8 + 4 + 4 + 1, forces 4 + 4 + 4 (+ neighbours from
// cache), project 4 + 4 + 4/3, extrapolate 1; types 4/3. FP64 where the
// reference's doubles round differently from floats; a quotient of two floats
// is the same either way (53 bits hold twice 24 + 2).
enum FaceOp { kNormalize, kForces, kProject, kExtrapolate };
struct FacePassArgs { double coef, dt, gs; int viscOn, doClamp; float vcap; int all; };
// Solid-adjacent interior face: the velocity of the solid cell beside it,
// the left one first (_applyBCSlice, js/solver.js:1153-1170): 0 for rock and
// the domain shell, the ball's velocity for a ball cell.
__device__ __forceinline__ float solid_face_velocity(const Dims& d, const GridDev& g, int comp, int tL, unsigned cL, unsigned cR) {
  return g.sv ? g.sv[comp * d.nCells + (tL == WS_SOLID ? cL : cR)] : 0.f;
}
template <int OP>
__device__ __forceinline__ void upper_face(const GridDev& g, unsigned f, const FacePassArgs& fa, float& umax) {
  if (OP == kNormalize) { g.vel[f] = 0.f; g.velO[f] = 0.f; g.valid[f] = 1; }
  if (OP == kForces) g.vel[f] = 0.f;
  if (OP == kProject && fa.doClamp) {
    float u = g.vel[f];
    if (u > fa.vcap) u = fa.vcap; else if (u < -fa.vcap) u = -fa.vcap;
    g.vel[f] = u; umax = fmaxf(umax, fabsf(u));
  }
}
template <int OP>
__device__ __forceinline__ void cell_pass(const Dims& d, const GridDev& g, int i, int j, int k, const FacePassArgs& fa, float& umax) {
  unsigned f[3];
  const unsigned c = cell_faces(d, i, j, k, f), nx = (unsigned)d.nx, nxy = nx * (unsigned)d.ny;
  const unsigned cl[3] = { c - 1u, c - nx, c - nxy };   // the cell below each face
  const bool edge[3] = { i == 0, j == 0, k == 0 };      // a domain plane
  const bool last[3] = { i == d.nx - 1, j == d.ny - 1, k == d.nz - 1 };
  // strides of each component's face grid along y and z
  const unsigned sJ[3] = { nx + 1u, nx, nx }, sK[3] = { nxy + (unsigned)d.ny, nxy + nx, nxy };
  if (OP == kExtrapolate) {
    uint8_t v[3];
#pragma unroll
    for (int a = 0; a < 3; a++) v[a] = g.valid[f[a]];
    uint8_t vv[3][6];
    float av[3][6];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (v[a]) continue;
      const unsigned o[6] = { f[a] - 1u, f[a] + 1u, f[a] - sJ[a], f[a] + sJ[a], f[a] - sK[a], f[a] + sK[a] };
      const bool in[6] = { !edge[0], a == 0 || !last[0], !edge[1], a == 1 || !last[1], !edge[2], a == 2 || !last[2] };
#pragma unroll
      for (int q = 0; q < 6; q++) { vv[a][q] = in[q] ? g.valid[o[q]] : (uint8_t)0; av[a][q] = in[q] ? g.vel[o[q]] : 0.f; }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (v[a]) continue;
      double sum = 0; int cnt = 0;
#pragma unroll
      for (int q = 0; q < 6; q++) if (vv[a][q] == 1) { sum += av[a][q]; cnt++; }
      if (cnt > 0) { g.vel[f[a]] = (float)(sum / cnt); g.valid[f[a]] = 2; }
    }
    // the domain's upper plane: always valid after the normalising pass, not after a caller's own fields
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (!last[a]) continue;
      const unsigned fu = f[a] + (a == 0 ? 1u : a == 1 ? nx : nxy);
      if (g.valid[fu]) continue;
      const unsigned o[6] = { fu - 1u, fu + 1u, fu - sJ[a], fu + sJ[a], fu - sK[a], fu + sK[a] };
      double sum = 0; int cnt = 0;
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const bool in = q >> 1 == a ? !(q & 1) : q & 1 ? !last[q >> 1] : !edge[q >> 1];
        if (in && g.valid[o[q]] == 1) { sum += g.vel[o[q]]; cnt++; }
      }
      if (cnt > 0) { g.vel[fu] = (float)(sum / cnt); g.valid[fu] = 2; }
    }
    return;
  }
  int t[3];
  const int tc = g.type[c];
#pragma unroll
  for (int a = 0; a < 3; a++) t[a] = edge[a] ? WS_SOLID : g.type[cl[a]];
  if (OP == kNormalize) {
    float2 A[3];
#pragma unroll
    for (int a = 0; a < 3; a++) A[a] = g.acc[f[a]];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const bool some = (double)A[a].y > 1e-8, solid = t[a] == WS_SOLID || tc == WS_SOLID;
      float u = some ? A[a].x / A[a].y : A[a].x;
      if (edge[a]) u = 0.f;
      else if (solid) u = solid_face_velocity(d, g, a, t[a], cl[a], c);
      g.vel[f[a]] = u; g.velO[f[a]] = u; g.valid[f[a]] = some || solid ? 1 : 0;
    }
  }
  if (OP == kForces) {
    const float* __restrict__ o = g.velO;
    float u[3], gv[3], nb[3][6];
    bool visc[3], grav[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const bool open = t[a] != WS_SOLID && tc != WS_SOLID;
      visc[a] = fa.viscOn && t[a] == WS_FLUID && tc == WS_FLUID;
      grav[a] = fa.gs > 0 && open && (t[a] == WS_FLUID || tc == WS_FLUID);
      u[a] = open ? o[f[a]] : 0.f;
      gv[a] = grav[a] ? g.gvel[f[a]] : 0.f;
      if (visc[a]) {
        const unsigned p[6] = { f[a] - 1u, f[a] + 1u, f[a] - sJ[a], f[a] + sJ[a], f[a] - sK[a], f[a] + sK[a] };
        const bool in[6] = { !edge[0], a == 0 || !last[0], !edge[1], a == 1 || !last[1], !edge[2], a == 2 || !last[2] };
#pragma unroll
        for (int q = 0; q < 6; q++) nb[a][q] = o[in[q] ? p[q] : f[a]];   // off the grid: the face's own value
      }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      float r = u[a];
      if (visc[a]) {
        const double c0 = u[a];
        double val = c0 * 6;
#pragma unroll
        for (int q = 0; q < 6; q++) val -= (double)nb[a][q];
        r = (float)(c0 + fa.coef * val);
      }
      if (grav[a]) r = (float)((double)r + (double)gv[a] * fa.dt * fa.gs);
      if (!edge[a] && (t[a] == WS_SOLID || tc == WS_SOLID)) r = solid_face_velocity(d, g, a, t[a], cl[a], c);
      g.vel[f[a]] = r;
    }
  }
  if (OP == kProject) {
    float u[3], ql[3];
    const float qc = g.q[c];
#pragma unroll
    for (int a = 0; a < 3; a++) { u[a] = g.vel[f[a]]; ql[a] = edge[a] ? 0.f : g.q[cl[a]]; }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const bool open = t[a] != WS_SOLID && tc != WS_SOLID;
      if (open) {
        const double pL = t[a] == WS_FLUID ? (double)ql[a] : 0.0, pR = tc == WS_FLUID ? (double)qc : 0.0;
        u[a] = (float)((double)u[a] - (pR - pL) * d.rdx);
      }
      if (fa.doClamp) {
        if (u[a] > fa.vcap) u[a] = fa.vcap; else if (u[a] < -fa.vcap) u[a] = -fa.vcap;
        umax = fmaxf(umax, fabsf(u[a]));
      }
      g.vel[f[a]] = u[a];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++)
    if (last[a]) upper_face<OP>(g, f[a] + (a == 0 ? 1u : a == 1 ? nx : nxy), fa, umax);
}
// One pass over the work list (all: over every brick), four bricks per block
// and iteration. Bound by load latency (L1 and L2 at a third of their rates).
// Normalise / forces / project / extrapolate, one thread per face of a brick
// before: 24.4 / 29.7 / 22.2 / 28.6 us at 128^3, now 13.3 / 15.5 / 10.4 / 15.6;
// 110 / 140 / 96 / 90 -> 87 / 73 / 50 / 64 at 256^3; with half a brick
// per warp instead of two rows of four, normalise and project took 19.3 and
// 14.0 us at 128^3, 129 and 61 at 256^3. Clearing in the raster pass instead of
// its own 10.1 -> 3.9 us at 128^3.
template <int OP>
__global__ void __launch_bounds__(256) k_faces(Dims d, GridDev g, BrickSet B, FacePassArgs fa, DevStatus* st) {
  const int nB = B.nbx * B.nby * B.nbz;
  if (OP == kNormalize && !fa.all) {                    // the substep's seeds have been read
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int t = t0; t < nB >> 4; t += gridDim.x * blockDim.x) reinterpret_cast<uint4*>(B.seed)[t] = make_uint4(0, 0, 0, 0);
    if (t0 < (nB & 15)) B.seed[(nB & ~15) + t0] = 0;
    if (t0 == 0) B.count[1] = *B.count;
  }
  if (OP == kProject && !fa.all && blockIdx.x == 0 && threadIdx.x == 0) { B.forceAll[0] = 0; B.forceAll[1] = 0; }
  const int n = fa.all ? nB : *B.count, step = gridDim.x * 4;
  int q, li, lj, lk;
  quad_cell(q, li, lj, lk);
  float umax = 0.f;
  int it = blockIdx.x * 4 + q;
  int b = fa.all ? it : it < n ? B.list[it] : 0;
  for (; it < n; it += step) {
    // the next brick's id is loaded before this brick's faces are touched
    const int bNext = fa.all ? it + step : it + step < n ? B.list[it + step] : 0;
    int bx, by, bz;
    brick_coords(B, b, bx, by, bz);
    const int i = bx * 4 + li, j = by * 4 + lj, k = bz * 4 + lk;
    if (i < d.nx && j < d.ny && k < d.nz) cell_pass<OP>(d, g, i, j, k, fa, umax);
    b = bNext;
  }
  if (OP == kProject && fa.doClamp) umax_reduce(umax, st);
}
static unsigned brick_grid(const BrickSet& B) {
  const int nB = B.nbx * B.nby * B.nbz;
  return (unsigned)std::min((nB + 3) / 4, 148 * 8);
}
void launch_faces_normalize_bc(const Dims& d, const GridDev& g, const BrickSet& B, bool all, cudaStream_t s) {
  FacePassArgs fa{}; fa.all = all;
  k_faces<kNormalize><<<brick_grid(B), 256, 0, s>>>(d, g, B, fa, nullptr);
}
void launch_faces_forces(const Dims& d, const GridDev& g, const BrickSet& B, bool all, double coef, int viscOn, double dt,
                         double gs, cudaStream_t s) {
  FacePassArgs fa{}; fa.coef = coef; fa.viscOn = viscOn; fa.dt = dt; fa.gs = gs; fa.all = all;
  k_faces<kForces><<<brick_grid(B), 256, 0, s>>>(d, g, B, fa, nullptr);
}
void launch_project(const Dims& d, const GridDev& g, const BrickSet& B, bool all, int doClamp, double maxSpeed,
                    DevStatus* st, cudaStream_t s) {
  FacePassArgs fa{}; fa.doClamp = doClamp; fa.vcap = (float)(maxSpeed * 1.1); fa.all = all;
  k_faces<kProject><<<brick_grid(B), 256, 0, s>>>(d, g, B, fa, st);
}
void launch_extrapolate(const Dims& d, const GridDev& g, const BrickSet& B, bool all, cudaStream_t s) {
  FacePassArgs fa{}; fa.all = all;
  k_faces<kExtrapolate><<<brick_grid(B), 256, 0, s>>>(d, g, B, fa, nullptr);
}
// the pressure setup over the brick list (or every brick), four bricks per block
__global__ void __launch_bounds__(256) k_pressure_setup(Dims d, GridDev g, uint8_t* __restrict__ diag8, double omega,
                                                        DevStatus* st, BrickSet B, int allBricks) {
  const bool every = allBricks || B.forceAll[1];        // every brick after a caller wrote q (q = 0 off the fluid)
  const int n = every ? B.nbx * B.nby * B.nbz : *B.count;
  uint8_t* mask = reinterpret_cast<uint8_t*>(g.fmask);
  int fluid = 0, odd = 0, q, li, lj, lk;
  quad_cell(q, li, lj, lk);
  for (int it = blockIdx.x * 4; it < n; it += gridDim.x * 4) {
    const int e = it + q, b = e >= n ? -1 : every ? e : B.list[e];
    int col = -1;
    if (b >= 0) {
      int bx, by, bz;
      brick_coords(B, b, bx, by, bz);
      const int i = bx * 4 + li, j = by * 4 + lj, k = bz * 4 + lk;
      if (i < d.nx && j < d.ny && k < d.nz &&
          cell_pressure_setup(d, g, diag8, omega, ((unsigned)k * (unsigned)d.ny + (unsigned)j) * (unsigned)d.nx + (unsigned)i, i, j, k, col)) {
        fluid++;
        odd |= col < 0;
      }
    }
    // bit 16 z + 4 y + x: the warp's two rows of a brick are one byte of its mask
    const unsigned m = __ballot_sync(0xffffffffu, col >= 0) >> (4 * q);
    if ((threadIdx.x & 19) == 0 && b >= 0) mask[8 * b + (threadIdx.x >> 5)] = (uint8_t)((m & 15u) | (m >> 12 & 0xf0u));
  }
  // one atomic per block: thousands of warps on one address take microseconds
  fluid = warp_sum(fluid);
  __shared__ int sFluid[8];
  if ((threadIdx.x & 31) == 0) sFluid[threadIdx.x >> 5] = fluid;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) fluid += sFluid[w];
    if (fluid) atomicAdd(&st->nFluid, fluid);
  }
  if (odd) atomicOr(&st->oddFluid, 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) st->sorOmega = omega;
}
void launch_pressure_setup(const Dims& d, const GridDev& g, uint8_t* diag8, double omega, DevStatus* st,
                           const BrickSet& B, bool allBricks, cudaStream_t s) {
  // a stage on its own may follow cell types of a caller's, without a raster pass between
  if (allBricks) cudaMemsetAsync(&st->oddFluid, 0, sizeof(int), s);
  k_pressure_setup<<<brick_grid(B), 256, 0, s>>>(d, g, diag8, omega, st, B, allBricks ? 1 : 0);
}

// ------------------------------------------------------------ field helpers
__global__ void k_extract_weight(Dims d, const float2* __restrict__ acc, float* __restrict__ out, long long off, long long n) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < n) out[t] = acc[off + t].y;
}
void launch_extract_weight(const Dims& d, const float2* acc, float* out, long long off, long long n, cudaStream_t s) {
  k_extract_weight<<<grid_for(n, 256), 256, 0, s>>>(d, acc, out, off, n);
}
