// ws_frame.cu — per-frame passes: thermal tick (js/solver.js:2715-2994),
// evaporation (:3008-3125), phase changes (:3145-3281), frame-end rescue
// (:3496-3587), density splat (:3785-3820) and the FP64 reductions
// (marching-tets volume js/surface.js:66-177, census js/main.js:176-186,
// kinetic energy js/solver.js:3914-3921).
#include "ws_kernels.cuh"
#include <algorithm>

// ------------------------------------------------------------ thermal: shadows + heating
// _heatShadowChunk, js/solver.js:2773-2918 — independent per particle.
__global__ void k_heat_shadow(Dims d, GridDev g, PartsDev P, TerrainDev t, HeatParams hp, double dt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  const double dx = d.dx, cx = d.cx, cy = d.cy, cz = d.cz;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const uint8_t* type = g.type;
  double lit = hp.hasSun ? 1 : 0;
  double PX = P.px[p], PY = P.py[p], PZ = P.pz[p];
  double dwx = PX - cx, dwy = PY - cy, dwz = PZ - cz;
  double dwl = sqrt(dwx * dwx + dwy * dwy + dwz * dwz); if (dwl == 0) dwl = 1e-9;
  double stpU = dx / dwl; int above = 0;
  for (int stU = 1; stU <= 4; stU++) {
    double qx = PX + dwx * stpU * stU, qy = PY + dwy * stpU * stU, qz = PZ + dwz * stpU * stU;
    int qi = jtrunc(over_dx(d, qx)), qj = jtrunc(over_dx(d, qy)), qk = jtrunc(over_dx(d, qz));
    if (qi < 0 || qj < 0 || qk < 0 || qi >= nx || qj >= ny || qk >= nz) break;
    if (type[((long long)qk * ny + qj) * nx + qi] != WS_FLUID) break;
    above++;
  }
  P.pDepth[p] = (uint8_t)above;
  if (hp.hasSun) {
    if (above >= 4) lit = 0;
    else {
      double lx = hp.sun[0] - PX, ly = hp.sun[1] - PY, lz = hp.sun[2] - PZ;
      double ld = sqrt(lx * lx + ly * ly + lz * lz); if (ld == 0) ld = 1e-9;
      double dxn = lx / ld, dyn = ly / ld, dzn = lz / ld;
      double ex = cx - PX, ey = cy - PY, ez = cz - PZ;
      double b = ex * dxn + ey * dyn + ez * dzn;
      if (t.has) {
        double d2c = ex * ex + ey * ey + ez * ez - b * b;
        if (b > 0 && d2c < t.Rlo2 * 0.96) lit = 0;
        else if (b > 0 || d2c < t.Rhi2 * 1.1) {
          double stp = dx * 1.5, mx = PX, my = PY, mz = PZ;
          double esc2 = (t.Rhi + 0.1) * (t.Rhi + 0.1);
          for (int st2 = 0; st2 < 26; st2++) {
            mx += dxn * stp; my += dyn * stp; mz += dzn * stp;
            double rex = mx - cx, rey = my - cy, rez = mz - cz;
            if (rex * rex + rey * rey + rez * rez > esc2) break;
            int ivx = jtrunc(over_dv(t, mx)); if (ivx < 0 || ivx >= t.n) break;
            int ivy = jtrunc(over_dv(t, my)); if (ivy < 0 || ivy >= t.n) break;
            int ivz = jtrunc(over_dv(t, mz)); if (ivz < 0 || ivz >= t.n) break;
            if (t.solid[((long long)ivz * t.n + ivy) * t.n + ivx]) { lit = 0; break; }
          }
        }
      } else if (b > 0) {
        double d2c2 = ex * ex + ey * ey + ez * ez - b * b;
        if (d2c2 < hp.coreR * hp.coreR) lit = 0;
      }
      if (lit != 0) {
        double od = 0, sx = PX, sy = PY, sz = PZ, half = dx;
        long long sj = nx + 1, sk = (long long)(ny + 1) * sj;
        for (int st = 0; st < 6 && st * half < 0.55; st++) {
          sx += dxn * half; sy += dyn * half; sz += dzn * half;
          int i0 = jtrunc(over_dx(d, sx)), j0 = jtrunc(over_dx(d, sy)), k0 = jtrunc(over_dx(d, sz));
          if (i0 < 0 || j0 < 0 || k0 < 0 || i0 >= nx || j0 >= ny || k0 >= nz) break;
          double vv = g.dens[k0 * sk + j0 * sj + i0];
          od += vv * half * 1.1;
          if (od > 3.5) break;
        }
        lit = od < 3.5 ? exp(-od) : 0;
      }
    }
  }
  P.pLight[p] = (float)lit;
  double T, pT = P.pT[p], Tamb = hp.Tamb, sunPow = hp.sunActivity / 3;
  int f = P.pflag[p];
  if (f == 2) {
    double amb = lit > 0.05 ? Tamb + 0.18 : 0.06, K = hp.hasSun ? 0.16 + (1 - lit) * 0.20 : 1.2;
    T = pT + (amb - pT) * K * dt; if (lit > 0) T += sunPow * 0.6 * lit * dt;
  } else if (f == 3) {
    double amb = lit > 0.05 ? Tamb + 0.18 : 0.06, K = hp.hasSun ? 0.10 + (1 - lit) * 0.12 : 0.9;
    T = pT + (amb - pT) * K * dt; if (lit > 0) T += sunPow * 0.35 * lit * dt;
  } else if (f == 4) {
    double amb = lit > 0.05 ? Tamb + 0.18 : 0.06, K = hp.hasSun ? 0.14 + (1 - lit) * 0.16 : 1.0;
    T = pT + (amb - pT) * K * dt; if (lit > 0) T += sunPow * 0.45 * lit * dt;
  } else {
    double amb = lit > 0.05 ? Tamb : 0;
    T = pT + (amb - pT) * (0.045 + (1 - lit) * hp.shadeCool) * dt; if (lit > 0) T += sunPow * lit * dt;
  }
  if (T > 1.15) T = 1.15; else if (T < 0) T = 0;
  P.pT[p] = (float)T;
}

// ------------------------------------------------------------ thermal: conduction
// Cell aggregates of _heatMeansSlice/_heatConductFlux/_heatApplySlice
// (:2921-2979) without a particle sort: counts and FP64 temperature sums per
// cell, then each cell gathers its six edge energies in the reference's
// accumulation order, then each particle applies its cell's update.
__device__ __forceinline__ long long heat_cell(const Dims& d, double x, double y, double z) {
  int gx = jtrunc(over_dx(d, x)); if (gx < 0) gx = 0; else if (gx >= d.nx) gx = d.nx - 1;
  int gy = jtrunc(over_dx(d, y)); if (gy < 0) gy = 0; else if (gy >= d.ny) gy = d.ny - 1;
  int gz = jtrunc(over_dx(d, z)); if (gz < 0) gz = 0; else if (gz >= d.nz) gz = d.nz - 1;
  return ((long long)gz * d.ny + gy) * d.nx + gx;
}
__global__ void k_heat_bin(Dims d, PartsDev P, int* __restrict__ cnt, double* __restrict__ sumT) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  long long c = heat_cell(d, P.px[p], P.py[p], P.pz[p]);
  atomicAdd(&cnt[c], 1);
  atomicAdd(&sumT[c], (double)P.pT[p]);
}
__global__ void k_heat_means(Dims d, const int* __restrict__ cnt, double* __restrict__ sumT) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells) return;
  sumT[c] = cnt[c] ? sumT[c] / cnt[c] : 0.0;        // in place: sum -> mean
}
__global__ void k_heat_flux(Dims d, const int* __restrict__ cnt, const double* __restrict__ mean,
                            double* __restrict__ change, double alpha) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= d.nCells) return;
  int nc = cnt[c];
  if (!nc) return;
  int nx = d.nx, ny = d.ny, nz = d.nz; long long nxy = (long long)nx * ny;
  int i, j, k; cell_ijk(d, c, i, j, k);
  double ch = 0;
  // contributions as the neighbour of an earlier cell (:2961 "-="): c-nxy, c-nx, c-1
  if (k > 0 && cnt[c - nxy]) { int a = cnt[c - nxy]; ch -= alpha * (double)(a < nc ? a : nc) * (mean[c] - mean[c - nxy]); }
  if (j > 0 && cnt[c - nx]) { int a = cnt[c - nx]; ch -= alpha * (double)(a < nc ? a : nc) * (mean[c] - mean[c - nx]); }
  if (i > 0 && cnt[c - 1]) { int a = cnt[c - 1]; ch -= alpha * (double)(a < nc ? a : nc) * (mean[c] - mean[c - 1]); }
  // own edges along +x, +y, +z (:2961 "+=")
  if (i < nx - 1 && cnt[c + 1]) { int a = cnt[c + 1]; ch += alpha * (double)(nc < a ? nc : a) * (mean[c + 1] - mean[c]); }
  if (j < ny - 1 && cnt[c + nx]) { int a = cnt[c + nx]; ch += alpha * (double)(nc < a ? nc : a) * (mean[c + nx] - mean[c]); }
  if (k < nz - 1 && cnt[c + nxy]) { int a = cnt[c + nxy]; ch += alpha * (double)(nc < a ? nc : a) * (mean[c + nxy] - mean[c]); }
  change[c] = ch;
}
__global__ void k_heat_apply_convect(Dims d, PartsDev P, const int* __restrict__ cnt, const double* __restrict__ mean,
                                     const double* __restrict__ change, double alphaA, int conduct, double Tamb, double dt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  double x = P.px[p], y = P.py[p], z = P.pz[p];
  float T = P.pT[p];
  if (conduct) {
    long long c = heat_cell(d, x, y, z);
    double deltaT = change[c] / cnt[c];
    T = (float)((double)T + alphaA * (mean[c] - (double)T) + deltaT);
    P.pT[p] = T;
  }
  if (P.pflag[p] != 0) return;                       // _heatConvectChunk :2982-2994
  double rx = x - d.cx, ry = y - d.cy, rz = z - d.cz;
  double rl = sqrt(rx * rx + ry * ry + rz * rz); if (rl == 0) rl = 1e-9;
  double ab = 3.0 * ((double)T - Tamb) * dt / rl;
  P.pvx[p] = (float)((double)P.pvx[p] + rx * ab);
  P.pvy[p] = (float)((double)P.pvy[p] + ry * ab);
  P.pvz[p] = (float)((double)P.pvz[p] + rz * ab);
}
void launch_heat(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, const HeatParams& hp,
                 double dt, int* cnt, double* sumT, double* change, cudaStream_t s) {
  if (P.nP <= 0) return;
  unsigned gp = grid_for(P.nP, 256), gc = grid_for(d.nCells, 256);
  k_heat_shadow<<<gp, 256, 0, s>>>(d, g, P, t, hp, dt);
  int conduct = hp.heatK > 0;
  if (conduct) {
    cudaMemsetAsync(cnt, 0, sizeof(int) * d.nCells, s);
    cudaMemsetAsync(sumT, 0, sizeof(double) * d.nCells, s);
    k_heat_bin<<<gp, 256, 0, s>>>(d, P, cnt, sumT);
    k_heat_means<<<gc, 256, 0, s>>>(d, cnt, sumT);
    double alpha = hp.heatK * dt * 0.15; if (alpha > 0.14) alpha = 0.14;
    k_heat_flux<<<gc, 256, 0, s>>>(d, cnt, sumT, change, alpha);
    k_heat_apply_convect<<<gp, 256, 0, s>>>(d, P, cnt, sumT, change, alpha, 1, hp.Tamb, dt);
  } else {
    k_heat_apply_convect<<<gp, 256, 0, s>>>(d, P, cnt, sumT, change, 0, 0, hp.Tamb, dt);
  }
}

// ------------------------------------------------------------ evaporation
// _evapChunk, js/solver.js:3028-3116. Candidates (surface-top liquid above
// the freezing point) are compacted in index order and walked as the
// reference's single _evS stream. With E ejections before it, candidate t
// (counted from the walk's start state s0) draws the state T^(t+1+6E)(s0),
// T the generator, each ejection taking six draws for its Box-Muller kick;
// it ejects when that draw u has u / 2^32 <= prob, i.e. u <= floor(prob 2^32).
// The walk is cut into windows of kEvW candidates. A window maps the
// ejection count before it to the count after it, monotonically; each window
// tabulates that map for a band of inputs around the expected count (the
// prefix sum of the probabilities), one warp per input, all windows in
// parallel; one warp then chains the windows through their tables (resolving
// a window directly when the count falls outside its band), and every window
// finally replays its own resolve to record its ejectors. A kick whose
// u1 < 1e-9 retry takes more than six draws (about one in 10^9) shifts every
// later position: the pass reports the first such ejection and the host starts
// a new pass after it.
__device__ __forceinline__ bool evap_candidate(const Dims& d, const GridDev& g, const PartsDev& P, int p,
                                               double freezeT, int& ci, int& cj, int& ck) {
  if (P.pflag[p] != 0) return false;
  double T = P.pT[p];
  if (T <= freezeT) return false;
  double PX = P.px[p], PY = P.py[p], PZ = P.pz[p];
  int i = jtrunc(over_dx(d, PX)), j = jtrunc(over_dx(d, PY)), k = jtrunc(over_dx(d, PZ));
  if (i < 1) i = 1; else if (i > d.nx - 2) i = d.nx - 2;
  if (j < 1) j = 1; else if (j > d.ny - 2) j = d.ny - 2;
  if (k < 1) k = 1; else if (k > d.nz - 2) k = d.nz - 2;
  if (g.type[((long long)k * d.ny + j) * d.nx + i] != WS_FLUID) return false;
  double ex = PX - d.cx, ey = PY - d.cy, ez = PZ - d.cz;
  double el = sqrt(ex * ex + ey * ey + ez * ez); if (el == 0) el = 1e-9;
  int ui = jtrunc(over_dx(d, PX + ex / el * d.dx)), uj = jtrunc(over_dx(d, PY + ey / el * d.dx)), uk = jtrunc(over_dx(d, PZ + ez / el * d.dx));
  if (ui < 0 || uj < 0 || uk < 0 || ui >= d.nx || uj >= d.ny || uk >= d.nz) return false;
  if (g.type[((long long)uk * d.ny + uj) * d.nx + ui] == WS_FLUID) return false;
  ci = i; cj = j; ck = k;
  return true;
}
__global__ void k_evap_flags(Dims d, GridDev g, PartsDev P, double freezeT, uint8_t* __restrict__ cand) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  int i, j, k;
  cand[p] = evap_candidate(d, g, P, p, freezeT, i, j, k) ? 1 : 0;
}
__device__ __forceinline__ double ev_gauss(uint32_t& s) {
  double u1;
  do { s = lcg_next(s); u1 = s / 4294967296.0; } while (u1 < 1e-9);
  s = lcg_next(s);
  return sqrt(-2 * log(u1)) * cos(6.283185306 * (s / 4294967296.0));
}
uint32_t evap_kick_end(uint32_t s) {             // the stream after a kick drawn from decision state s
  for (int g = 0; g < 3; g++) {
    do { s = lcg_next(s); } while (s < 5u);       // u1 = s / 2^32 < 1e-9 exactly when s < 5
    s = lcg_next(s);
  }
  return s;
}
// Six steps of the _evS generator (x -> 1664525 x + 1013904223 mod 2^32) as one affine map.
constexpr uint32_t lcg_pow_a(int n) { return n == 0 ? 1u : 1664525u * lcg_pow_a(n - 1); }
constexpr uint32_t lcg_pow_c(int n) { return n == 0 ? 0u : 1664525u * lcg_pow_c(n - 1) + 1013904223u; }
constexpr uint32_t kLcg6A = lcg_pow_a(6), kLcg6C = lcg_pow_c(6);
constexpr double kEvapC = 3.5, kEvapTCap = 1.15;   // EVAP_STEEPNESS and T_CAP, js/solver.js:3040-3041
constexpr int kEvW = 4096;                       // candidates per window
constexpr int kEvKMax = 1024;                    // widest band of tabulated inputs per window
__device__ __forceinline__ void lcg_affine(uint32_t k, uint32_t& A, uint32_t& C) {   // T^k(x) = A x + C
  uint32_t a = 1664525u, c = 1013904223u;
  A = 1u; C = 0u;
  while (k) { if (k & 1u) { A = A * a; C = C * a + c; } c = c * (a + 1u); a = a * a; k >>= 1; }
}
// The candidate ejects when its draw u satisfies u <= thr (thr = -1: never;
// 2^32: always, prob >= 1 or NaN as in !(rnd > prob)).
__global__ void k_evap_thr(const PartsDev P, double freezeT, double rate, double dt, const int* __restrict__ list,
                           const int* __restrict__ nCp, long long* __restrict__ thr) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= *nCp) return;
  double prob = rate * dt * exp(kEvapC * ((double)P.pT[list[t]] - freezeT));
  long long v;
  if (!(prob < 1)) v = 4294967296ll;
  else if (prob < 0) v = -1;
  else v = (long long)floor(prob * 4294967296.0);
  thr[t] = v;
}
// One warp resolves a window of n candidates entering with Ein ejections:
// b[j] = T^(j'+1)(s0) for the window's j-th candidate (j' its index in the
// pass), so its draw after E ejections is T^(6E)(b[j]). Returns the count
// after the window; emit(j, E, u) runs on the lane of each ejector.
template <class Emit>
__device__ __forceinline__ int ev_resolve(const uint32_t* b, const long long* thr, int n, int Ein, Emit emit) {
  const int lane = threadIdx.x & 31;
  uint32_t A, C;
  lcg_affine(6u * (uint32_t)Ein, A, C);
  int E = Ein, i = 0;
  while (i < n) {
    const int idx = i + lane;
    uint32_t u = 0;
    bool hit = false;
    if (idx < n) { u = A * b[idx] + C; hit = (long long)u <= thr[idx]; }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (!bal) { i += 32; continue; }
    const int f = __ffs(bal) - 1;
    if (lane == f) emit(idx, E, u);
    E++; i += f + 1;
    C = kLcg6A * C + kLcg6C; A = kLcg6A * A;
  }
  return E;
}
__device__ __forceinline__ int ev_windows(int nC, int t0) { return nC > t0 ? (nC - t0 + kEvW - 1) / kEvW : 0; }
__global__ void __launch_bounds__(256) k_evap_wsum(const long long* __restrict__ thr, const int* __restrict__ nCp,
                                                   int t0, double* __restrict__ wsum) {
  __shared__ double red[8];
  const int nC = *nCp, w = blockIdx.x;
  if (w >= ev_windows(nC, t0)) return;
  const int lo = t0 + w * kEvW, hi = min(nC, lo + kEvW);
  double acc = 0;
  for (int t = lo + (int)threadIdx.x; t < hi; t += blockDim.x) {
    const long long v = thr[t];
    acc += v < 0 ? 0.0 : v >= 4294967296ll ? 1.0 : (double)v * (1.0 / 4294967296.0);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0;
    for (int k = 0; k < 8; k++) tot += red[k];
    wsum[w] = tot;
  }
}
// Band origins: L[w] = floor(expected ejections before window w) - K/2, K set
// from the expected total (eight standard deviations of a Poisson count, + 64).
__global__ void __launch_bounds__(1024) k_evap_band(const double* __restrict__ wsum, const int* __restrict__ nCp,
                                                    int t0, int* __restrict__ L, DevStatus* st) {
  __shared__ double red[32];
  __shared__ double sTot;
  const int nW = ev_windows(*nCp, t0);
  const int tid = (int)threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double v = 0;
  for (int w = tid; w < nW; w += 1024) v += wsum[w];
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (tid == 0) { double tot = 0; for (int k = 0; k < 32; k++) tot += red[k]; sTot = tot; }
  __syncthreads();
  int keff = ((int)(8.0 * sqrt(sTot) + 64.0) + 31) & ~31;
  keff = keff < 64 ? 64 : keff > kEvKMax ? kEvKMax : keff;
  double carry = 0;
  for (int c0 = 0; c0 < nW; c0 += 1024) {
    __syncthreads();                              // red[] and sTot of the previous chunk are consumed
    const int w = c0 + tid;
    const double x = w < nW ? wsum[w] : 0.0;
    double inc = x;
    for (int o = 1; o < 32; o <<= 1) { double y = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += y; }
    if (lane == 31) red[wid] = inc;
    __syncthreads();
    if (wid == 0) {
      double r = red[lane], ri = r;
      for (int o = 1; o < 32; o <<= 1) { double y = __shfl_up_sync(0xffffffffu, ri, o); if (lane >= o) ri += y; }
      red[lane] = ri - r;                         // exclusive warp offsets
      if (lane == 31) sTot = ri;
    }
    __syncthreads();
    const double excl = carry + red[wid] + inc - x;
    if (w < nW) { const int c = (int)floor(excl) - keff / 2; L[w] = c < 0 ? 0 : c; }
    carry += sTot;
  }
  if (tid == 0) { st->evKeff = keff; st->evIrr = ~0ull; st->evNC = *nCp; }
}
// Each window: its candidates' base states and thresholds in shared memory,
// then one warp per tabulated input. A surface of 20k candidates has five
// windows, so several blocks share a window's inputs, as many as the grid has for
// each of the windows that hold candidates (known on the device only; the
// number of windows that the particles could fill, 3700 at 256^3 with 15.3M, left
// eight warps each). The stage takes 145 us at 64^3 with 193k particles (250 with
// one block of 32 warps a window), 357 at 128^3 with 1.86M (425), 2275 at 256^3
// (2460; 3140 with eight warps).
constexpr int kEvTableThreads = 256;
__global__ void __launch_bounds__(kEvTableThreads) k_evap_table(const long long* __restrict__ thr, const int* __restrict__ nCp,
                                                                int t0, const uint32_t* __restrict__ sStart,
                                                                const int* __restrict__ L, const DevStatus* __restrict__ st,
                                                                uint32_t* __restrict__ bOut, unsigned short* __restrict__ table) {
  __shared__ uint32_t sb[kEvW];
  __shared__ long long sthr[kEvW];
  constexpr int warps = kEvTableThreads / 32;
  const int nC = *nCp, keff = st->evKeff, nW = ev_windows(nC, t0);
  if (nW == 0) return;
  const int parts = max(1, min((keff + warps - 1) / warps, (int)gridDim.x / nW));
  uint32_t A, C;
  lcg_affine(kEvTableThreads, A, C);
  for (int item = (int)blockIdx.x; item < nW * parts; item += (int)gridDim.x) {
    const int w = item / parts, part = item - w * parts;
    const int lo = t0 + w * kEvW, n = min(kEvW, nC - lo);
    uint32_t bj = lcg_jump(*sStart, (uint32_t)(lo - t0 + (int)threadIdx.x + 1));
    for (int j = (int)threadIdx.x; j < n; j += kEvTableThreads, bj = A * bj + C) {
      sb[j] = bj;
      if (part == 0) bOut[lo + j] = bj;
      sthr[j] = thr[lo + j];
    }
    __syncthreads();
    const int Lw = L[w];
    for (int k = part * warps + (int)(threadIdx.x >> 5); k < keff; k += warps * parts) {
      const int eo = ev_resolve(sb, sthr, n, Lw + k, [](int, int, uint32_t) {});
      if ((threadIdx.x & 31) == 0) table[(size_t)w * kEvKMax + k] = (unsigned short)(eo - (Lw + k));
    }
    __syncthreads();                              // the window's states and thresholds are read
  }
}
// One warp: the ejection count entering every window.
__global__ void __launch_bounds__(32) k_evap_chain(const int* __restrict__ nCp, int t0, const int* __restrict__ L,
                                                   const unsigned short* __restrict__ table,
                                                   const uint32_t* __restrict__ b, const long long* __restrict__ thr,
                                                   const uint32_t* __restrict__ sStart, int* __restrict__ Ew,
                                                   DevStatus* st) {
  const int nC = *nCp, nW = ev_windows(nC, t0), keff = st->evKeff;
  int E = 0;
  int Lnext = nW > 0 ? L[0] : 0;
  for (int w = 0; w < nW; w++) {
    const int Lw = Lnext;
    if (w + 1 < nW) Lnext = L[w + 1];
    if (threadIdx.x == 0) Ew[w] = E;
    const int rel = E - Lw;
    if (rel >= 0 && rel < keff) {
      E += table[(size_t)w * kEvKMax + rel];
    } else {
      const int lo = t0 + w * kEvW;
      E = ev_resolve(b + lo, thr + lo, min(kEvW, nC - lo), E, [](int, int, uint32_t) {});
    }
  }
  if (threadIdx.x == 0) {
    st->evNEj = E;
    st->evSEnd = lcg_jump(*sStart, (uint32_t)(nC > t0 ? nC - t0 : 0) + 6u * (uint32_t)E);
  }
}
// One block per window: its candidates into shared memory, then one warp
// replays its resolve and records each ejector (particle and decision state).
// Bound by that warp's chain of 128 and more steps (20 us; from global memory 35).
__global__ void __launch_bounds__(256) k_evap_emit(const int* __restrict__ nCp, int t0, const uint32_t* __restrict__ b,
                            const long long* __restrict__ thr, const int* __restrict__ Ew, const int* __restrict__ list,
                            int eoff, int* __restrict__ ejP, uint32_t* __restrict__ ejS, DevStatus* st) {
  __shared__ uint32_t sb[kEvW];
  __shared__ long long sthr[kEvW];
  const int nC = *nCp, w = (int)blockIdx.x;
  if (w >= ev_windows(nC, t0)) return;
  const int lo = t0 + w * kEvW, n = min(kEvW, nC - lo);
  for (int j = (int)threadIdx.x; j < n; j += 256) { sb[j] = b[lo + j]; sthr[j] = thr[lo + j]; }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  ev_resolve(sb, sthr, n, Ew[w], [&](int j, int E, uint32_t u) {
    ejP[eoff + E] = list[lo + j];
    ejS[eoff + E] = u;
    // Regular kick: its three u1 draws (1, 3 and 5 after the decision) have states >= 5.
    const uint32_t s1 = lcg_next(u), s3 = lcg_next(lcg_next(s1)), s5 = lcg_next(lcg_next(s3));
    if (s1 < 5u || s3 < 5u || s5 < 5u)
      atomicMin(&st->evIrr, ((unsigned long long)(unsigned)E << 32) | (unsigned)(lo - t0 + j));
  });
}
// :3083-3113 for one ejection, its kick drawn from the recorded stream state.
__global__ void k_evap_apply(Dims d, GridDev g, PartsDev P, double freezeT, const int* __restrict__ ejP,
                             const uint32_t* __restrict__ ejS, int nEj) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nEj) return;
  const int p = ejP[e];
  int i, j, k;
  evap_candidate(d, g, P, p, freezeT, i, j, k);
  const double T = P.pT[p];
  double tau = (T - freezeT) / (kEvapTCap - freezeT);
  if (tau < 0) tau = 0; else if (tau > 1) tau = 1;
  const double sig = 0.30 + 0.32 * sqrt(tau);
  uint32_t sl = ejS[e];
  double kx = sig * ev_gauss(sl); double ky = sig * ev_gauss(sl); double kz = sig * ev_gauss(sl);
  P.pflag[p] = 2; P.pAir[p] = 0.f;
  double PX = P.px[p], PY = P.py[p], PZ = P.pz[p];
  double ex2 = PX - d.cx, ey2 = PY - d.cy, ez2 = PZ - d.cz;
  double el2 = ex2 * ex2 + ey2 * ey2 + ez2 * ez2;
  double elL = sqrt(el2); if (elL == 0) elL = 1e-9;
  double kUp = (kx * ex2 + ky * ey2 + kz * ez2) / el2;
  if (kUp < 0) { kx -= 2 * kUp * ex2 / elL; ky -= 2 * kUp * ey2 / elL; kz -= 2 * kUp * ez2 / elL; }
  int nx = d.nx, ny = d.ny;
  double guS = g.vel[((long long)k * ny + j) * (nx + 1) + i];
  double gvS = g.vel[d.uN + ((long long)k * (ny + 1) + j) * nx + i];
  double gwS = g.vel[d.uN + d.vN + ((long long)k * ny + j) * nx + i];
  double nl2 = 1 / el2;
  double vN = ((double)P.pvx[p] * ex2 + (double)P.pvy[p] * ey2 + (double)P.pvz[p] * ez2) * nl2;
  double gN = (guS * ex2 + gvS * ey2 + gwS * ez2) * nl2;
  P.pvx[p] = (float)(vN * ex2 + (guS - gN * ex2) + kx);
  P.pvy[p] = (float)(vN * ey2 + (gvS - gN * ey2) + ky);
  P.pvz[p] = (float)(vN * ez2 + (gwS - gN * ez2) + kz);
}
static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
static size_t ev_max_windows(int cap) { return (size_t)(cap + kEvW - 1) / kEvW + 1; }
size_t evaporation_scratch_bytes(int cap) {
  const size_t c = (size_t)cap, nw = ev_max_windows(cap);
  return align256(8 * c) + 4 * align256(4 * c) + align256(8 * nw) + 2 * align256(4 * nw) + align256(2 * kEvKMax * nw);
}
EvapScratch evap_carve(void* base, int cap) {
  const size_t c = (size_t)cap, nw = ev_max_windows(cap);
  char* q = (char*)base; EvapScratch e;
  e.thr = (long long*)q; q += align256(8 * c);
  e.b = (uint32_t*)q; q += align256(4 * c);
  e.ejP = (int*)q; q += align256(4 * c);
  e.ejS = (uint32_t*)q; q += align256(4 * c);
  q += align256(4 * c);                           // reserved
  e.wsum = (double*)q; q += align256(8 * nw);
  e.L = (int*)q; q += align256(4 * nw);
  e.Ew = (int*)q; q += align256(4 * nw);
  e.table = (unsigned short*)q;
  return e;
}
void launch_evap_prepare(const Dims& d, const GridDev& g, const PartsDev& P, double freezeT, double rate, double dt,
                         uint8_t* cand, int* blockCounts, int* list, int* nC, const EvapScratch& es, cudaStream_t s) {
  const int gp = grid_for(P.nP, 256);
  k_evap_flags<<<gp, 256, 0, s>>>(d, g, P, freezeT, cand);
  launch_compact(cand, P.nP, 2, blockCounts, list, nC, s);
  k_evap_thr<<<gp, 256, 0, s>>>(P, freezeT, rate, dt, list, nC, es.thr);
}
void launch_evap_pass(int nP, const int* list, const int* nC, const EvapScratch& es, int t0, int eoff,
                      const uint32_t* sStart, DevStatus* st, cudaStream_t s) {
  const int nw = (int)ev_max_windows(nP);
  k_evap_wsum<<<nw, 256, 0, s>>>(es.thr, nC, t0, es.wsum);
  k_evap_band<<<1, 1024, 0, s>>>(es.wsum, nC, t0, es.L, st);
  // twelve rounds of the four blocks an SM holds: with four or eight a window's
  // share is too coarse at 256^3 (3150 us), with 32 the windows' loads come back
  const int blocks = (int)std::min<long long>((long long)nw * (kEvKMax / 32), 148 * 48);
  k_evap_table<<<blocks, kEvTableThreads, 0, s>>>(es.thr, nC, t0, sStart, es.L, st, es.b, es.table);
  k_evap_chain<<<1, 32, 0, s>>>(nC, t0, es.L, es.table, es.b, es.thr, sStart, es.Ew, st);
  k_evap_emit<<<nw, 256, 0, s>>>(nC, t0, es.b, es.thr, es.Ew, list, eoff, es.ejP, es.ejS, st);
}
void launch_evap_apply(const Dims& d, const GridDev& g, const PartsDev& P, double freezeT, const EvapScratch& es,
                       int nEj, cudaStream_t s) {
  if (nEj > 0) k_evap_apply<<<grid_for(nEj, 256), 256, 0, s>>>(d, g, P, freezeT, es.ejP, es.ejS, nEj);
}

// ------------------------------------------------------------ phase changes
// _updatePhaseChanges, js/solver.js:3152-3281: steam counts per cell
// (integer atomics, exact), then independent per-particle transitions.
__device__ __forceinline__ long long clamp_cell(const Dims& d, double x, double y, double z, int& i, int& j, int& k) {
  i = jtrunc(over_dx(d, x)); j = jtrunc(over_dx(d, y)); k = jtrunc(over_dx(d, z));
  if (i < 0) i = 0; else if (i >= d.nx) i = d.nx - 1;
  if (j < 0) j = 0; else if (j >= d.ny) j = d.ny - 1;
  if (k < 0) k = 0; else if (k >= d.nz) k = d.nz - 1;
  return ((long long)k * d.ny + j) * d.nx + i;
}
__global__ void k_steam_count(Dims d, PartsDev P, int* __restrict__ cnt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP || P.pflag[p] != 2) return;
  int i, j, k;
  atomicAdd(&cnt[clamp_cell(d, P.px[p], P.py[p], P.pz[p], i, j, k)], 1);
}
__device__ __forceinline__ uint32_t js_mul_u32(double a, double b) {
  double m = fmod(a * b, 4294967296.0); if (m < 0) m += 4294967296.0;
  return (uint32_t)m;
}
__device__ __forceinline__ uint32_t spin_hash(uint32_t a, uint32_t b, uint32_t c) {   // :3145-3150
  uint32_t s = a ^ js_mul_u32(b, 2654435769.0) ^ js_mul_u32(c, 2246822507.0) ^ js_mul_u32(1370176631.0, 3266489909.0);
  s = lcg_next(s);
  s ^= s >> 13; s = js_mul_u32(s, 1540483477.0); s ^= s >> 15;
  return s;
}
__global__ void k_phase_update(Dims d, GridDev g, PartsDev P, PhaseParams pp, const int* __restrict__ cnt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  const uint8_t* type = g.type;
  int nx = d.nx, ny = d.ny, nz = d.nz; long long nxy = (long long)nx * ny;
  int f = P.pflag[p], i, j, k;
  double T = P.pT[p];
  if (f == 0) {
    if (T <= pp.snowT && T > 1e-3) {
      long long cB = clamp_cell(d, P.px[p], P.py[p], P.pz[p], i, j, k);
      bool atSurf = (k > 0 && type[cB - nxy] != WS_FLUID) || (k < nz - 1 && type[cB + nxy] != WS_FLUID) ||
                    (j > 0 && type[cB - nx] != WS_FLUID) || (j < ny - 1 && type[cB + nx] != WS_FLUID) ||
                    (i > 0 && type[cB - 1] != WS_FLUID) || (i < nx - 1 && type[cB + 1] != WS_FLUID);
      if (atSurf) { P.pflag[p] = 5; P.pvx[p] = P.pvy[p] = P.pvz[p] = 0.f; P.pAir[p] = 1.f; }
    }
  } else if (f == 5) {
    if (T >= pp.meltT) {
      long long c = clamp_cell(d, P.px[p], P.py[p], P.pz[p], i, j, k);
      P.pflag[p] = type[c] == WS_FLUID ? 0 : 4;
      P.pAir[p] = 0.f; P.pWx[p] = P.pWy[p] = P.pWz[p] = 0.f;
    }
  } else if (T > 1e-3) {
    if (f == 2) {
      if (T <= pp.rainT && (double)P.pAir[p] >= pp.rainLiftAge) {
        P.pflag[p] = 4; P.pAir[p] = 0.f; P.pvx[p] = P.pvy[p] = P.pvz[p] = 0.f; P.pWx[p] = P.pWy[p] = P.pWz[p] = 0.f;
        f = 4;
      } else if (T <= pp.cloudT) {
        double rx = (double)P.px[p] - d.cx, ry = (double)P.py[p] - d.cy, rz = (double)P.pz[p] - d.cz;
        if (sqrt(rx * rx + ry * ry + rz * rz) >= pp.cloudBase) {
          i = jtrunc(over_dx(d, P.px[p])); j = jtrunc(over_dx(d, P.py[p])); k = jtrunc(over_dx(d, P.pz[p]));
          int i0 = i > 0 ? i - 1 : 0, i1 = i < nx - 1 ? i + 1 : nx - 1;
          int j0 = j > 0 ? j - 1 : 0, j1 = j < ny - 1 ? j + 1 : ny - 1;
          int k0 = k > 0 ? k - 1 : 0, k1 = k < nz - 1 ? k + 1 : nz - 1;
          double sum = 0;
          for (int kk = k0; kk <= k1; kk++) for (int jj = j0; jj <= j1; jj++) {
            long long row = ((long long)kk * ny + jj) * nx;
            for (int ii = i0; ii <= i1; ii++) sum += cnt[row + ii];
          }
          if (sum / 27 >= pp.cloudP) { P.pflag[p] = 3; P.pAir[p] = 0.f; f = 3; }
        }
      }
    } else if (f == 3) {
      if (T >= pp.cloudT + 0.05) { P.pflag[p] = 2; f = 2; }
    } else if ((f == 1 || f == 4) && T <= pp.snowT) {   // spray and rain freeze (:3253)
      P.pflag[p] = 5; P.pvx[p] = P.pvy[p] = P.pvz[p] = 0.f; P.pAir[p] = 0.f; P.pWx[p] = P.pWy[p] = P.pWz[p] = 0.f;
    }
  }
}
// spin bookkeeping (:3259-3280), a separate pass over the final flags
__global__ void k_phase_spin(PartsDev P, uint32_t tick, double dt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP) return;
  int f = P.pflag[p];
  if (f != 2 && f != 3) return;
  float wx = P.pWx[p], wy = P.pWy[p], wz = P.pWz[p];
  if (f == 2 && P.pAir[p] <= 1e-6f && wx == 0.f && wy == 0.f && wz == 0.f) {
    uint32_t sd = 0x51ab3c77u;
    double h1 = spin_hash(sd, (uint32_t)p, tick) / 4294967296.0;
    double h2 = spin_hash(sd + 1, (uint32_t)p, tick) / 4294967296.0;
    double h3 = spin_hash(sd + 2, (uint32_t)p, tick) / 4294967296.0;
    double zz = 2 * h2 - 1, rr = sqrt(dmax(0, 1 - zz * zz)), th = 6.283185306 * h1;
    double Tp = P.pT[p]; if (!(Tp > 0.05)) Tp = 0.05; else if (Tp > 1.15) Tp = 1.15;
    double wSpd = 3.0 * sqrt(Tp) * (0.5 + h3);
    wx = (float)(rr * cos(th) * wSpd); wy = (float)(zz * wSpd); wz = (float)(rr * sin(th) * wSpd);
  }
  double wm = sqrt((double)wx * wx + (double)wy * wy + (double)wz * wz);
  if (wm > 1e-6) P.pPh[p] = (float)((double)P.pPh[p] + wm * dt);
  double damp = dmax(0, 1 - 0.12 * dt);
  P.pWx[p] = (float)(wx * damp); P.pWy[p] = (float)(wy * damp); P.pWz[p] = (float)(wz * damp);
}
void launch_phase(const Dims& d, const GridDev& g, const PartsDev& P, const PhaseParams& pp, int* cnt, cudaStream_t s) {
  if (P.nP <= 0) return;
  cudaMemsetAsync(cnt, 0, sizeof(int) * d.nCells, s);
  unsigned gp = grid_for(P.nP, 256);
  k_steam_count<<<gp, 256, 0, s>>>(d, P, cnt);
  k_phase_update<<<gp, 256, 0, s>>>(d, g, P, pp, cnt);
  if (pp.spinOn && pp.dt > 0) k_phase_spin<<<gp, 256, 0, s>>>(P, pp.tick, pp.dt);
}

// ------------------------------------------------------------ frame-end rescue
// _pushSurfaceChunk, js/solver.js:3496-3587 — independent per particle.
__global__ void k_push_surface(Dims d, GridDev g, PartsDev P, TerrainDev t, double oceanR, double coreR, double atmosphereH) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP || !t.has) return;
  const double cx = d.cx, cy = d.cy, cz = d.cz, dx = d.dx;
  double x = P.px[p], y = P.py[p], z = P.pz[p];
  float fvx = P.pvx[p], fvy = P.pvy[p], fvz = P.pvz[p];
  double ex = x - cx, ey = y - cy, ez = z - cz;
  double er = sqrt(ex * ex + ey * ey + ez * ez); if (er == 0) er = 1e-9;
  bool fixed = false, rockFixed = false, velChanged = false;
  double outer = d.domainR - dx * 0.02;
  double skyHi = oceanR + atmosphereH - 1e-3 * dx;
  if (er > skyHi) {
    x = cx + ex / er * skyHi; y = cy + ey / er * skyHi; z = cz + ez / er * skyHi;
    double outward = ((double)fvx * ex + (double)fvy * ey + (double)fvz * ez) / er;
    if (outward > 0) { fvx = (float)(fvx - ex / er * outward); fvy = (float)(fvy - ey / er * outward); fvz = (float)(fvz - ez / er * outward); velChanged = true; }
    ex = x - cx; ey = y - cy; ez = z - cz; er = skyHi;
    fixed = true;
  }
  if (er <= d.domainR && rock_cell_at(d, g.staticTypes, x, y, z)) {
    rockFixed = true;
    int tries = 0;
    while (rock_cell_at(d, g.staticTypes, x, y, z) && tries < d.nx * 2) {
      x += ex / er * dx * 0.5; y += ey / er * dx * 0.5; z += ez / er * dx * 0.5; tries++;
    }
    double exR = x - cx, eyR = y - cy, ezR = z - cz;
    double erR = sqrt(exR * exR + eyR * eyR + ezR * ezR); if (erR == 0) erR = 1e-9;
    double wantR = terrain_radius_at(t, coreR, x, y, z) + dx * 0.06;
    if (erR > wantR) { x = cx + exR / erR * wantR; y = cy + eyR / erR * wantR; z = cz + ezR / erR * wantR; }
    int kR = 0;
    while (rock_cell_at(d, g.staticTypes, x, y, z) && kR < 4) {
      x += exR / erR * dx * 0.5; y += eyR / erR * dx * 0.5; z += ezR / erR * dx * 0.5; kR++;
    }
    fixed = true;
  } else if (P.pflag[p] == 0 && er <= d.domainR) {
    double Rt = terrain_radius_at(t, coreR, x, y, z);
    if (er < Rt - dx * 0.5) {
      rockFixed = true;
      x = cx + ex / er * (Rt + dx * 0.05); y = cy + ey / er * (Rt + dx * 0.05); z = cz + ez / er * (Rt + dx * 0.05);
      int t2 = 0;
      while (rock_cell_at(d, g.staticTypes, x, y, z) && t2 < 8) {
        x += ex / er * dx * 0.5; y += ey / er * dx * 0.5; z += ez / er * dx * 0.5; t2++;
      }
      fixed = true;
    }
  }
  double finalR = sqrt((x - cx) * (x - cx) + (y - cy) * (y - cy) + (z - cz) * (z - cz));
  double capR = P.pflag[p] == 0 ? outer : skyHi;
  if (finalR > capR) {
    x = cx + (x - cx) * capR / finalR; y = cy + (y - cy) * capR / finalR; z = cz + (z - cz) * capR / finalR;
    fixed = true;
  }
  if (fixed) {
    P.px[p] = (float)x; P.py[p] = (float)y; P.pz[p] = (float)z;
    double vr = ((double)fvx * ex + (double)fvy * ey + (double)fvz * ez) / er;
    if (rockFixed && vr < 0) { fvx = (float)(fvx - ex / er * vr); fvy = (float)(fvy - ey / er * vr); fvz = (float)(fvz - ez / er * vr); velChanged = true; }
  }
  if (velChanged) { P.pvx[p] = fvx; P.pvy[p] = fvy; P.pvz[p] = fvz; }
}
void launch_push_surface(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t,
                         double oceanR, double coreR, double atmosphereH, cudaStream_t s) {
  if (P.nP <= 0) return;
  k_push_surface<<<grid_for(P.nP, 256), 256, 0, s>>>(d, g, P, t, oceanR, coreR, atmosphereH);
}

// ------------------------------------------------------------ density splat
// _splatInto, js/solver.js:3792-3820 (float atomics on the corner lattice)
__global__ void k_splat(Dims d, GridDev g, PartsDev P, double spacing) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP || P.pflag[p] != 0) return;
  double dx = d.dx, r = 1.6 * spacing, r2 = r * r;
  long long sj = d.nx + 1, sk = (long long)(d.ny + 1) * sj;
  double X = P.px[p], Y = P.py[p], Z = P.pz[p];
  double fi = floor(over_dx(d, X)), fj = floor(over_dx(d, Y)), fk = floor(over_dx(d, Z));
  int i0 = !(fi >= 0) ? 0 : (fi > d.nx - 1 ? d.nx - 1 : (int)fi);
  int j0 = !(fj >= 0) ? 0 : (fj > d.ny - 1 ? d.ny - 1 : (int)fj);
  int k0 = !(fk >= 0) ? 0 : (fk > d.nz - 1 ? d.nz - 1 : (int)fk);
  double fx = X - i0 * dx, fy = Y - j0 * dx, fz = Z - k0 * dx;
  for (int kk = 0; kk < 2; kk++) {
    double czz = kk == 0 ? fz : fz - dx;
    for (int jj = 0; jj < 2; jj++) {
      double cyy = jj == 0 ? fy : fy - dx;
      for (int ii = 0; ii < 2; ii++) {
        double cxx = ii == 0 ? fx : fx - dx;
        double d2 = cxx * cxx + cyy * cyy + czz * czz;
        if (d2 >= r2) continue;
        double ww = 1 - d2 / r2; ww = ww * ww;
        atomicAdd(&g.dens[(k0 + kk) * sk + (j0 + jj) * sj + (i0 + ii)], (float)ww);
      }
    }
  }
}
void launch_splat(const Dims& d, const GridDev& g, const PartsDev& P, double spacing, cudaStream_t s) {
  long long nd = (long long)(d.nx + 1) * (d.ny + 1) * (d.nz + 1);
  cudaMemsetAsync(g.dens, 0, sizeof(float) * nd, s);
  if (P.nP <= 0) return;
  k_splat<<<grid_for(P.nP, 256), 256, 0, s>>>(d, g, P, spacing);
}

// whether this block is the last of `blocks` to come here, with the others'
// global writes visible; the ticket is back at zero afterwards. Every thread
// of those blocks calls.
__device__ __forceinline__ bool last_block(unsigned* ticket, unsigned blocks) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == blocks - 1;
    if (last) *ticket = 0;
    __threadfence();
  }
  __syncthreads();
  return last;
}

// ------------------------------------------------------------ marching tets (FP64)
// MarchingTetrahedra.build (js/surface.js:66-177): six tets per cell, up to
// two triangles each, vertices in the reference's order (cells in index
// order, then tets, then case triangles), signed volume in FP64.
// Corner c of a cell is at (x, y, z) = (((c ^ c >> 1) & 1), (c >> 1) & 1, c >> 2).
constexpr int kTets[6][4] = { {0,5,1,6},{0,1,2,6},{0,2,3,6},{0,3,7,6},{0,7,4,6},{0,4,5,6} };
constexpr int kTetEdges[6][2] = { {0,1},{1,2},{2,0},{0,3},{1,3},{2,3} };
constexpr int kTetTris[16] = { 0,1,1,2,1,2,2,1,1,2,2,1,2,1,1,0 };
constexpr int kTetCases[16][2][3] = {
  {{0,0,0},{0,0,0}}, {{0,2,3},{0,0,0}}, {{0,1,4},{0,0,0}}, {{2,3,4},{2,4,1}},
  {{2,1,5},{0,0,0}}, {{0,3,5},{0,5,1}}, {{0,4,5},{0,5,2}}, {{3,5,4},{0,0,0}},
  {{3,4,5},{0,0,0}}, {{0,2,5},{0,5,4}}, {{0,1,5},{0,5,3}}, {{2,1,5},{0,0,0}},
  {{2,1,4},{2,4,3}}, {{0,1,4},{0,0,0}}, {{0,2,3},{0,0,0}}, {{0,0,0},{0,0,0}} };
// The 25 directed edges that the six tets of a cell name (an edge met in both
// directions rounds differently in each), and per sign pattern of the eight
// corners the directed edges that its triangles use (at most 18) and their
// number of triangles (at most 12).
constexpr int kMtEdges = 25, kMtVerts = 18;
struct MtTables {
  unsigned mask[256];
  uint8_t tris[256];
  uint8_t from[kMtEdges], to[kMtEdges], id[6][6], tet[6][4], cases[16][2][3], nTri[16];
};
constexpr MtTables mt_tables() {
  MtTables t{};
  int n = 0;
  for (int q = 0; q < 6; q++) {
    for (int c = 0; c < 4; c++) t.tet[q][c] = (uint8_t)kTets[q][c];
    for (int e = 0; e < 6; e++) {
      const int a = kTets[q][kTetEdges[e][0]], b = kTets[q][kTetEdges[e][1]];
      int id = 0;
      while (id < n && !(t.from[id] == a && t.to[id] == b)) id++;
      if (id == n) { t.from[n] = (uint8_t)a; t.to[n] = (uint8_t)b; n++; }
      t.id[q][e] = (uint8_t)id;
    }
  }
  for (int code = 0; code < 16; code++) {
    t.nTri[code] = (uint8_t)kTetTris[code];
    for (int e = 0; e < 2; e++)
      for (int v = 0; v < 3; v++) t.cases[code][e][v] = (uint8_t)kTetCases[code][e][v];
  }
  for (int cfg = 0; cfg < 256; cfg++)
    for (int q = 0; q < 6; q++) {
      int code = 0;
      for (int c = 0; c < 4; c++) if (cfg >> kTets[q][c] & 1) code |= 1 << c;
      t.tris[cfg] = (uint8_t)(t.tris[cfg] + kTetTris[code]);
      for (int e = 0; e < kTetTris[code]; e++)
        for (int v = 0; v < 3; v++) t.mask[cfg] |= 1u << t.id[q][kTetCases[code][e][v]];
    }
  return t;
}
__device__ const MtTables g_mt = mt_tables();

// Three passes find the cells that emit triangles, in index order, with the
// place of their first triangle: the sign pattern of every cell and the
// (cells, triangles) of each 1024; a scan of those; the list. They are bound
// by the corner field's read and their launches.
constexpr int kMtBlock = 1024;                           // cells per block of the count and list passes
// counts of a block, packed: cells << 34 | triangles (up to 2^30 cells of 12)
__global__ void __launch_bounds__(256) k_mt_count(Dims d, const float* __restrict__ dens, float iso, uint8_t* __restrict__ cfg,
                                                  unsigned long long* __restrict__ tot) {
  __shared__ unsigned sw[8];
  unsigned mine = 0;                                     // cells << 16 | triangles
  const unsigned sj = (unsigned)d.nx + 1u, sk = ((unsigned)d.ny + 1u) * sj;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const long long c = blockIdx.x * (long long)kMtBlock + q * 256 + threadIdx.x;
    unsigned m = 0;
    if (c < d.nCells) {
      int i, j, k; cell_ijk(d, c, i, j, k);
      const float* p = dens + ((unsigned)k * sk + (unsigned)j * sj + (unsigned)i);
      const float v[8] = { p[0], p[1], p[sj + 1], p[sj], p[sk], p[sk + 1], p[sk + sj + 1], p[sk + sj] };
#pragma unroll
      for (int e = 0; e < 8; e++) m |= (v[e] > iso ? 1u : 0u) << e;
      if (m != 0 && m != 255u) {
        bool low = false;                                // a corner at or below iso: a NaN alone is neither
#pragma unroll
        for (int e = 0; e < 8; e++) low |= v[e] <= iso;
        if (!low) m = 0;
        const unsigned n = g_mt.tris[m];
        if (n) mine += 1u << 16 | n;
      }
    }
    cfg[c] = (uint8_t)m;                                 // the array is padded to whole blocks
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) mine += sw[w];
    tot[blockIdx.x] = (unsigned long long)(mine >> 16) << 34 | (mine & 0xffffu);
  }
}
// exclusive scan in place; the total lands in tot[nb], the emission's ticket (0) behind it
__global__ void __launch_bounds__(1024) k_mt_scan(unsigned long long* __restrict__ tot, int nb) {
  __shared__ unsigned long long ws[32];
  unsigned long long carry = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    const unsigned long long v = i < nb ? tot[i] : 0;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) { const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
      unsigned long long a = ws[lane];
      for (int o = 1; o < 32; o <<= 1) { const unsigned long long y = __shfl_up_sync(0xffffffffu, a, o); if (lane >= o) a += y; }
      ws[lane] = a;
    }
    __syncthreads();
    if (i < nb) tot[i] = x - v + (w > 0 ? ws[w - 1] : 0) + carry;
    carry += ws[31];
    __syncthreads();                                     // ws is rewritten by the next round
  }
  if (threadIdx.x == 0) { tot[nb] = carry; tot[nb + 1] = 0; }
}
// (cell, its first triangle) of every listed cell
__global__ void __launch_bounds__(256) k_mt_list(const uint8_t* __restrict__ cfg, const unsigned long long* __restrict__ tot,
                                                 uint2* __restrict__ list) {
  __shared__ unsigned sw[8];
  const long long c0 = blockIdx.x * (long long)kMtBlock + threadIdx.x * 4;
  const unsigned four = *reinterpret_cast<const unsigned*>(cfg + c0);
  unsigned n[4], mine = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) { n[q] = g_mt.tris[(four >> (8 * q)) & 255u]; if (n[q]) mine += 1u << 16 | n[q]; }
  unsigned x = mine;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 1; o < 32; o <<= 1) { const unsigned y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
  if (lane == 31) sw[w] = x;
  __syncthreads();
  if (!mine) return;
  unsigned before = x - mine;
  for (int q = 0; q < w; q++) before += sw[q];
  const unsigned long long t = tot[blockIdx.x];
  unsigned at = (unsigned)(t >> 34) + (before >> 16), tri = (unsigned)t + (before & 0xffffu);
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (n[q]) { list[at++] = make_uint2((unsigned)(c0 + q), tri); tri += n[q]; }
}
// The triangles of 16 listed cells per block and round, each step over all
// threads: corner values and gradients, the vertices of the crossed directed
// edges (each once: 13 on average, where a cell's triangles name 21), the
// triangles' orientation and volume from those, and the output, whose floats
// of one round are contiguous. Bound by instruction and shared-memory latency
// (FP64 division and square root, five per vertex) at the ten blocks an SM
// whose vertices fit. A thread per cell that walked its triangles, once to
// count and once to emit, took 53 + 95 us for 1.3M vertices at 128^3 (29 + 35
// at 48^3, where its chain was the whole time); this, with the sums of the last
// block, which writes them to host memory: 57 and 18. Rounds of 32
// cells and 128 threads: the same.
// maxVerts negative: the volume only. A mesh beyond maxVerts: its vertex count
// only, at once (the scan has it), so that the caller makes room and emits once.
// A fault latched in err before leaves the vertices of the last mesh as they are.
constexpr int kMtCells = 16, kMtThreads = 4 * kMtCells;
__global__ void __launch_bounds__(kMtThreads) k_mt_emit(Dims d, const float* __restrict__ dens, double iso, float isoF,
                                                 const uint2* __restrict__ list, const unsigned long long* __restrict__ total,
                                                 long long maxVerts, float* pos, float* __restrict__ nrm,
                                                 double* __restrict__ partials, unsigned* ticket, double* __restrict__ out,
                                                 const int* __restrict__ err) {
  __shared__ float cv[kMtCells][9];
  __shared__ double gr[3][kMtCells * 8];
  __shared__ double P[3][kMtCells * kMtVerts], N[3][kMtCells * kMtVerts];
  __shared__ unsigned short vdesc[kMtCells * kMtVerts], tv[kMtCells * 12][3];
  __shared__ int ci[kMtCells], cj[kMtCells], ck[kMtCells], sNV, sNT;
  __shared__ unsigned mask[kMtCells], tri0;
  __shared__ unsigned short vBase[kMtCells], tBase[kMtCells];
  __shared__ uint8_t cfg[kMtCells], sFrom[kMtEdges], sTo[kMtEdges], sId[6][6], sTet[6][4], sCase[16][2][3], sNTri[16];
  __shared__ double sv[kMtThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  const int fault = err ? *err : 0;                        // in flight with the total
  const unsigned n = (unsigned)(*total >> 34);
  const double nVerts = 3.0 * (double)(*total & ((1ull << 34) - 1));
  if (maxVerts >= 0 && nVerts > (double)maxVerts) {
    if (blockIdx.x == 0 && tid == 0) out[1] = nVerts;
    return;
  }
  const unsigned blocks = min(gridDim.x, max((n + kMtCells - 1) / kMtCells, 1u));   // those with cells (one without any)
  if (blockIdx.x >= blocks) return;
  if (fault) pos = nullptr;
  for (int t = tid; t < 16 * 6; t += kMtThreads) ((uint8_t*)sCase)[t] = ((const uint8_t*)g_mt.cases)[t];
  if (tid < kMtEdges) { sFrom[tid] = g_mt.from[tid]; sTo[tid] = g_mt.to[tid]; }
  if (tid < 36) ((uint8_t*)sId)[tid] = ((const uint8_t*)g_mt.id)[tid];
  if (tid < 24) ((uint8_t*)sTet)[tid] = ((const uint8_t*)g_mt.tet)[tid];
  if (tid < 16) sNTri[tid] = g_mt.nTri[tid];
  const unsigned sj = (unsigned)d.nx + 1u, sk = ((unsigned)d.ny + 1u) * sj;
  const double dx = d.dx, r2dx = 0.5 * d.rdx;
  double vol = 0;
  for (unsigned ch = blockIdx.x * kMtCells; ch < n; ch += gridDim.x * kMtCells) {
    // corners: value, sign pattern and gradient (central differences, clamped to the lattice)
#pragma unroll
    for (int q = 0; q < kMtCells * 8; q += kMtThreads) {
      const int t = q + tid, cell = t >> 3, c = t & 7;
      float v = 0.f;
      int i = 0, j = 0, k = 0;
      if (ch + cell < n) {
        cell_ijk(d, list[ch + cell].x, i, j, k);
        const int x = i + ((c ^ c >> 1) & 1), y = j + ((c >> 1) & 1), z = k + (c >> 2);
        const int ip = min(x + 1, d.nx), im = max(x - 1, 0), jp = min(y + 1, d.ny), jm = max(y - 1, 0);
        const int kp = min(z + 1, d.nz), km = max(z - 1, 0);
        const unsigned zy = (unsigned)z * sk + (unsigned)y * sj, zx = (unsigned)z * sk + (unsigned)x, yx = (unsigned)y * sj + (unsigned)x;
        v = dens[zy + x];
        const double ddx = (double)dens[zy + ip] - (double)dens[zy + im];
        const double ddy = (double)dens[zx + (unsigned)jp * sj] - (double)dens[zx + (unsigned)jm * sj];
        const double ddz = (double)dens[yx + (unsigned)kp * sk] - (double)dens[yx + (unsigned)km * sk];
        // dx a power of two: the division by 2 dx is the exact product
        gr[0][t] = d.dxPow2 ? ddx * r2dx : ddx / (2 * dx);
        gr[1][t] = d.dxPow2 ? ddy * r2dx : ddy / (2 * dx);
        gr[2][t] = d.dxPow2 ? ddz * r2dx : ddz / (2 * dx);
        cv[cell][c] = v;
      }
      const unsigned m = (__ballot_sync(0xffffffffu, v > isoF) >> (lane & 24)) & 255u;
      if (c == 0) { cfg[cell] = ch + cell < n ? (uint8_t)m : 0; ci[cell] = i; cj[cell] = j; ck[cell] = k; }
    }
    __syncthreads();
    if (tid < kMtCells) {
      const unsigned m = cfg[tid], e = g_mt.mask[m];
      const int own = __popc(e) << 16 | g_mt.tris[m];
      int x = own;
      const unsigned all = kMtCells == 32 ? 0xffffffffu : (1u << (kMtCells & 31)) - 1u;
      for (int o = 1; o < kMtCells; o <<= 1) { const int y = __shfl_up_sync(all, x, o); if (lane >= o) x += y; }
      mask[tid] = e;
      vBase[tid] = (unsigned short)((x - own) >> 16); tBase[tid] = (unsigned short)((x - own) & 0xffff);
      if (tid == kMtCells - 1) { sNV = x >> 16; sNT = x & 0xffff; }
      if (tid == 0) tri0 = list[ch].y;
    }
    __syncthreads();
    {
      const int cell = tid >> 2, part = tid & 3;         // four threads list a cell's edges and triangles
      const unsigned e = mask[cell], m = cfg[cell];
      for (int id = part; id < kMtEdges; id += 4)
        if (e >> id & 1) vdesc[vBase[cell] + __popc(e & ((1u << id) - 1u))] = (unsigned short)(cell << 5 | id);
      int at = tBase[cell];
      if (m)
        for (int t = 0; t < 6; t++) {
          const int code = (m >> sTet[t][0] & 1) | (m >> sTet[t][1] & 1) << 1 | (m >> sTet[t][2] & 1) << 2 | (m >> sTet[t][3] & 1) << 3;
          for (int u = 0; u < sNTri[code]; u++, at++)
            if ((at & 3) == part)
              for (int vi = 0; vi < 3; vi++) {
                const int id = sId[t][sCase[code][u][vi]];
                tv[at][vi] = (unsigned short)(vBase[cell] + __popc(e & ((1u << id) - 1u)));
              }
        }
    }
    __syncthreads();
    const int nV = sNV, nT = sNT;
    for (int t = tid; t < nV; t += kMtThreads) {
      const int cell = vdesc[t] >> 5, id = vdesc[t] & 31, a = sFrom[id], b = sTo[id];
      const double va = cv[cell][a], vb = cv[cell][b], den = vb - va;
      double tt = den != 0 ? (iso - va) / den : 0.5;
      if (tt < 0) tt = 0; else if (tt > 1) tt = 1;
      const int ax = (a ^ a >> 1) & 1, ay = (a >> 1) & 1, az = a >> 2, bx = (b ^ b >> 1) & 1, by = (b >> 1) & 1, bz = b >> 2;
      P[0][t] = ((ci[cell] + ax) + (bx - ax) * tt) * dx;
      P[1][t] = ((cj[cell] + ay) + (by - ay) * tt) * dx;
      P[2][t] = ((ck[cell] + az) + (bz - az) * tt) * dx;
      const int A = cell * 8 + a, B = cell * 8 + b;
      const double nx = -(gr[0][A] + (gr[0][B] - gr[0][A]) * tt), ny = -(gr[1][A] + (gr[1][B] - gr[1][A]) * tt);
      const double nz = -(gr[2][A] + (gr[2][B] - gr[2][A]) * tt);
      double nl = sqrt(nx * nx + ny * ny + nz * nz); if (nl == 0) nl = 1;
      N[0][t] = nx / nl; N[1][t] = ny / nl; N[2][t] = nz / nl;
    }
    __syncthreads();
    for (int t = tid; t < nT; t += kMtThreads) {
      const int a = tv[t][0];
      int b = tv[t][1], c = tv[t][2];
      const double ux = P[0][b] - P[0][a], uy = P[1][b] - P[1][a], uz = P[2][b] - P[2][a];
      const double vx = P[0][c] - P[0][a], vy = P[1][c] - P[1][a], vz = P[2][c] - P[2][a];
      const double fx = uy * vz - uz * vy, fy = uz * vx - ux * vz, fz = ux * vy - uy * vx;
      const double gx = N[0][a] + N[0][b] + N[0][c], gy = N[1][a] + N[1][b] + N[1][c], gz = N[2][a] + N[2][b] + N[2][c];
      if (fx * gx + fy * gy + fz * gz < 0) {             // outward: swap the last two vertices
        const int o = b; b = c; c = o;
        tv[t][1] = (unsigned short)b; tv[t][2] = (unsigned short)c;
      }
      vol += (P[0][a] * (P[1][b] * P[2][c] - P[1][c] * P[2][b]) - P[1][a] * (P[0][b] * P[2][c] - P[0][c] * P[2][b]) +
              P[2][a] * (P[0][b] * P[1][c] - P[0][c] * P[1][b])) / 6;
    }
    __syncthreads();
    // the next round's corners, before its first barrier, touch none of what this reads
    if (pos)
      for (int f = tid; f < nT * 9; f += kMtThreads) {
        const int t = f / 9, r = f - t * 9, vi = r / 3, q = r - vi * 3, v = tv[t][vi];
        pos[(long long)tri0 * 9 + f] = (float)P[q][v];
        nrm[(long long)tri0 * 9 + f] = (float)N[q][v];
      }
  }
  vol = warp_sum(vol);
  if (lane == 0) sv[tid >> 5] = vol;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kMtThreads / 32; w++) vol += sv[w];
    partials[blockIdx.x] = vol;
  }
  // the last block: the volumes in a fixed order, and the vertex count
  if (!last_block(ticket, blocks)) return;
  vol = 0;
  for (unsigned i = tid; i < blocks; i += kMtThreads) vol += __ldcg(partials + i);
  vol = warp_sum(vol);
  if (lane == 0) sv[tid >> 5] = vol;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kMtThreads / 32; w++) vol += sv[w];
    out[0] = vol; out[1] = nVerts;
  }
}
// scratch: list (8 bytes a cell), block totals and ticket, partial volumes, sign patterns
static int mt_blocks(long long nCells) { return (int)grid_for(nCells, kMtBlock); }
constexpr int kMtGrid = 148 * 10;
size_t mt_scratch_bytes(long long nCells) {
  const size_t nb = (size_t)mt_blocks(nCells);
  return 8 * (size_t)nCells + 8 * (nb + 2) + 8 * kMtGrid + kMtBlock * nb;
}
struct MtScratch { uint2* list; unsigned long long* tot; double* partials; uint8_t* cfg; int nb; };
static MtScratch mt_carve(void* scratch, long long nCells) {
  MtScratch m;
  char* q = (char*)scratch;
  m.nb = mt_blocks(nCells);
  m.list = (uint2*)q; q += 8 * (size_t)nCells;
  m.tot = (unsigned long long*)q; q += 8 * (size_t)(m.nb + 2);
  m.partials = (double*)q; q += 8 * kMtGrid;
  m.cfg = (uint8_t*)q;
  return m;
}
// the largest float at or below iso: a float exceeds iso exactly when it exceeds that
static float iso_floor(double iso) {
  float f = (float)iso;
  if ((double)f > iso) f = std::nextafterf(f, -INFINITY);
  return f;
}
int launch_mt_list(const Dims& d, const float* dens, double iso, void* scratch, cudaStream_t s) {
  const MtScratch m = mt_carve(scratch, d.nCells);
  k_mt_count<<<m.nb, 256, 0, s>>>(d, dens, iso_floor(iso), m.cfg, m.tot);
  k_mt_scan<<<1, 1024, 0, s>>>(m.tot, m.nb);
  k_mt_list<<<m.nb, 256, 0, s>>>(m.cfg, m.tot, m.list);
  return 3;
}
int launch_mt_emit(const Dims& d, const float* dens, double iso, long long maxVerts, float* pos, float* nrm, double* out,
                   const int* err, void* scratch, cudaStream_t s) {
  const MtScratch m = mt_carve(scratch, d.nCells);
  const int grid = (int)std::min<long long>(grid_for(d.nCells, kMtCells), kMtGrid);
  k_mt_emit<<<grid, kMtThreads, 0, s>>>(d, dens, iso, iso_floor(iso), m.list, m.tot + m.nb, maxVerts, pos, nrm, m.partials,
                                           (unsigned*)(m.tot + m.nb + 1), out, err);
  return 1;
}

// ------------------------------------------------------------ particle reductions
// mode 0: kinetic energy sum of 0.5 mp v^2 (FP64); mode 1: census counts
// (liquid 0/1/4, ice 5, vapour 2/3) as exact FP64 integers. Both read their
// input once (12 or 1 bytes per particle) and are bound by that read and the
// launch: persistent blocks, four particles per thread and step (the
// arrays are separate allocations and p % 4 == 0, so the 16- and 4-byte
// loads are aligned), one partial per block. The last block sums the
// partials, one warp per value, lanes striding the blocks and a fixed
// butterfly, so the sums are the same on every call, and writes them where the
// host reads them. A single thread adding one partial per 256 particles took
// 562 us of the 576 of a call at 1.86M particles; a second kernel and a copy
// back, 29 us a call; this, 18.
constexpr int kReduceBlocks = 148 * 2, kReduceThreads = 512;
__global__ void __launch_bounds__(kReduceThreads) k_particle_reduce(PartsDev P, int mode, double mp, double* __restrict__ partials,
                                                         unsigned* ticket, double* __restrict__ out) {
  __shared__ double s0[kReduceThreads / 32], s1[kReduceThreads / 32], s2[kReduceThreads / 32];
  double a = 0, b = 0, c = 0;
  auto energy = [&](float x, float y, float z) {
    const double vx = x, vy = y, vz = z;
    a += 0.5 * mp * (vx * vx + vy * vy + vz * vz);
  };
  auto count = [&](int f) {
    if (f == 0 || f == 1 || f == 4) a += 1; else if (f == 5) b += 1; else if (f == 2 || f == 3) c += 1;
  };
  const int n4 = P.nP >> 2, stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int t = t0; t < n4; t += stride) {
    if (mode == 0) {
      const float4 x = reinterpret_cast<const float4*>(P.pvx)[t], y = reinterpret_cast<const float4*>(P.pvy)[t];
      const float4 z = reinterpret_cast<const float4*>(P.pvz)[t];
      energy(x.x, y.x, z.x); energy(x.y, y.y, z.y); energy(x.z, y.z, z.z); energy(x.w, y.w, z.w);
    } else {
      const uchar4 f = reinterpret_cast<const uchar4*>(P.pflag)[t];
      count(f.x); count(f.y); count(f.z); count(f.w);
    }
  }
  for (int p = (n4 << 2) + t0; p < P.nP; p += stride) {
    if (mode == 0) energy(P.pvx[p], P.pvy[p], P.pvz[p]);
    else count(P.pflag[p]);
  }
  a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { s0[wid] = a; s1[wid] = b; s2[wid] = c; }
  __syncthreads();
  if (threadIdx.x < 3) {
    const double* w = threadIdx.x == 0 ? s0 : threadIdx.x == 1 ? s1 : s2;
    double t = 0;
    for (int k = 0; k < kReduceThreads / 32; k++) t += w[k];
    partials[3 * blockIdx.x + threadIdx.x] = t;
  }
  if (!last_block(ticket, gridDim.x) || wid >= 3) return;
  double v = 0;                                              // one warp per value
  for (int i = lane; i < (int)gridDim.x; i += 32) v += __ldcg(partials + 3 * i + wid);
  v = warp_sum(v);
  if (lane == 0) out[wid] = v;
}
void launch_particle_reduce(const PartsDev& P, int mode, double mp, double* partials, unsigned* ticket, double* out, cudaStream_t s) {
  // one partial per 256 particles at most: the caller's buffer holds three per 256 of capacity
  const int nb = (int)std::min<long long>(grid_for(P.nP > 0 ? P.nP : 1, kReduceThreads), kReduceBlocks);
  k_particle_reduce<<<nb, kReduceThreads, 0, s>>>(P, mode, mp, partials, ticket, out);
}

// ------------------------------------------------------------ subsurface currents
// js/solver.js:3624-3782. The curl of a drifting sum-of-sines vector
// potential on a lattice of stride 4 cells (float storage), then a capped
// relaxation of deep fluid particles toward its tangential part. The nine
// waves come from the reference's fixed seeded LCG (host, CurrWaves).
__global__ void k_curr_field(CurrField F, double t, double ampl) {
  long long gi = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long gN = (long long)F.gnx * F.gny * F.gnz;
  if (gi >= gN) return;
  const int ii = (int)(gi % F.gnx), jj = (int)((gi / F.gnx) % F.gny), kk = (int)(gi / ((long long)F.gnx * F.gny));
  const double wx2 = ii * F.sx, wy2 = jj * F.sx, wz2 = kk * F.sx;
  double ux = 0, uy = 0, uz = 0;
  for (int o = 0; o < 3; o++) {
    const double* w0 = F.w + (o * 3 + 0) * 5;
    const double* w1 = F.w + (o * 3 + 1) * 5;
    const double* w2 = F.w + (o * 3 + 2) * 5;
    const double dph = F.drift[o] * t;
    const double thx = w0[0] * wx2 + w0[1] * wy2 + w0[2] * wz2 + dph + w0[4];
    const double thy = w1[0] * wx2 + w1[1] * wy2 + w1[2] * wz2 + dph + w1[4];
    const double thz = w2[0] * wx2 + w2[1] * wy2 + w2[2] * wz2 + dph + w2[4];
    ux += w2[3] * w2[1] * cos(thz) - w1[3] * w1[2] * cos(thy);
    uy += w0[3] * w0[2] * cos(thx) - w2[3] * w2[0] * cos(thz);
    uz += w1[3] * w1[0] * cos(thy) - w0[3] * w0[1] * cos(thx);
  }
  F.cfx[gi] = (float)(ux * ampl); F.cfy[gi] = (float)(uy * ampl); F.cfz[gi] = (float)(uz * ampl);
}
__global__ void k_currents(Dims d, PartsDev P, CurrField F, double oceanR, double shell, double relax, int kmax) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP || P.pflag[p] != 0) return;
  const double dvCap = 0.15, invS = 1 / F.sx;
  double rx = P.px[p] - d.cx, ry = P.py[p] - d.cy, rz = P.pz[p] - d.cz;
  double rl = sqrt(rx * rx + ry * ry + rz * rz); if (rl == 0) rl = 1e-9;
  const double dpt = (oceanR - rl) / shell;
  double wgt = (dpt - 0.06) * 4.0;
  if (wgt <= 0) return;
  if (wgt > 1) wgt = 1;
  const double qa = P.px[p] * invS, qb = P.py[p] * invS, qc = P.pz[p] * invS;
  int i0 = jtrunc(qa), j0 = jtrunc(qb), k0 = jtrunc(qc);
  if (i0 > F.gnx - 2) i0 = F.gnx - 2; else if (i0 < 0) i0 = 0;
  if (j0 > F.gny - 2) j0 = F.gny - 2; else if (j0 < 0) j0 = 0;
  if (k0 > kmax) k0 = kmax; else if (k0 < 0) k0 = 0;
  double ta = qa - i0; if (ta > 1) ta = 1; else if (ta < 0) ta = 0;
  double tb = qb - j0; if (tb > 1) tb = 1; else if (tb < 0) tb = 0;
  double tc = qc - k0; if (tc > 1) tc = 1; else if (tc < 0) tc = 0;
  const long long gnx = F.gnx, gxy = (long long)F.gnx * F.gny, g = (k0 * (long long)F.gny + j0) * gnx + i0;
  const double a0 = 1 - ta, a1 = ta, b0 = 1 - tb, b1 = tb, c0 = 1 - tc, c1 = tc;
  auto samp = [&](const float* f) -> double {
    return ((double)f[g] * a0 + (double)f[g + 1] * a1) * b0 * c0 + ((double)f[g + gnx] * a0 + (double)f[g + gnx + 1] * a1) * b1 * c0 +
           ((double)f[g + gxy] * a0 + (double)f[g + gxy + 1] * a1) * b0 * c1 +
           ((double)f[g + gxy + gnx] * a0 + (double)f[g + gxy + gnx + 1] * a1) * b1 * c1;
  };
  const double Ux = samp(F.cfx), Uy = samp(F.cfy), Uz = samp(F.cfz);
  const double ir = 1 / rl;
  const double Ur = (Ux * rx + Uy * ry + Uz * rz) * ir;
  const double Tx = (Ux - rx * ir * Ur) * wgt, Ty = (Uy - ry * ir * Ur) * wgt, Tz = (Uz - rz * ir * Ur) * wgt;
  const double vr = ((double)P.pvx[p] * rx + (double)P.pvy[p] * ry + (double)P.pvz[p] * rz) * ir;
  const double vx = P.pvx[p] - rx * ir * vr, vy = P.pvy[p] - ry * ir * vr, vz = P.pvz[p] - rz * ir * vr;
  double ex = relax * (Tx - vx), ey = relax * (Ty - vy), ez = relax * (Tz - vz);
  const double e2 = ex * ex + ey * ey + ez * ez;
  if (e2 > dvCap * dvCap) { const double es = dvCap / sqrt(e2); ex *= es; ey *= es; ez *= es; }
  P.pvx[p] = (float)(P.pvx[p] + ex); P.pvy[p] = (float)(P.pvy[p] + ey); P.pvz[p] = (float)(P.pvz[p] + ez);
}
void launch_currents(const Dims& d, const PartsDev& P, const CurrField& F, double simTime, double strength,
                     double oceanR, double coreR, double dt, cudaStream_t s) {
  const double shell = oceanR - coreR;
  if (!(strength > 0) || !(shell > 0)) return;
  const long long gN = (long long)F.gnx * F.gny * F.gnz;
  k_curr_field<<<grid_for(gN, 256), 256, 0, s>>>(F, simTime, strength * 2);
  double relax = 2.2 * dt; if (relax > 0.35) relax = 0.35;
  if (P.nP > 0) k_currents<<<grid_for(P.nP, 256), 256, 0, s>>>(d, P, F, oceanR, shell, relax, d.nz / 4);
}

// ---------------------------------------------------------------- metaballs
// Metaballs.build's kernel field (js/surface.js:248-283): every liquid
// particle adds (1 - d^2/R^2)^2 to the corners of the (m+1)^3 lattice within
// R (stencil +-rad around the rounded lattice position, clamped to the
// lattice). The reference sums in Float32 in particle order; here each corner
// accumulates in FP64 (any order) and is rounded to float once, so the field
// is deterministic and within the reference's own float rounding of it.
__device__ __forceinline__ double js_round(double x) { double r = floor(x); return (x - r >= 0.5) ? r + 1 : r; }
// One thread per particle over the lattice points within R along each axis (2
// to 3 of the stencil's 2 rad + 1), each tested exactly; distances along an
// axis step by one, exact in double for positions on the lattice. Bound by the
// reductions since: 135 us for 1.86M particles at 128^3 over the whole stencil
// with a division per point, 82 with a product, now 46 (48^3, 60k: 11.9, 5.3).
// Summing two or four neighbours' shares in registers first: 159 and 294 us
// (instructions).
__global__ void __launch_bounds__(256) k_mb_splat(PartsDev P, int m, double mdx, double rmdx, int pow2, double R, double R2, double iR2,
                                                  int rad, double* __restrict__ acc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.nP || P.pflag[p] != 0) return;
  const double X = P.px[p], Y = P.py[p], Z = P.pz[p];
  const double gx = pow2 ? X * rmdx : X / mdx, gy = pow2 ? Y * rmdx : Y / mdx, gz = pow2 ? Z * rmdx : Z / mdx;
  // outside (-8, m + 8) (or NaN) the reference's clamped ranges are empty
  if (!(gx > -8 && gx < m + 8 && gy > -8 && gy < m + 8 && gz > -8 && gz < m + 8)) return;
  const int i0 = (int)js_round(gx), j0 = (int)js_round(gy), k0 = (int)js_round(gz);
  const int ia = max(max(i0 - rad, (int)ceil(gx - R)), 0), ib = min(min(i0 + rad, (int)floor(gx + R)), m);
  const int ja = max(max(j0 - rad, (int)ceil(gy - R)), 0), jb = min(min(j0 + rad, (int)floor(gy + R)), m);
  const int ka = max(max(k0 - rad, (int)ceil(gz - R)), 0), kb = min(min(k0 + rad, (int)floor(gz + R)), m);
  const unsigned sj = (unsigned)m + 1u;
  const double ex0 = ia - gx, ey0 = ja - gy;
  double ez = ka - gz;
  double* plane = acc + (unsigned long long)((unsigned)ka * sj + (unsigned)ja) * sj + (unsigned)ia;
  for (int k = ka; k <= kb; k++, ez += 1.0, plane += (unsigned long long)sj * sj) {
    const double dz2 = ez * ez;
    double ey = ey0;
    double* row = plane;
    for (int j = ja; j <= jb; j++, ey += 1.0, row += sj) {
      const double dy2 = dz2 + ey * ey;
      if (dy2 >= R2) continue;
      double ex = ex0;
      for (int i = ia; i <= ib; i++, ex += 1.0) {
        const double d2 = dy2 + ex * ex;
        if (d2 >= R2) continue;
        const double u = 1 - d2 * iR2;
        atomicAdd(row + (i - ia), u * u);
      }
    }
  }
}
__global__ void k_mb_round(const double* __restrict__ acc, float* __restrict__ field, long long n, const int* __restrict__ err) {
  const bool keep = *err != 0;                             // a latched fault leaves the last field
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
    { const float v = (float)acc[c]; if (!keep) field[c] = v; }
}
void launch_metaball_field(const PartsDev& P, int m, double mdx, double R2, int rad, double* acc, float* field,
                           const int* err, cudaStream_t s) {
  const long long corners = (long long)(m + 1) * (m + 1) * (m + 1);
  cudaMemsetAsync(acc, 0, sizeof(double) * (size_t)corners, s);
  // the bound along an axis a little wide: the exact test is on the squares
  if (P.nP > 0)
    k_mb_splat<<<grid_for(P.nP, 256), 256, 0, s>>>(P, m, mdx, 1.0 / mdx, is_pow2(mdx) ? 1 : 0, std::sqrt(R2) * (1 + 1e-12), R2,
                                                   1.0 / R2, rad, acc);
  k_mb_round<<<(int)std::min<long long>(grid_for(corners, 256), 148 * 16), 256, 0, s>>>(acc, field, corners, err);
}
