// ws_sor_tb.cu — the pressure solve of _pressureSolve (js/solver.js:1368-1404)
// on every SM at once: red-black SOR over shared-memory regions.
//
// Partition. The grid is cut into 4x4x4-cell bricks; the pressure setup
// leaves one 64-bit mask of interior fluid cells per brick. Bricks holding a
// fluid cell are taken in Morton order and split into one contiguous chunk
// per CTA with equal shares of weight (fluid cells plus kBrickWeight per
// brick), so each CTA owns a compact patch of the ocean shell.
//
// Region. A CTA works on the fluid cells of its owned bricks (d = 0) and on
// those of the surrounding bricks by their L1 distance d in cells to the
// owned bricks' boxes. d changes by at most one between neighbouring cells
// and a red-black half-sweep moves information one cell, so after loading
// exact values for d <= H the CTA can run H half-sweeps (H / 2 iterations) on
// its own: half-sweep t updates the cells with d <= H - t, and after the last
// one the owned cells hold exactly the values of the global sweep. Each
// update reads the same six neighbours in the same order with the same
// arithmetic as the reference's sweep (sor_update), so the iterates are
// bitwise those of the plain red-black solve. H is 4 where every CTA's region
// fits shared memory with it, else 2: a larger H halves the exchanges, and
// costs the cells of two more layers.
//
// Storage. Only fluid cells are stored, colour by colour and by d inside a
// colour (colour 0 d = 0 .. H - 1, then colour 1 d = 0 .. H): a half-sweep
// updates a prefix of its colour, an update entry's own q has the entry's
// index, and neighbours of neighbouring entries sit mostly in neighbouring
// banks. A cell's index is its brick's base in its (colour, d) class plus the
// set bits below it in the class mask. An entry is one 16-byte record (the
// byte offsets of its six neighbours, 16 bits each, the right-hand side, and
// the stencil count in the offsets' unused low bits; omega / count comes from a
// table), a cell 4 bytes: about 10,000 entries fit one SM, 1.3M fluid cells of
// a thin ocean the chip. (Before, q was dense over the region's bricks with 24
// bytes an entry; that held 4096 entries, and grids above 160^3 read lists
// from L2 in every half-sweep.)
//
// Exchange. After each epoch of H half-sweeps a CTA writes the owned cells
// that some other CTA's halo holds into its own packed list (two of them, by
// epoch parity) as 64-bit words (q's bits | tag << 32), one single-copy-atomic
// relaxed store per cell and no fence or flag; before the next epoch every
// thread loads its halo words and polls a word again until its tag is the
// epoch's. The tag travels in the same word as the value, so a matching tag
// proves the value, and a CTA waits only for the values it needs. The lists
// are in brick order on both sides, so a warp's words share sectors: words
// scattered over a grid-sized array took half of the solve in L2 traffic and
// polls. Double buffering makes the write of epoch e + 2 safe against
// neighbours still reading epoch e: a CTA computes epoch e + 2 only after
// reading its neighbours' epoch e + 1 words, which each neighbour wrote after
// it had read this CTA's epoch e words. That needs every reader of a CTA to be
// read by it, and cells alone do not give it (a CTA may hold a cell near a
// foreign brick whose own fluid lies beyond the halo). So a list begins with
// one word that stands for the CTA, and a CTA fetches that word of every owner
// of an active brick around its own; brick adjacency is symmetric.
// Tags count on from solve to solve (tagBase; after a timed-out wait past the
// epochs that any CTA can have run, ws_sor_tags.h), so a word left by an earlier
// solve never matches and nothing has to be cleared.
//
// Overlap. Colour 0's owned cells are stored with those first that touch no
// foreign brick: their part of an epoch's first half-sweep reads no halo, so
// it runs between the publication and the wait.
//
// Residual check. Every sorCheckEvery iterations (epochs end on check
// iterations) the FP64 partial ||b - A q||^2 and ||b||^2 of the owned cells
// is published, all CTAs wait for all partials (a counter) and sum them in
// CTA order, so every CTA takes the same stop decision. Partials alternate
// between two buffers so a CTA running ahead cannot overwrite one that a
// slower CTA still sums.
//
// The plan (brick weights, Morton scan, chunks, regions) is built inside the
// same cooperative launch, separated by three grid barriers. When some
// region does not fit even with H = 2, or a fluid cell lies on the domain's
// outermost layer (only by a caller's upload), every CTA leaves the solve to
// a fallback: grids up to 160^3 sweep the owned bricks in global memory with
// a grid barrier per half-sweep, larger ones leave the solved flag clear for
// the list kernels that follow (ws_sor.cu). Same arithmetic, same iterates.
//
// What bounds it and what it measured stands at k_sor_tb.
//
// Every wait is bounded: after kTbSpinLimit polls the CTA latches
// WS_DERR_TIMEOUT, stops, and the waits of the others run out in turn. The
// cooperative launch guarantees that all CTAs are resident, so a healthy
// run never reaches the limit.
#include "ws_kernels.cuh"
#include "ws_sor_tags.h"
#include <algorithm>
#include <cstddef>

namespace {

typedef unsigned long long u64;

constexpr int kTbThreads = 1024;
constexpr int kRbMax = 896;                 // region bricks per CTA
constexpr int kHMax = 4;                    // half-sweeps per epoch where the regions fit
constexpr int kHashSlots = 2048;            // open-addressing table of region bricks
constexpr int kQMax = 16384;                // stored cells per CTA (the neighbour indices hold 16 bits)
constexpr int kPubMax = 8192;               // published words per CTA
constexpr int kFetchMax = 8192;             // fetched words per CTA
constexpr long long kTbSpinLimit = 4000000LL;
constexpr int kMaxCtas = 1024;
constexpr int kTbSmem = 229376;             // dynamic shared memory: the 227 KB of a block less the static part
// Chunk weight of an active brick: its interior fluid cells plus this much.
// Equal shares of fluid alone gave CTAs 13-55 owned bricks at 128^3 (bricks
// at the shell's edges hold few fluid cells), and the CTA with the most
// bricks has the largest region, which every other CTA waits for at the end
// of the plan; the per-brick term evens out the brick counts too.
constexpr int kBrickWeight = 16;

// device control block; all but tagBase zeroed before every solve
struct TbCtl {
  unsigned barCount;             // arrivals at the grid barriers of this solve
  unsigned resCount;             // residual partials published so far (all checks)
  int over4, over2;              // some region does not fit with H = 4, with H = 2
  int solved;                    // 1: this launch solved the system (the list kernels leave at once)
  int pad[11];
  unsigned tagBase;              // exchange tags of this solve start after it
};

// What one CTA can hold on this grid (tb_caps); the plan checks its counts
// against them, so a list never outgrows its place.
struct TbCaps { int own, pub, fetch, rows; };

struct TbArgs {
  Dims d;
  float* q;
  u64* xq;                       // exchange: per CTA two lists of caps.pub words (q bits | tag << 32)
  unsigned* xmap;                // [2][nCells]: place of a published cell (owner * 2 * caps.pub + position), H = 2 and 4
  const float* rhs;
  const float* pw;               // omega/diag, negative off the fluid
  const uint8_t* diag8;
  const u64* fmask;              // per linear brick: its interior fluid cells (bit 16 z + 4 y + x)
  const DevStatus* st;           // the setup's omega and odd-fluid flag
  int nbx, nby, nbz, mbits;      // bricks per axis; Morton cube side 2^mbits
  int2* cntPart;                 // per CTA: (active bricks, chunk weight) of its Morton chunk
  int* actLin;                   // active brick t -> linear brick index
  int* wPre;                     // linear (active) brick -> chunk weight before it
  int* chunkStart;               // CTA -> first owned active brick ([P] = number of active bricks)
  TbCaps caps;
  unsigned* glist;               // per CTA: global cell of each owned cell, colour 0 first (caps.own)
  unsigned short* dense;         // per CTA: stored index of each region cell (64 caps.rows), where shared memory has no room
  unsigned short* plist;         // per CTA: stored index of each published cell (caps.pub)
  uint2* flist;                  // per CTA: (place in xq, stored index) of each halo cell (caps.fetch)
  double2* resPart;              // 2 x P residual partials
  TbCtl* ctl;
  double om1;
  int iters, check, listFallback;
  int regionPath;                // the path number that the solve in shared memory reports
  double tol;
  int* err;
  int* outIters;
  double* outRel;
  int* outPath;
};

// Plan-time tables in shared memory. The first lie where the solve's values
// and records go: they are read for the last time when the dense index table
// is filled. The second lie at the end of the block's shared memory, the dense
// table before them where it clears both the first tables and the records,
// else in global memory.
struct TbPlan {
  u64 mask[kRbMax];                       // interior fluid cells of each region brick
  u64 cm[kHMax][kRbMax];                  // halo brick: its cells at d = 1 .. 4; owned brick: [0], [1] its cells to publish
                                          // with H = 2, 4, [2] its cells with a foreign face neighbour
  int hkey[kHashSlots];
  short hval[kHashSlots];
  unsigned dirs[kRbMax];                  // halo brick: which of the 27 bricks around it this CTA owns; owned: which are foreign
  // bases of a brick's cells in the lists. Owned: [0] colour 0 without, [4] with
  // a foreign face neighbour, [1] colour 1, [2], [3] published cells; halo:
  // [2 (d - 1) + colour], [8], [9] fetched cells with H = 2, 4
  unsigned short base[2 * kHMax + 2][kRbMax];
};
struct TbPlan2 {
  uchar4 rbXYZ[kRbMax];                   // brick coordinates
  unsigned short rbNb[6][kRbMax];         // face neighbours' slots (kNone: not in the region)
};
constexpr unsigned short kNone = 0xffffu;
static_assert(kMaxCtas <= kTbThreads, "one thread per CTA builds the list of neighbours");
static_assert(sizeof(TbPlan) + sizeof(TbPlan2) <= (size_t)kTbSmem, "plan tables");

// bits of the cells with x + y + z odd
constexpr u64 kOdd = 0xa5a55a5aa5a55a5aull;
// cells of a brick within L1 distance d of the box of the brick in direction
// n27 = (ox + 1) + 3 (oy + 1) + 9 (oz + 1)
constexpr int axis_dist(int o, int c) { return o < 0 ? c + 1 : o > 0 ? 4 - c : 0; }
struct NearTable { u64 m[27][kHMax]; };
constexpr NearTable make_near() {
  NearTable t{};
  for (int n = 0; n < 27; n++)
    for (int c = 0; c < 64; c++) {
      const int dd = axis_dist(n % 3 - 1, c & 3) + axis_dist((n / 3) % 3 - 1, (c >> 2) & 3) + axis_dist(n / 9 - 1, c >> 4);
      for (int d = 1; d <= kHMax; d++)
        if (dd <= d) t.m[n][d - 1] |= 1ull << c;
    }
  return t;
}
__device__ const NearTable kNear = make_near();

__device__ __forceinline__ unsigned compact1by2(unsigned x) {
  x &= 0x09249249u;
  x = (x ^ (x >> 2)) & 0x030c30c3u;
  x = (x ^ (x >> 4)) & 0x0300f00fu;
  x = (x ^ (x >> 8)) & 0xff0000ffu;
  x = (x ^ (x >> 16)) & 0x000003ffu;
  return x;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

// Bounded grid barrier number n (counted from 1) on the arrivals of this
// solve: one reduction to arrive and a poll until all have. (An arrival that
// read the count back and a last CTA that reset it and raised a generation
// word took three round trips to L2 in a row, about 2 us more.) false when a
// wait timed out.
__device__ bool tb_grid_barrier(TbCtl* ctl, unsigned n, int* err, int* sAbort) {
  __syncthreads();
  if (threadIdx.x == 0) {
    fence_acq_rel_gpu();
    atomicAdd(&ctl->barCount, 1u);
    if (!bounded_wait_geq(&ctl->barCount, n * gridDim.x, kTbSpinLimit, err)) *sAbort = 1;
    fence_acq_rel_gpu();
    if (*(volatile int*)err & WS_DERR_TIMEOUT) *sAbort = 1;
  }
  __syncthreads();
  return *(volatile int*)sAbort == 0;
}

// the CTA that owns an active brick with chunk weight `wpre` before
// it in Morton order (NF: the total weight)
__device__ __forceinline__ int owner_of(long long wpre, int P, long long NF) {
  if (NF <= 0) return 0;
  long long o = wpre * P / NF;
  return (int)(o < P - 1 ? o : P - 1);
}
__device__ __forceinline__ bool interior(const Dims& d, int i, int j, int k) {
  return i >= 1 && j >= 1 && k >= 1 && i + 2 <= d.nx && j + 2 <= d.ny && k + 2 <= d.nz;
}
// linear brick of Morton code m, -1 outside the grid
__device__ __forceinline__ int morton_brick(const TbArgs& a, long long m) {
  const int bx = (int)compact1by2((unsigned)m), by = (int)compact1by2((unsigned)(m >> 1)), bz = (int)compact1by2((unsigned)(m >> 2));
  return bx < a.nbx && by < a.nby && bz < a.nbz ? (bz * a.nby + by) * a.nbx + bx : -1;
}

__device__ __forceinline__ bool hash_insert(TbPlan& S, TbPlan2& S2, int key, u64 mask, int* nRegion, int* sOverflow, int fixedSlot,
                                            int nbx, int nby) {
  unsigned h = ((unsigned)key * 2654435761u) >> 21;          // 11 bits
  for (int probe = 0; probe < kHashSlots; probe++, h = (h + 1) & (kHashSlots - 1)) {
    int prev = atomicCAS(&S.hkey[h], -1, key);
    if (prev == -1) {
      int slot = fixedSlot >= 0 ? fixedSlot : atomicAdd(nRegion, 1);
      S.hval[h] = (short)(slot < kRbMax ? slot : -1);
      if (slot < kRbMax) {
        const int t = key / nbx;
        S.mask[slot] = mask; S.dirs[slot] = 0u;
        S2.rbXYZ[slot] = make_uchar4((unsigned char)(key - t * nbx), (unsigned char)(t % nby), (unsigned char)(t / nby), 0);
      }
      else *sOverflow = 1;
      return true;
    }
    if (prev == key) return false;
  }
  *sOverflow = 1;
  return false;
}
__device__ __forceinline__ int hash_find(const TbPlan& S, int key) {
  unsigned h = ((unsigned)key * 2654435761u) >> 21;
  for (int probe = 0; probe < kHashSlots; probe++, h = (h + 1) & (kHashSlots - 1)) {
    int k = S.hkey[h];
    if (k == key) return S.hval[h];
    if (k == -1) return -1;
  }
  return -1;
}
// slot of the brick (ox, oy, oz) bricks away from slot s, -1 when not in the region
__device__ __forceinline__ int slot_at(const TbArgs& a, const TbPlan& S, const TbPlan2& S2, int s, int ox, int oy, int oz) {
  const uchar4 b = S2.rbXYZ[s];
  const int x = (int)b.x + ox, y = (int)b.y + oy, z = (int)b.z + oz;
  if (x < 0 || y < 0 || z < 0 || x >= a.nbx || y >= a.nby || z >= a.nbz) return -1;
  return hash_find(S, (z * a.nby + y) * a.nbx + x);
}
__device__ __forceinline__ unsigned cell_global(const TbArgs& a, const TbPlan2& S, int s, int c) {
  const uchar4 b = S.rbXYZ[s];
  const unsigned i = b.x * 4u + (c & 3), j = b.y * 4u + ((c >> 2) & 3), k = b.z * 4u + (c >> 4);
  return (k * (unsigned)a.d.ny + j) * (unsigned)a.d.nx + i;
}
__device__ __forceinline__ int bits_below(u64 m, int c) { return __popcll(m & ((1ull << c) - 1ull)); }

// block-wide exclusive scan of two ints (1024 threads); totals returned
__device__ __forceinline__ int2 block_scan2(int a, int b, int2& total, int2* sw) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int xa = a, xb = b;
  for (int o = 1; o < 32; o <<= 1) {
    int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
    if (lane >= o) { xa += ya; xb += yb; }
  }
  if (lane == 31) sw[wid] = make_int2(xa, xb);
  __syncthreads();
  if (wid == 0) {
    int2 v = lane < (int)(blockDim.x >> 5) ? sw[lane] : make_int2(0, 0);
    int ca = v.x, cb = v.y;
    for (int o = 1; o < 32; o <<= 1) {
      int ya = __shfl_up_sync(0xffffffffu, ca, o), yb = __shfl_up_sync(0xffffffffu, cb, o);
      if (lane >= o) { ca += ya; cb += yb; }
    }
    sw[lane] = make_int2(ca - v.x, cb - v.y);            // exclusive warp offsets
    if (lane == 31) sw[32] = make_int2(ca, cb);
  }
  __syncthreads();
  int2 base = sw[wid];
  total = sw[32];
  int2 r = make_int2(base.x + xa - a, base.y + xb - b);
  __syncthreads();                                         // sw reusable
  return r;
}

// one cell update of the reference's sweep (js/solver.js:1397-1404; sor_update)
__device__ __forceinline__ float relax(float qc, float pw, float rhs, const float* v, double om1) {
  return sor_update(qc, pw, rhs, v[0], v[1], v[2], v[3], v[4], v[5], om1);
}

// publish this CTA's partial for check number k, wait for all, sum in a
// fixed order (lane l adds partials l, l + 32, ..., then a fixed butterfly);
// every CTA gets the same value. false when the wait timed out.
__device__ bool global_residual(const TbArgs& a, double2 part, int k, double* sRel, int* sAbort) {
  const int P = gridDim.x;
  double2* buf = a.resPart + (size_t)(k & 1) * P;
  if (threadIdx.x == 0) {
    __stcg(&buf[blockIdx.x], part);
    fence_acq_rel_gpu();
    atomicAdd(&a.ctl->resCount, 1u);
    if (!bounded_wait_geq(&a.ctl->resCount, (unsigned)P * (unsigned)(k + 1), kTbSpinLimit, a.err)) *sAbort = 1;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double rr = 0, bb = 0;
    if (!*(volatile int*)sAbort)
      for (int b = threadIdx.x; b < P; b += 32) { const double2 v = __ldcg(&buf[b]); rr += v.x; bb += v.y; }
    for (int o = 16; o > 0; o >>= 1) {
      rr += __shfl_xor_sync(0xffffffffu, rr, o);
      bb += __shfl_xor_sync(0xffffffffu, bb, o);
    }
    if (threadIdx.x == 0) *sRel = bb > 0 ? sqrt(rr) / sqrt(bb) : sqrt(rr);
  }
  __syncthreads();
  return *(volatile int*)sAbort == 0;
}

// Offsets of the (colour, d) classes for epochs of H half-sweeps: colour 0
// stores d = 0 .. H - 1 (all of them update entries), colour 1 d = 0 .. H (the
// entries d <= H - 2 first).
struct TbLayout {
  int H, NE, NQ, c1;             // entries, stored cells, first cell of colour 1
  int off[2][kHMax + 1];         // first cell of a class
  int n[2][kHMax + 1];           // its cells
  int nA;                        // colour 0, d = 0: cells without a foreign face neighbour (stored first)
  int cum[2][kHMax];             // cells of a colour with d <= index
  int pub, fetch;                // words published and fetched: the cells and the CTAs' own words
};
// bytes of the solve's values and records: the cells, the zero cell and one that takes the CTAs' own words, then the entries
__host__ __device__ __forceinline__ int record_at(int NQ) { return (4 * (NQ + 2) + 15) & ~15; }
// where a region of R bricks has its dense index table in shared memory: before
// the second tables, clear of the first and of the records; -1 without room
__host__ __device__ __forceinline__ int dense_at(int R, int NQ, int NE) {
  const int at = (kTbSmem - (int)sizeof(TbPlan2)) / 16 * 16 - R * 128;
  return at >= (int)sizeof(TbPlan) && at >= record_at(NQ) + 16 * NE ? at : -1;
}
// whether the solve's values and records fit with epochs of H half-sweeps
__device__ __forceinline__ bool make_layout(TbLayout& L, const TbCaps& c, int R, int H, int pub, int fetch) {
  L.H = H; L.pub = pub; L.fetch = fetch;
  int at = 0;
  for (int d = 0; d < H; d++) { L.off[0][d] = at; at += L.n[0][d]; }
  L.c1 = at;
  for (int d = 0; d <= H; d++) {
    if (d == H - 1) L.NE = at;
    L.off[1][d] = at; at += L.n[1][d];
  }
  L.NQ = at;
  for (int col = 0; col < 2; col++) {
    int sum = 0;
    for (int d = 0; d < kHMax; d++) { sum += L.n[col][d]; L.cum[col][d] = sum; }
  }
  return L.NQ < kQMax && pub <= c.pub && fetch <= c.fetch && L.n[0][0] + L.n[1][0] <= c.own &&
         record_at(L.NQ) + 16 * L.NE <= (kTbSmem - (int)sizeof(TbPlan2)) / 16 * 16 &&
         (R <= c.rows || dense_at(R, L.NQ, L.NE) >= 0);
}

}  // namespace

extern __shared__ __align__(16) unsigned char tb_smem_raw[];

// The whole solve in one cooperative launch of one 1024-thread CTA per SM.
//
// What bounds it: not bytes (DRAM under 1%), but latency and shared memory.
// A half-sweep costs about 600 cycles whatever its length (record, gathers,
// FP64 chain, store, barrier) plus about 28 cycles per 32 entries of an SM
// (4 wavefronts of the record, six gathers at 1.8 ways, FP64 conversions); an
// exchange about 1.2 us, partly behind the first half-sweep. 1024 threads with
// two entries each in flight: 512 with four were a third slower. Measured
// (fixed-iteration fits, before -> now, us): 32^3 (2.9k fluid cells) plan
// 32 -> 30, iteration 1.36 -> 1.14; 97^3 (75k) 67 -> 52, 4.05 -> 1.69; 128^3
// (160k) 65 -> 55, 4.17 -> 2.13; 256^3 (1.09M, lists before) 143 -> 144,
// 17.6 -> 5.9. A residual check costs 18 us more at 256^3 (the reload before
// it overlaps nothing, and the pass); posted and collected an epoch later, with
// the judged state stored meanwhile, a solve took 1612 instead of 1527 us.
__global__ void __launch_bounds__(kTbThreads, 1) k_sor_tb(TbArgs a) {
  __shared__ int sAbort, sOverflow, nRegion, sT0, sT1, sA;
  __shared__ TbLayout sL;
  __shared__ int sCnt[16];
  __shared__ unsigned sOwn[kMaxCtas / 32];             // the CTAs that own active bricks around this one's
  __shared__ float sPw[8];
  __shared__ int2 sScan[33];
  __shared__ double2 sRed[32];
  __shared__ double sRel;
  __shared__ long long sNF;
  const int P = gridDim.x, p = blockIdx.x, tid = threadIdx.x, T = kTbThreads;
  const int lane = tid & 31, warp = tid >> 5;
  const Dims& d = a.d;
  int it = 0, path = a.regionPath;
  unsigned epoch = 0, nBar = 0;
  double rel = -1;
  bool solved = false;
  const unsigned tag0 = *(volatile const unsigned*)&a.ctl->tagBase;
  if (tid == 0) { sAbort = 0; sOverflow = 0; nRegion = 0; }
  if (tid < 8) sPw[tid] = tid ? (float)(a.st->sorOmega / (double)tid) : 0.f;   // as the setup rounds pw
  __syncthreads();

  // ---- phase 0: weight of a chunk of Morton codes per CTA
  const long long MC = 1LL << (3 * a.mbits);
  const long long per = (MC + P - 1) / P;
  const long long c0 = std::min(MC, (long long)p * per), c1 = std::min(MC, c0 + per);
  if (p == 0) {
    for (int q = tid; q <= P; q += T) a.chunkStart[q] = q == 0 ? 0 : 0x7fffffff;
  }
  {
    int actSum = 0, wSum = 0;
    for (long long m = c0 + tid; m < c1; m += T) {
      const int lin = morton_brick(a, m);
      const int cnt = lin >= 0 ? __popcll(__ldcg(a.fmask + lin)) : 0;
      if (cnt) { actSum++; wSum += cnt + kBrickWeight; }
    }
    actSum = warp_sum(actSum); wSum = warp_sum(wSum);
    if (lane == 0) sScan[warp] = make_int2(actSum, wSum);
    __syncthreads();
    if (tid < 32) {
      int2 v = sScan[tid];
      v.x = warp_sum(v.x); v.y = warp_sum(v.y);
      if (tid == 0) __stcg(&a.cntPart[p], v);
    }
  }
  if (!tb_grid_barrier(a.ctl, ++nBar, a.err, &sAbort)) goto done;

  // ---- phase 1: this chunk's active bricks in order, the weight before each,
  // and the CTA chunk starts
  {
    if (tid < 32) {
      long long bA = 0, bW = 0, tA = 0, tW = 0;
      for (int b = tid; b < P; b += 32) {
        const int2 v = __ldcg(&a.cntPart[b]);
        if (b < p) { bA += v.x; bW += v.y; }
        tA += v.x; tW += v.y;
      }
      bA = warp_sum(bA); bW = warp_sum(bW); tA = warp_sum(tA); tW = warp_sum(tW);
      if (tid == 0) { sT0 = (int)bA; sT1 = (int)bW; sA = (int)tA; sNF = tW; }
    }
    __syncthreads();
    int baseA = sT0, baseW = sT1;
    const int A = sA;
    const long long NF = sNF;
    for (long long m0 = c0; m0 < c1; m0 += T) {
      const long long m = m0 + tid;
      const int lin = m < c1 ? morton_brick(a, m) : -1;
      const int cnt = lin >= 0 ? __popcll(__ldcg(a.fmask + lin)) : 0;
      const int act = cnt > 0, w = act ? cnt + kBrickWeight : 0;
      int2 tot;
      const int2 ex = block_scan2(act, w, tot, sScan);
      if (act) {
        const int t = baseA + ex.x;
        const long long wpre = baseW + ex.y;
        a.actLin[t] = lin; a.wPre[lin] = (int)wpre;
        // the next active brick starts every CTA q whose first unit of weight
        // (prefix ceil(q NF / P)) lies in (wpre, wpre + w]
        const long long qlo = wpre * P / NF + 1, qhi = std::min((long long)P - 1, (wpre + w) * P / NF);
        for (long long q = qlo; q <= qhi; q++) a.chunkStart[q] = t + 1;
        if (t == A - 1) a.chunkStart[P] = A;
      }
      baseA += tot.x; baseW += tot.y;
    }
  }
  if (!tb_grid_barrier(a.ctl, ++nBar, a.err, &sAbort)) goto done;
  // no interior fluid cell: the reference returns before its first sweep
  // (js/solver.js:1330); every CTA read the same total, so all leave here
  if (sA == 0 && !a.st->oddFluid) { rel = 0; solved = true; goto done; }

  // ---- phase 2: this CTA's region
  {
    TbPlan& S = *reinterpret_cast<TbPlan*>(tb_smem_raw);
    TbPlan2& S2 = *reinterpret_cast<TbPlan2*>(tb_smem_raw + (kTbSmem - sizeof(TbPlan2)) / 16 * 16);
    const int A = sA;
    const long long NF = sNF;
    if (tid == 0) {
      int s0 = __ldcg(&a.chunkStart[p]), s1 = __ldcg(&a.chunkStart[p + 1]);
      if (s0 > A) s0 = A;
      if (s1 > A) s1 = A;
      sT0 = s0; sT1 = s1 > s0 ? s1 : s0;
      nRegion = sT1 - sT0;
      if (nRegion > kRbMax) sOverflow = 1;
    }
    for (int h = tid; h < kHashSlots; h += T) S.hkey[h] = -1;
    if (tid < kMaxCtas / 32) sOwn[tid] = 0u;
    __syncthreads();
    const int t0 = sT0, O = sT1 - sT0;
    if (!sOverflow) {
      for (int s = tid; s < O; s += T) {
        const int lin = __ldcg(&a.actLin[t0 + s]);
        hash_insert(S, S2, lin, __ldcg(a.fmask + lin), &nRegion, &sOverflow, s, a.nbx, a.nby);
      }
      __syncthreads();
      // the active bricks among the owned bricks' 26 neighbours that other CTAs own
      for (int item = tid; item < O * 26; item += T) {
        const int s = item / 26, n26 = item - s * 26, n27 = n26 < 13 ? n26 : n26 + 1;
        const uchar4 b = S2.rbXYZ[s];
        const int x = (int)b.x + n27 % 3 - 1, y = (int)b.y + (n27 / 3) % 3 - 1, z = (int)b.z + n27 / 9 - 1;
        if (x < 0 || y < 0 || z < 0 || x >= a.nbx || y >= a.nby || z >= a.nbz) continue;
        const int lin2 = (z * a.nby + y) * a.nbx + x;
        const u64 m = __ldcg(a.fmask + lin2);
        const int wp = __ldcg(&a.wPre[lin2]);
        const int ow = m ? owner_of(wp, P, NF) : p;
        if (ow == p) continue;
        if (hash_insert(S, S2, lin2, m, &nRegion, &sOverflow, -1, a.nbx, a.nby)) atomicOr(&sOwn[ow >> 5], 1u << (ow & 31));
      }
      __syncthreads();
    }
    if (tid == 0 && nRegion > kRbMax) sOverflow = 1;
    __syncthreads();
    const int R = sOverflow ? 0 : nRegion;
    // halo bricks: which of the bricks around them this CTA owns; owned
    // bricks: which are foreign; and every brick's six face neighbours
    for (int item = tid; item < R * 27; item += T) {
      const int s = item / 27, n27 = item - s * 27, ox = n27 % 3 - 1, oy = (n27 / 3) % 3 - 1, oz = n27 / 9 - 1;
      const int slot = slot_at(a, S, S2, s, ox, oy, oz);
      if (slot >= 0 && (slot < O) != (s < O)) atomicOr(&S.dirs[s], 1u << n27);
      const int dir = n27 == 12 ? 0 : n27 == 14 ? 1 : n27 == 10 ? 2 : n27 == 16 ? 3 : n27 == 4 ? 4 : n27 == 22 ? 5 : -1;
      if (dir >= 0) S2.rbNb[dir][s] = slot >= 0 ? (unsigned short)slot : kNone;
    }
    __syncthreads();
    // class masks: a halo brick's cells at each d; an owned brick's cells
    // that some halo stores with H = 2 and 4 (colour 0 to d = H - 1, 1 to H)
    if (tid < R) {
      const int s = tid;
      u64 le[kHMax] = { 0, 0, 0, 0 };
      for (unsigned m = S.dirs[s]; m; m &= m - 1) {
        const int n27 = __ffs(m) - 1;
#pragma unroll
        for (int q = 0; q < kHMax; q++) le[q] |= kNear.m[n27][q];
      }
      const u64 f = S.mask[s];
      // colour of a brick's cell: 4 divides the brick's origin, so it is the parity of x + y + z inside
      if (s < O) {
        S.cm[0][s] = f & ((le[0] & ~kOdd) | (le[1] & kOdd)); S.cm[1][s] = f & ((le[2] & ~kOdd) | (le[3] & kOdd));
        S.cm[2][s] = f & le[0];
      } else {
#pragma unroll
        for (int q = 0; q < kHMax; q++) S.cm[q][s] = f & le[q] & ~(q ? le[q > 0 ? q - 1 : 0] : 0ull);
      }
    }
    __syncthreads();
    // the cells a halo brick contributes to the fetch list: all it stores
    auto fetched = [&](int s, bool h4) -> u64 {
      const u64 d1 = S.cm[0][s], d2 = d1 | S.cm[1][s];
      if (!h4) return (d1 & ~kOdd) | (d2 & kOdd);
      const u64 d3 = d2 | S.cm[2][s];
      return (d3 & ~kOdd) | ((d3 | S.cm[3][s]) & kOdd);
    };
    // bases: one warp per list scans the bricks' counts
    if (warp < 15) {
      const bool owned = warp < 5;                 // rows 0 .. 4 of the owned bricks, 0 .. 9 of the halo bricks
      const int row = owned ? warp : warp - 5;
      const int lo = owned ? 0 : O, hi = owned ? std::min(O, R) : R;   // none when the region overflowed
      int run = 0;
      for (int s0 = lo; s0 < hi; s0 += 32) {
        const int s = s0 + lane;
        u64 m = 0;
        if (s < hi) {
          if (owned) m = row == 0 ? S.mask[s] & ~S.cm[2][s] & ~kOdd : row == 1 ? S.mask[s] & kOdd
                       : row == 4 ? S.cm[2][s] & ~kOdd : S.cm[row - 2][s];
          else m = row < 8 ? S.cm[row >> 1][s] & (row & 1 ? kOdd : ~kOdd) : fetched(s, row == 9);
        }
        const int v = __popcll(m);
        int x = v;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        if (s < hi) S.base[row][s] = (unsigned short)(run + x - v);
        run += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) sCnt[warp] = run;
    }
    __syncthreads();
    if (tid == 0) {
      int nb = 0;                                  // one word per CTA around this one, and this one's own
      for (int w = 0; w < kMaxCtas / 32; w++) nb += __popc(sOwn[w]);
      sCnt[2]++; sCnt[3]++; sCnt[13] += nb; sCnt[14] += nb;
      sL.nA = sCnt[0];
      sL.n[0][0] = sCnt[0] + sCnt[4]; sL.n[1][0] = sCnt[1];
      for (int q = 0; q < kHMax; q++) { sL.n[0][q + 1] = sCnt[5 + 2 * q]; sL.n[1][q + 1] = sCnt[6 + 2 * q]; }
      const bool no = sOverflow || a.st->oddFluid != 0;
      if (no || !make_layout(sL, a.caps, R, 2, sCnt[2], sCnt[13])) atomicOr(&a.ctl->over2, 1);
      if (no || !make_layout(sL, a.caps, R, 4, sCnt[3], sCnt[14])) atomicOr(&a.ctl->over4, 1);
    }
    // where the other CTAs find this one's cells, for both epoch lengths
    for (int x = tid; x < std::min(O, R) * 64; x += T) {
      const int s = x >> 6, c = x & 63;
#pragma unroll
      for (int w = 0; w < 2; w++) {
        const u64 m = S.cm[w][s];
        if ((m >> c) & 1ull)
          __stcg(a.xmap + (size_t)w * (size_t)d.nCells + cell_global(a, S2, s, c),
                 (unsigned)p * (2u * (unsigned)a.caps.pub) + 1u + (unsigned)(S.base[2 + w][s] + bits_below(m, c)));
      }
    }
    if (!tb_grid_barrier(a.ctl, ++nBar, a.err, &sAbort)) goto done;
    if (tid == 0) {
      const bool over4 = ld_acquire(reinterpret_cast<const unsigned*>(&a.ctl->over4)) != 0;
      const bool over2 = ld_acquire(reinterpret_cast<const unsigned*>(&a.ctl->over2)) != 0;
      sOverflow = over4 && over2;
      if (!sOverflow) make_layout(sL, a.caps, R, over4 ? 2 : 4, sCnt[over4 ? 2 : 3], sCnt[over4 ? 13 : 14]);
    }
    __syncthreads();

    if (sOverflow == 0) {
      const TbLayout& L = sL;
      const int which = L.H == 2 ? 0 : 1;
      uint4* rec = reinterpret_cast<uint4*>(tb_smem_raw + record_at(L.NQ));
      const int room = dense_at(R, L.NQ, L.NE);
      unsigned short* dense = room >= 0 ? reinterpret_cast<unsigned short*>(tb_smem_raw + room)
                                        : a.dense + (size_t)p * 64 * a.caps.rows;
      unsigned* gl = a.glist + (unsigned)p * (unsigned)a.caps.own;
      unsigned short* pl = a.plist + (unsigned)p * (unsigned)a.caps.pub;
      uint2* fl = a.flist + (unsigned)p * (unsigned)a.caps.fetch;
      if (tid == 0) pl[0] = (unsigned short)L.NQ;
      if (tid < P && ((sOwn[tid >> 5] >> (tid & 31)) & 1u)) {
        int at = L.fetch - 1;                      // the list's end: the CTAs' own words
        for (int w = kMaxCtas / 32 - 1; w > (tid >> 5); w--) at -= __popc(sOwn[w]);
        at -= __popc(sOwn[tid >> 5] & ~((2u << (tid & 31)) - 1u));
        fl[at] = make_uint2((unsigned)tid * (2u * (unsigned)a.caps.pub), (unsigned)L.NQ + 1u);
      }
      // the stored index of every region cell (NQ, the zero cell, for the
      // others), its global cell, and the lists of published and fetched cells
      for (int x = tid; x < R * 64; x += T) {
        const int s = x >> 6, c = x & 63, col = (int)((kOdd >> c) & 1ull);
        const u64 cmask = col ? kOdd : ~kOdd, f = S.mask[s];
        int e = L.NQ;
        if ((f >> c) & 1ull) {
          if (s < O) {
            const u64 b = S.cm[2][s];
            if (col) e = L.off[1][0] + S.base[1][s] + bits_below(f & kOdd, c);
            else if ((b >> c) & 1ull) e = L.nA + S.base[4][s] + bits_below(b & ~kOdd, c);
            else e = S.base[0][s] + bits_below(f & ~b & ~kOdd, c);
          } else {
            for (int q = 0; q < L.H + col - 1; q++) {
              const u64 m = S.cm[q][s];
              if ((m >> c) & 1ull) e = L.off[col][q + 1] + S.base[2 * q + col][s] + bits_below(m & cmask, c);
            }
          }
        }
        dense[x] = (unsigned short)e;
        if (e == L.NQ) continue;
        const unsigned g = cell_global(a, S2, s, c);
        if (s < O) {
          gl[col ? e - L.c1 + L.n[0][0] : e] = g;
          const u64 m = S.cm[which][s];
          if ((m >> c) & 1ull) pl[1 + S.base[2 + which][s] + bits_below(m, c)] = (unsigned short)e;
        } else {
          fl[S.base[8 + which][s] + bits_below(fetched(s, which != 0), c)] =
              make_uint2(__ldcg(a.xmap + (size_t)which * (size_t)d.nCells + g), (unsigned)e);
        }
      }
      __syncthreads();
      // the values and every entry's record, over the first tables
      float* sq = reinterpret_cast<float*>(tb_smem_raw);
      if (tid == 0) sq[L.NQ] = 0.f;
#pragma unroll 2
      for (int x = tid; x < R * 64; x += T) {
        const int e = dense[x], s = x >> 6, c = x & 63, cx = c & 3, cy = (c >> 2) & 3, cz = c >> 4;
        if (e >= L.NQ) continue;
        const unsigned g = cell_global(a, S2, s, c);
        sq[e] = __ldcg(a.q + g);
        if (e >= L.NE) continue;
        const float rhs = __ldcg(a.rhs + g);
        const unsigned k = __ldcg(a.diag8 + g);
        auto nbr = [&](int dir, bool in, int step, int wrap) -> unsigned {
          if (in) return (unsigned)dense[x + step] << 2;
          const unsigned t = S2.rbNb[dir][s];
          return (t == kNone ? (unsigned)L.NQ : (unsigned)dense[(int)t * 64 + c + wrap]) << 2;
        };
        const unsigned w0 = nbr(0, cx > 0, -1, 3) | (nbr(1, cx < 3, 1, -3) << 16);
        const unsigned w1 = nbr(2, cy > 0, -4, 12) | (nbr(3, cy < 3, 4, -12) << 16);
        const unsigned w2 = nbr(4, cz > 0, -16, 48) | (nbr(5, cz < 3, 16, -48) << 16);
        rec[e] = make_uint4(w0 | (k & 3u), w1 | (k >> 2), w2, __float_as_uint(rhs));
      }
    }
  }
  __syncthreads();

  if (sOverflow == 0) {
    // ---- phase 3: iterations
    const int H = sL.H, NQ = sL.NQ, c1s = sL.c1, nA = sL.nA, n00 = sL.n[0][0], n10 = sL.n[1][0];
    const int nPub = sL.pub, nFetch = sL.fetch;
    float* sq = reinterpret_cast<float*>(tb_smem_raw);
    const uint4* rec = reinterpret_cast<const uint4*>(tb_smem_raw + record_at(NQ));
    const unsigned* gl = a.glist + (unsigned)p * (unsigned)a.caps.own;
    const unsigned short* pl = a.plist + (unsigned)p * (unsigned)a.caps.pub;
    const uint2* fl = a.flist + (unsigned)p * (unsigned)a.caps.fetch;
    // a thread keeps its first four cells to fetch and to publish
    unsigned fg[4];
    unsigned short fe[4], pe[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int l = tid + u * T;
      const uint2 v = l < nFetch ? fl[l] : make_uint2(0u, 0u);
      fg[u] = v.x; fe[u] = (unsigned short)v.y;
      pe[u] = l < nPub ? pl[l] : (unsigned short)0;
    }
    __syncthreads();
    const double om1 = a.om1;
    int nChecks = 0;
    bool fresh = true, checked = false;
    // the halo values of epoch `ep`: four loads in flight per thread, then
    // each word polled again (bounded) until its tag is the epoch's
    auto wait_and_reload = [&](unsigned ep) -> bool {
      const u64* src = a.xq + (ep & 1u) * (unsigned)a.caps.pub;
      const unsigned target = tag0 + ep;
      u64 v[4];
      auto settle = [&](int e, const u64* w, u64 val) {
        long long n = 0;
        while ((unsigned)(val >> 32) != target) {
          if (++n > kTbSpinLimit || *(volatile int*)&sAbort) {
            if (n > kTbSpinLimit) atomicOr(a.err, WS_DERR_TIMEOUT);
            sAbort = 1;
            break;
          }
          val = ld_relaxed_u64(w);
        }
        sq[e] = __uint_as_float((unsigned)val);
      };
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = tid + u * T < nFetch ? ld_relaxed_u64(src + fg[u]) : 0ull;
#pragma unroll
      for (int u = 0; u < 4; u++) if (tid + u * T < nFetch) settle(fe[u], src + fg[u], v[u]);
      for (int l = tid + 4 * T; l < nFetch; l += T) {
        const uint2 f = fl[l];
        settle((int)f.y, src + f.x, ld_relaxed_u64(src + f.x));
      }
      __syncthreads();
      return *(volatile int*)&sAbort == 0;
    };
    auto publish = [&](unsigned ep) {
      u64* dst = a.xq + ((unsigned)p * 2u + (ep & 1u)) * (unsigned)a.caps.pub;
      const u64 tag = (u64)(tag0 + ep) << 32;
#pragma unroll
      for (int u = 0; u < 4; u++) if (tid + u * T < nPub) st_relaxed_u64(dst + tid + u * T, tag | __float_as_uint(sq[pe[u]]));
      for (int l = tid + 4 * T; l < nPub; l += T) st_relaxed_u64(dst + l, tag | __float_as_uint(sq[pl[l]]));
    };
    // the six neighbour values of a record, and its stencil count
    auto at = [&](unsigned off) -> float { return *reinterpret_cast<const float*>(tb_smem_raw + off); };
    auto gather = [&](const uint4& r, float (&v)[6]) {
      v[0] = at(r.x & 0xfffcu); v[1] = at(r.x >> 16); v[2] = at(r.y & 0xfffcu);
      v[3] = at(r.y >> 16); v[4] = at(r.z & 0xfffcu); v[5] = at(r.z >> 16);
    };
    auto count_of = [](const uint4& r) -> unsigned { return (r.x & 3u) | ((r.y & 3u) << 2); };
    // entries [lo, hi): two updates per thread in flight where a thread has
    // two entries (e and e + T are of one colour, so neither reads what the
    // other writes); a thread with one entry reads nothing extra
    auto sweep = [&](int lo, int hi) {
      for (int e1 = lo + tid; e1 < hi; e1 += 2 * T) {
        const uint4 r1 = rec[e1];
        float v[6];
        gather(r1, v);
        const float p1 = sPw[count_of(r1)];
        const int e2 = e1 + T;
        if (e2 < hi) {
          const uint4 r2 = rec[e2];
          float u[6];
          gather(r2, u);
          const float p2 = sPw[count_of(r2)];
          const float q1 = relax(sq[e1], p1, __uint_as_float(r1.w), v, om1);
          const float q2 = relax(sq[e2], p2, __uint_as_float(r2.w), u, om1);
          sq[e1] = q1;
          sq[e2] = q2;
        } else {
          sq[e1] = relax(sq[e1], p1, __uint_as_float(r1.w), v, om1);
        }
      }
    };
    // residual of the owned cells of the state in sq (halo values fresh)
    auto check_residual = [&]() -> bool {
      double rr = 0, bb = 0;
      for (int x = tid; x < n00 + n10; x += T) {
        const int e = x < n00 ? x : c1s + (x - n00);
        const uint4 rc = rec[e];
        float v[6];
        gather(rc, v);
        double sum = (double)v[0];
        sum += (double)v[1]; sum += (double)v[2]; sum += (double)v[3]; sum += (double)v[4]; sum += (double)v[5];
        const double b = __uint_as_float(rc.w);
        const double r = b + sum - (double)count_of(rc) * (double)sq[e];
        rr += r * r; bb += b * b;
      }
      rr = warp_sum(rr); bb = warp_sum(bb);
      if (lane == 0) sRed[warp] = make_double2(rr, bb);
      __syncthreads();
      double2 part = make_double2(0, 0);
      if (warp == 0) {
        const double2 v = sRed[lane];
        part = make_double2(warp_sum(v.x), warp_sum(v.y));
      }
      __syncthreads();
      if (!global_residual(a, part, nChecks++, &sRel, &sAbort)) return false;
      rel = sRel;
      return true;
    };
    while (it < a.iters) {
      int m = std::min(H >> 1, a.iters - it);
      if (a.check > 0) m = std::min(m, a.check - it % a.check);
      const int s = 2 * m;
      if (fresh) {
        sweep(0, sL.cum[0][s - 1]);
      } else {
        // the cells that read no halo first. With H = 4 some of them are
        // published (colour 0 to d = 3): the barrier keeps their new values
        // behind every thread's publication of the old ones
        if (H != 2) __syncthreads();
        sweep(0, nA);
        if (!wait_and_reload(epoch)) goto done;
        sweep(nA, sL.cum[0][s - 1]);
      }
      __syncthreads();
      for (int t = 2; t <= s; t++) {
        const int base = t & 1 ? 0 : c1s;
        sweep(base, base + sL.cum[t & 1 ? 0 : 1][s - t]);
        __syncthreads();
      }
      it += m;
      epoch++;
      publish(epoch);
      fresh = false;
      checked = false;
      const bool doCheck = a.check > 0 && it % a.check == 0;
      if (doCheck || it >= a.iters) {
        if (!wait_and_reload(epoch)) goto done;
        fresh = true;
        if (!check_residual()) goto done;
        checked = true;
        if (doCheck && rel <= a.tol) break;
      }
    }
    if (!checked && !check_residual()) goto done;           // no iteration ran: residual of the start
    // the result lands in the solve's own q buffer
    for (int x = tid; x < n00 + n10; x += T) {
      const int e = x < n00 ? x : c1s + (x - n00);
      __stcg(a.q + gl[x], sq[e]);
    }
    solved = true;
  } else if (!a.listFallback) {
    solved = true;
    // ---- fallback: red-black sweeps over the owned bricks in global memory,
    // a grid barrier per half-sweep
    path = 4;
    const int t0 = sT0;
    const int O = sT1 - sT0;
    const double om1 = a.om1;
    const long long nxl = d.nx, nxy = (long long)d.nx * d.ny;
    int nChecks = 0;
    auto cell_of = [&](int item, int col, long long& g) -> bool {
      const int s = item >> 5, kk = item & 31, row = kk >> 1, cy = row & 3, cz = row >> 2;
      const int cx = ((col + cy + cz) & 1) + 2 * (kk & 1);
      const int lin = __ldcg(&a.actLin[t0 + s]);
      const int bx = lin % a.nbx, tq = lin / a.nbx, by = tq % a.nby, bz = tq / a.nby;
      const int i = bx * 4 + cx, j = by * 4 + cy, k = bz * 4 + cz;
      if (i >= d.nx || j >= d.ny || k >= d.nz || !interior(d, i, j, k)) return false;
      g = ((long long)k * d.ny + j) * d.nx + i;
      return __ldcg(a.pw + g) >= 0.f;
    };
    auto residual = [&]() -> bool {
      double rr = 0, bb = 0;
      for (int col = 0; col < 2; col++)
        for (int item = tid; item < O * 32; item += T) {
          long long g;
          if (!cell_of(item, col, g)) continue;
          const float* qc = a.q + g;
          double sum = (double)__ldcg(qc - 1);
          sum += (double)__ldcg(qc + 1); sum += (double)__ldcg(qc - nxl); sum += (double)__ldcg(qc + nxl);
          sum += (double)__ldcg(qc - nxy); sum += (double)__ldcg(qc + nxy);
          const double b = a.rhs[g];
          const double r = b + sum - (double)a.diag8[g] * (double)__ldcg(qc);
          rr += r * r; bb += b * b;
        }
      rr = warp_sum(rr); bb = warp_sum(bb);
      if (lane == 0) sRed[tid >> 5] = make_double2(rr, bb);
      __syncthreads();
      double2 part = make_double2(0, 0);
      if (tid < 32) {
        const double2 v = sRed[tid];
        part = make_double2(warp_sum(v.x), warp_sum(v.y));
      }
      __syncthreads();
      if (!global_residual(a, part, nChecks++, &sRel, &sAbort)) return false;
      rel = sRel;
      return true;
    };
    bool checked = false;
    while (it < a.iters) {
      for (int col = 0; col < 2; col++) {
        for (int item = tid; item < O * 32; item += T) {
          long long g;
          if (!cell_of(item, col, g)) continue;
          float* qc = a.q + g;
          float v[6];
          v[0] = __ldcg(qc - 1); v[1] = __ldcg(qc + 1); v[2] = __ldcg(qc - nxl);
          v[3] = __ldcg(qc + nxl); v[4] = __ldcg(qc - nxy); v[5] = __ldcg(qc + nxy);
          __stcg(qc, relax(__ldcg(qc), a.pw[g], a.rhs[g], v, om1));
        }
        if (!tb_grid_barrier(a.ctl, ++nBar, a.err, &sAbort)) goto done;
      }
      it++;
      checked = false;
      const bool doCheck = a.check > 0 && it % a.check == 0;
      if (doCheck) {
        if (!residual()) goto done;
        checked = true;
        if (rel <= a.tol) break;
      }
    }
    if (!checked && !residual()) goto done;
  }
done:
  if (p == 0 && tid == 0) {
    // every CTA read the tag base before its first barrier, which this CTA has passed
    *(volatile unsigned*)&a.ctl->tagBase = tb_next_tag_base(tag0, epoch, sAbort, a.iters);
    if (solved || sAbort) a.ctl->solved = 1;         // after a timed-out wait nothing else runs either
    if (solved || sAbort) { *a.outIters = it; *a.outRel = rel; *a.outPath = path; }
  }
}

// ---------------------------------------------------------------- host side
struct TbState {
  void* slab = nullptr;
  TbCtl* ctl = nullptr;
  u64* xq = nullptr;
  int2* cntPart = nullptr;
  int *actLin = nullptr, *wPre = nullptr, *chunkStart = nullptr;
  unsigned *xmap = nullptr, *glist = nullptr;
  unsigned short *plist = nullptr, *dense = nullptr;
  uint2* flist = nullptr;
  double2* resPart = nullptr;
  int P = 0, nbx = 0, nby = 0, nbz = 0, mbits = 0;
  TbCaps caps{};
};
// The most that one of P CTAs can hold on a grid of nB bricks. Its owned bricks but
// the last weigh less than its share of the total (at most 80 a brick) together, and
// a brick weighs 17 at least. A halo cell lies within L1 distance 4 of an
// owned brick: 704 cells around each. The dense tables need global memory only
// where they may have no room beside the records. With every list at its maximum a
// 24^3 handle held 58 MB for the solve, so 10.
static TbCaps tb_caps(const Dims& d, long long nB, int P) {
  const long long weight = (kBrickWeight + 64) * nB / P + kBrickWeight + 64, bricks = std::min(nB, weight / (kBrickWeight + 1));
  const long long cells = (long long)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  const long long own = std::min(cells, std::min(64 * bricks, weight)), halo = std::min(cells, 704 * bricks);
  const long long region = std::min<long long>(kRbMax, std::min(nB, 27 * bricks)), all = std::min<long long>(kQMax - 1, own + halo);
  TbCaps c;
  c.own = (int)std::min<long long>(kQMax, own);
  c.pub = (int)std::min<long long>(kPubMax, own + 1);
  c.fetch = (int)std::min<long long>(kFetchMax, halo + P);
  c.rows = dense_at((int)region, (int)all, (int)all) >= 0 ? 0 : (int)region;
  return c;
}

// null when the solve cannot run on this device (too little shared memory or
// co-residency) or grid (a brick coordinate beyond 8 bits); the state is
// then left unallocated.
cudaError_t sor_tb_init(void** statePtr, const Dims& d, int device) {
  *statePtr = nullptr;
  int smCount = 0, optin = 0;
  cudaDeviceGetAttribute(&smCount, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (smCount < 1 || smCount > kMaxCtas || optin < kTbSmem) return cudaSuccess;
  if (std::max(d.nx, std::max(d.ny, d.nz)) > 1020) return cudaSuccess;
  if (cudaFuncSetAttribute(k_sor_tb, cudaFuncAttributeMaxDynamicSharedMemorySize, kTbSmem) != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  int perSM = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_sor_tb, kTbThreads, kTbSmem) != cudaSuccess || perSM < 1) {
    cudaGetLastError();
    return cudaSuccess;
  }
  TbState* S = new TbState();
  *statePtr = S;
  S->P = smCount;
  S->nbx = (d.nx + 3) / 4; S->nby = (d.ny + 3) / 4; S->nbz = (d.nz + 3) / 4;
  int mb = 0;
  while ((1 << mb) < std::max(S->nbx, std::max(S->nby, S->nbz))) mb++;
  S->mbits = mb;
  const long long nB = (long long)S->nbx * S->nby * S->nbz;
  // every buffer from one allocation (exchange words zeroed: tags start at 1)
  S->caps = tb_caps(d, nB, smCount);
  const size_t P = (size_t)smCount, words = 2 * (size_t)S->caps.pub * P;
  size_t at = 0;
  auto place = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~(size_t)255; return o; };
  const size_t oCtl = place(sizeof(TbCtl)), oXq = place(sizeof(u64) * words), oCnt = place(sizeof(int2) * P);
  const size_t zeroed = at;
  const size_t oAct = place(sizeof(int) * (size_t)nB), oPre = place(sizeof(int) * (size_t)nB);
  const size_t oChunk = place(sizeof(int) * (P + 1)), oMap = place(sizeof(unsigned) * 2 * (size_t)d.nCells);
  const size_t oG = place(sizeof(unsigned) * S->caps.own * P), oP = place(sizeof(unsigned short) * S->caps.pub * P);
  const size_t oD = place(sizeof(unsigned short) * 64 * S->caps.rows * P), oF = place(sizeof(uint2) * S->caps.fetch * P);
  const size_t oRes = place(sizeof(double2) * 2 * P);
  cudaError_t e;
  if ((e = cudaMalloc(&S->slab, at)) != cudaSuccess) return e;
  if ((e = cudaMemset(S->slab, 0, zeroed)) != cudaSuccess) return e;
  unsigned char* base = (unsigned char*)S->slab;
  S->ctl = (TbCtl*)(base + oCtl); S->xq = (u64*)(base + oXq); S->cntPart = (int2*)(base + oCnt);
  S->actLin = (int*)(base + oAct); S->wPre = (int*)(base + oPre); S->chunkStart = (int*)(base + oChunk);
  S->xmap = (unsigned*)(base + oMap); S->glist = (unsigned*)(base + oG); S->plist = (unsigned short*)(base + oP);
  S->dense = (unsigned short*)(base + oD); S->flist = (uint2*)(base + oF); S->resPart = (double2*)(base + oRes);
  return cudaSuccess;
}

void sor_tb_free(void* statePtr) {
  TbState* S = (TbState*)statePtr;
  if (!S) return;
  cudaFree(S->slab);
  delete S;
}
const int* sor_tb_solved(void* statePtr) { return &((TbState*)statePtr)->ctl->solved; }

// the control block reset and the solve (two stream operations, one kernel).
// listFallback: leave a system that does not fit to the list kernels
cudaError_t launch_sor_tb(void* statePtr, const Dims& d, const GridDev& g, const uint8_t* diag8, double omega,
                          int iters, int check, double tol, DevStatus* st, bool listFallback, bool report,
                          cudaStream_t s) {
  TbState* S = (TbState*)statePtr;
  cudaError_t e = cudaMemsetAsync(S->ctl, 0, offsetof(TbCtl, tagBase), s);
  if (e != cudaSuccess) return e;
  TbArgs a;
  a.d = d; a.q = g.q; a.xq = S->xq; a.rhs = g.rhs; a.pw = g.pw; a.diag8 = diag8; a.fmask = g.fmask; a.st = st;
  a.nbx = S->nbx; a.nby = S->nby; a.nbz = S->nbz; a.mbits = S->mbits;
  a.cntPart = S->cntPart; a.actLin = S->actLin; a.wPre = S->wPre; a.chunkStart = S->chunkStart;
  a.xmap = S->xmap; a.glist = S->glist; a.plist = S->plist; a.dense = S->dense; a.caps = S->caps; a.flist = S->flist; a.resPart = S->resPart; a.ctl = S->ctl;
  a.om1 = 1 - omega; a.iters = iters; a.check = check; a.tol = tol; a.err = &st->err;
  a.listFallback = listFallback ? 1 : 0;
  a.regionPath = report && listFallback ? 1 : 3;   // ws_scalars.sorPath has one number for both above 160^3
  const SorOut out(st, report);
  a.outIters = out.iters; a.outRel = out.rel; a.outPath = out.path;
  void* args[] = { &a };
  return cudaLaunchCooperativeKernel((void*)k_sor_tb, dim3(S->P), dim3(kTbThreads), args, kTbSmem, s);
}
