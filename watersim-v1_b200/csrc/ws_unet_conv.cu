// ws_unet_conv.cu — 3x3x3 convolution of the warm-start U-Net as an
// implicit GEMM on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// One CTA computes a sub-tile of 8 (x) x 16 (y) x ZT (z) output voxels of one
// active tile. For each 16-channel slice of the input it stages, in shared
// memory, the (8+2) x (16+2) x (ZT+2) halo of that slice (two 8-channel
// chunks, voxel-major, 16 bytes per voxel per chunk) and the slice's weights
// for all 27 taps. One elected thread then issues, for every output plane z
// and tap (dz, dy, dx), one tcgen05.mma of M = 128 (the 8 x 16 voxels of the
// plane), N = cout, K = 16 (the channel slice), BF16 inputs, FP32
// accumulator in tensor memory. The A operand of a tap is the halo shifted by
// (dz, dy, dx): with the no-swizzle K-major layout each 8-row core matrix is
// the 8 x-consecutive voxels of one y-row (128 contiguous bytes), the stride
// between core matrices along M is one halo row (160 bytes) and the stride
// between the two K chunks is one halo chunk, so a shift only moves the
// descriptor's start address. Inactive neighbour tiles and voxels outside
// the grid are staged as zeros. The epilogue reads the accumulators with
// tcgen05.ld (each warp its 32-lane quarter), adds bias and ReLU (forward)
// or applies a ReLU mask (backward data), and stores BF16 NDHWC.
//
// Every mbarrier wait is bounded; on a timeout the CTA latches
// WS_DERR_TIMEOUT, waits once more (bounded) for its MMAs, frees its tensor
// memory and returns.
#include "ws_unet.cuh"
#include <algorithm>

namespace unet {

static constexpr long long kWaitLimit = 1LL << 24;
constexpr int kConvThreads = 256;                   // threads of every kernel here

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, no swizzle: start, leading (K-chunk) and
// stride (8-row group) byte offsets in 16-byte units, descriptor version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// instruction descriptor of kind::f16: D f32, A bf16, B bf16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16_m128(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
               :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (long long n = 0; n < kWaitLimit; n++)
    if (mbar_try(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Output planes per work item. 16 channels: eight (a whole tile), bound by the
// MMAs' operand reads, which more planes per halo plane share. 32: four, so that
// two or three CTAs an SM overlap staging and MMAs (4500 and 5500 cycles a slice)
// where a tile per item gives it one: a whole prediction takes 207 us at 64^3 (229
// with eight planes), 267 at 97^3 (269), 327 at 128^3 (327), 1304 at 256^3 with four
// levels (1320); in the training at 128^3, whose half-resolution level has about as
// many tiles as SMs, those layers' mean is 25.3 us (32.1; 29.8 with two). 48 to 128:
// two, as on the coarse levels a tile per item would leave most SMs idle (the 32^3
// level has 32 tiles) and each CTA would walk four or more input slices in turn;
// four for 48 changed nothing.
template <int COUT> struct ConvShape {
  static constexpr int ZT = COUT == 16 ? 8 : COUT == 32 ? 4 : COUT <= 128 ? 2 : 1;
  static constexpr int HX = kTX + 2, HY = kTY + 2, HZ = ZT + 2;
  static constexpr int HV = HX * HY * HZ;           // halo voxels
  static constexpr int KSTR = HV * 16;              // bytes of one 8-channel halo chunk
  static constexpr int WCH = 27 * 2 * COUT * 16;    // bytes of one 16-channel weight slice
  static constexpr int NCOL = ZT * COUT;
  static constexpr int TCOLS = NCOL <= 32 ? 32 : NCOL <= 64 ? 64 : NCOL <= 128 ? 128 : NCOL <= 256 ? 256 : 512;
  // shared memory per CTA, padded so that the CTAs one SM can hold never
  // ask for more than the 512 tensor-memory columns together (233472 bytes
  // of shared memory per SM, 1 KB of it reserved per CTA)
  static constexpr int MAXCTA = 512 / TCOLS;
  static constexpr int SMEM_MIN = 233472 / (MAXCTA + 1) + 1;
  static constexpr int SMEM = 2 * KSTR + WCH > SMEM_MIN ? 2 * KSTR + WCH : SMEM_MIN;
  static constexpr int PERSM = 233472 / (SMEM + 1280) > 1 ? 233472 / (SMEM + 1280) : 1;   // CTAs one SM holds
};

// 16-byte asynchronous global -> shared copy; src_size 0 writes zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_size) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(src_size) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// queue the copies of one 16-channel slice of the halo of sub-tile (X0, Y0, Z0).
// The activity of the (up to) 3x3x3 tiles the halo touches is read once into
// shared memory, so no copy waits on a global load of its own.
template <int COUT>
__device__ __forceinline__ void stage_halo(const ConvArgs& a, int X0, int Y0, int Z0, int kk, uint32_t hbase,
                                           uint8_t* s_act) {
  using S = ConvShape<COUT>;
  constexpr int HX = S::HX, HY = S::HY, HV = S::HV, KSTR = S::KSTR;
  const int tx0 = X0 / kTX - 1, ty0 = Y0 / kTY - 1, tz0 = (Z0 + kTZ - 1) / kTZ - 1;   // tile of the halo's low corner
  if (threadIdx.x < 27) {
    const int t = threadIdx.x, tx = tx0 + t % 3, ty = ty0 + (t / 3) % 3, tz = tz0 + t / 9;
    s_act[t] = (tx >= 0 && ty >= 0 && tz >= 0 && tx < a.ntx && ty < a.nty && tz < a.ntz)
                   ? a.active[(tz * a.nty + ty) * a.ntx + tx] : (uint8_t)0;
  }
  __syncthreads();
  const int cnx = (a.nx + 1) >> 1, cny = (a.ny + 1) >> 1;
  // the slice's source: both 8-channel chunks come from one (the channel
  // splits c0 are multiples of 16)
  const int c = kk * 16;
  const bool first = c < a.c0, up = first && a.up0;
  const bf16* src = first ? a.src0 + c : a.src1 + (c - a.c0);
  const int stride = first ? a.c0 : a.c1;
  const int sx = up ? cnx : a.nx, sy = up ? cny : a.ny, sh = up ? 1 : 0;
  // one voxel per thread and pass, both 8-channel chunks of the slice; the
  // passes are unrolled so that their address chains overlap (a block has two
  // warps per scheduler: one chain after the other took 4.4 us per tile)
  constexpr int PASSES = (HV + kConvThreads - 1) / kConvThreads;
#pragma unroll
  for (int it = 0; it < PASSES; it++) {
    const int hv = (int)threadIdx.x + it * kConvThreads;
    if (it == PASSES - 1 && hv >= HV) break;
    const int hx = hv % HX, t2 = hv / HX, hy = t2 % HY, hz = t2 / HY;
    const int gx = X0 - 1 + hx, gy = Y0 - 1 + hy, gz = Z0 - 1 + hz;
    const bool in = (unsigned)gx < (unsigned)a.nx && (unsigned)gy < (unsigned)a.ny && (unsigned)gz < (unsigned)a.nz &&
                    s_act[((gz / kTZ - tz0) * 3 + (gy / kTY - ty0)) * 3 + (gx / kTX - tx0)];
    const bf16* p = in ? src + ((size_t)((gz >> sh) * sy + (gy >> sh)) * sx + (gx >> sh)) * stride : src;   // any valid address when nothing is read
    const uint32_t n = in ? 16u : 0u;
    cp_async16(hbase + (uint32_t)(hv * 16), p, n);
    cp_async16(hbase + (uint32_t)(KSTR + hv * 16), p + 8, n);
  }
}
template <int COUT>
__device__ __forceinline__ void stage_weights(const ConvArgs& a, int kk, uint32_t wbase) {
  constexpr int WCH = ConvShape<COUT>::WCH;
  const char* src = reinterpret_cast<const char*>(a.w) + (size_t)kk * WCH;
#pragma unroll 4
  for (int i = threadIdx.x; i < WCH / 16; i += kConvThreads) cp_async16(wbase + (uint32_t)(i * 16), src + (size_t)i * 16, 16);
}

// Persistent over the work items (active tile x z sub-tile): tensor memory
// is allocated once per CTA; weights stay resident when the input has a
// single 16-channel slice; the next item's first slice is fetched while
// the current item's accumulators are drained.
template <int COUT>
__global__ void __launch_bounds__(kConvThreads, ConvShape<COUT>::PERSM) k_conv3(ConvArgs a) {
  using S = ConvShape<COUT>;
  constexpr int ZT = S::ZT, HX = S::HX, HY = S::HY, KSTR = S::KSTR;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ uint8_t s_act[27];

  constexpr int sub = kTZ / ZT;
  const int nItems = *a.nTiles * sub;
  if ((int)blockIdx.x >= nItems) return;            // uniform over the CTA
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t hbase = smem_u32(smem), wbase = hbase + 2 * KSTR;
  const int cin = a.c0 + a.c1, nslices = cin >> 4;
  const bool wres = nslices == 1;                   // weights loaded once

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&s_tmem)), "r"((uint32_t)S::TCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) { mbar_init(&mbar, 1); s_abort = 0; }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s_tmem;
  constexpr uint32_t idesc = idesc_bf16_m128(COUT);
  // N = 2 and 3 COUT (two or three z taps); with ZT = 2 at most two z taps meet one plane
  constexpr uint32_t idesc2 = idesc_bf16_m128(2 * COUT);
  constexpr uint32_t idesc3 = idesc_bf16_m128((ZT >= 3 ? 3 : 2) * COUT);
  static_assert((ZT >= 3 ? 3 : ZT) * COUT <= 256 && COUT % 16 == 0, "MMA N out of range");
  uint32_t phase = 0;
  bool pending = false;

  auto origin = [&](int item, int& X0, int& Y0, int& Z0) {
    const int tile = a.tiles[item / sub];
    const int tx = tile % a.ntx, ty = (tile / a.ntx) % a.nty, tz = tile / (a.ntx * a.nty);
    X0 = tx * kTX; Y0 = ty * kTY; Z0 = tz * kTZ + (item % sub) * ZT;
  };
  int X0, Y0, Z0;
  origin(blockIdx.x, X0, Y0, Z0);
  stage_halo<COUT>(a, X0, Y0, Z0, 0, hbase, s_act);
  stage_weights<COUT>(a, 0, wbase);
  for (int item = blockIdx.x; item < nItems; item += gridDim.x) {
    for (int kk = 0; kk < nslices; kk++) {
      cp_async_wait_all();
      fence_proxy_async();                           // generic-proxy writes -> tensor-core reads
      __syncthreads();
      if (threadIdx.x == 0) {
        fence_after();
        // Per in-plane tap g = (dy, dx), halo plane p feeds output planes
        // p - dz for dz = 0..2: one MMA with the B rows of those z taps side
        // by side along N (k_pack orders them dz = 2, 1, 0) writes the
        // accumulators of planes p - dzhi .. p - dzlo, which are adjacent in
        // tensor memory. Each A tile is then read once per (g, p) instead of
        // once per (g, dz, z). The first tap group initialises every
        // accumulator plane by plane (dz = 0 first), the later groups only
        // accumulate. Descriptors are base descriptors plus 16-byte offsets
        // in the start-address field.
        const uint64_t ad0 = smem_desc(hbase, KSTR, HX * 16), bd0 = smem_desc(wbase, 3 * COUT * 16, 128);
        constexpr int GB = 6 * COUT;                 // 16-byte units of one tap group (2 K halves x 3 z taps)
#pragma unroll
        for (int z = 0; z < ZT; z++)
#pragma unroll
          for (int dz = 0; dz < 3; dz++)
            mma_bf16(tmem + (uint32_t)(z * COUT), ad0 + (uint64_t)((z + dz) * HY * HX),
                     bd0 + (uint64_t)((2 - dz) * COUT), idesc, (kk | dz) != 0);
#pragma unroll 1
        for (int g = 1; g < 9; g++) {
          const int dy = g / 3, dx = g % 3;
          const uint64_t ag = ad0 + (uint64_t)(dy * HX + dx), bg = bd0 + (uint64_t)(g * GB);
#pragma unroll
          for (int p = 0; p < ZT + 2; p++) {
            const int dzlo = p > ZT - 1 ? p - (ZT - 1) : 0, dzhi = p < 2 ? p : 2;
            const uint32_t id = dzhi - dzlo == 0 ? idesc : dzhi - dzlo == 1 ? idesc2 : idesc3;
            mma_bf16(tmem + (uint32_t)((p - dzhi) * COUT), ag + (uint64_t)(p * HY * HX),
                     bg + (uint64_t)((2 - dzhi) * COUT), id, 1u);
          }
        }
        mma_commit(&mbar);
      }
      pending = true;
      const bool ok = mbar_wait(&mbar, phase);       // the staged operands are free again
      if (!ok) { s_abort = 1; atomicOr(a.err, WS_DERR_TIMEOUT); }
      __syncthreads();
      if (s_abort) break;
      pending = false;
      phase ^= 1u;
      if (kk + 1 < nslices) {
        stage_halo<COUT>(a, X0, Y0, Z0, kk + 1, hbase, s_act);
        stage_weights<COUT>(a, kk + 1, wbase);
      }
    }
    if (s_abort) break;
    // fetch the next item's first slice while this item's accumulators drain
    const int cX = X0, cY = Y0, cZ = Z0;
    const int next = item + gridDim.x;
    if (next < nItems) {
      origin(next, X0, Y0, Z0);
      stage_halo<COUT>(a, X0, Y0, Z0, 0, hbase, s_act);
      if (!wres) stage_weights<COUT>(a, 0, wbase);
    }
    fence_after();
    {
      const int q = warp & 3;                        // tensor-memory lane quarter of this warp
      const int m = q * 32 + lane;                   // accumulator row = voxel of the plane
      const int gx = cX + (m & 7), gy = cY + (m >> 3);
#pragma unroll 1
      for (int cg = 0; cg < COUT / 16; cg++) {
        const int c = cg * 16;
        float bias[16];                              // this channel group's bias, once for all planes
#pragma unroll
        for (int i = 0; i < 16; i++) bias[i] = a.mode == 0 ? __ldg(a.bias + c + i) : 0.f;
        for (int z = warp >> 2; z < ZT; z += 2) {
          const int gz = cZ + z;
          const bool in = gx < a.nx && gy < a.ny && gz < a.nz;
          const size_t vox = ((size_t)gz * a.ny + gy) * a.nx + gx;
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(z * COUT + cg * 16), r);
          if (!in) continue;
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
          if (a.mode == 0) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = fmaxf(v[i] + bias[i], 0.f);
          } else if (a.mask) {
            const uint4* mp = reinterpret_cast<const uint4*>(a.mask + vox * COUT + c);
            uint4 mk[2] = { __ldg(mp), __ldg(mp + 1) };
            const bf16* mb = reinterpret_cast<const bf16*>(mk);
#pragma unroll
            for (int i = 0; i < 16; i++) if (!(__bfloat162float(mb[i]) > 0.f)) v[i] = 0.f;
          }
          uint4 o[2];
          __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
          for (int i = 0; i < 8; i++) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
          uint4* dst = c < a.split
              ? reinterpret_cast<uint4*>(a.out0 + vox * a.split + c)
              : reinterpret_cast<uint4*>(a.out1 + vox * (COUT - a.split) + (c - a.split));
          dst[0] = o[0]; dst[1] = o[1];
        }
      }
    }
    fence_before();                                  // accumulators read before the next item's MMAs
  }
  if (s_abort && pending) mbar_wait(&mbar, phase);    // bounded: let the issued MMAs drain
  cp_async_wait_all();
  fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)S::TCOLS) : "memory");
}

// ------------------------------------------------------------ weight gradient
// dW[co][ci][t] += sum_v X(v + off_t)[ci] dZ(v)[co] over the voxels of
// active tiles, on the tensor cores. A work item is one active tile and one
// 16-channel input slice; the tile's dZ and the slice's halo are staged in
// shared memory. K is voxels: 16 (two x-rows of a plane) per MMA, both
// operands MN-major (a core matrix is 8 channels, 16 bytes, by 8 voxels).
//
// An MMA this small is bound by the shared-memory reads of its operands, so
// one MMA covers as many taps as the operands' strides allow:
//  - along M the z taps: with dZ stored plane by plane, the rows of planes
//    p - 2, p - 1, p, ... are one run of 8-channel chunks at a fixed stride,
//    and against halo plane p they are the taps dz = 2, 1, 0. 16 and 32
//    output channels take four planes (M = 64, 128; the fourth is not used),
//    64 take p - 1, p (M = 128) and p - 2 (M = 64). Zero planes below and
//    above the tile stand for the planes that are not there.
//  - along N the x taps: the B rows of taps dx = 0, 1, 2 are the same halo
//    bytes one voxel (16 bytes) further, so the stride between 8-channel
//    groups is 16 bytes and N = 24 holds three taps of 8 input channels
//    (M = 128 wants a multiple of 16: N = 32, the fourth group not used).
// That leaves (dy, channel half) = 6 accumulators and 10 planes x 8 K steps x
// 6 = 480 MMAs per item (C = 64: 432 + 384) instead of 1728 of M = 64, N = 16
// with one tap each, a quarter of the rows used at 16 channels.
//
// The accumulators stay in tensor memory over a CTA's whole run of items of
// one slice (items are slice-major, a contiguous range per CTA) and drain
// once per run into FP32 atomics. The bias gradient (slice 0) is summed by all
// threads from the staged dZ while the MMAs run. Of an item's time at 16 channels
// (two CTAs per SM) the MMAs are about 60% (23 cycles each, their operands'
// 2.8 KB at 128 bytes per cycle); at 32 and 64 (one CTA) 63% and 58%, staging the
// rest. Measured on the 128^3 planet (627 finest tiles): the ten layers of a
// sample 2.89 -> 0.59 ms.
//
// one pass covers output channels coOff .. coOff + cout - 1 (cout <= 64) of a
// dZ with dzStride channels per voxel
struct DwTcArgs { ConvArgs src; const bf16* dz; int cout, dzStride, coOff; float* dw; float* db; };
template <int C> struct DwShape {
  static constexpr int CH = C / 8;                  // 8-channel chunks of dZ
  static constexpr int PLANE = CH * 128 * 16;       // bytes of one z plane of dZ
  static constexpr int ZPAD = C == 64 ? 1 : 2;      // zero planes on either side of the tile
  static constexpr int NPLANE = kTZ + 2 * ZPAD;
  static constexpr int HALO = 2 * ConvShape<16>::KSTR;
  // the halo lies behind the dZ: the rows of the unused fourth plane at the
  // tile's top read its bytes, and 16 spare bytes end the last x tap group
  static constexpr int SMEM = NPLANE * PLANE + HALO + 128;
  static constexpr int ROWS = C == 16 ? 64 : 128;   // M of the first MMA kind
  static constexpr int NCOL = C == 16 ? 24 : 32;
  static constexpr int TCOLS = C == 64 ? 512 : 256; // 6 accumulators of 32 columns, twice at 64 channels
  static constexpr int PERSM = C == 16 ? 2 : 1;     // CTAs one SM holds (shared memory)
};
static_assert(DwShape<16>::SMEM * 2 + 4096 <= 233472 && DwShape<32>::SMEM <= 231424 && DwShape<64>::SMEM <= 231424,
              "halo and dZ of a tile fit the CTAs' shared memory");
// instruction descriptor: D f32, A and B bf16, both MN-major. With M = 64 the
// accumulator rows 16q..16q+15 sit in tensor-memory lanes 32q..32q+15 (the
// lower half of each 32-lane subpartition).
constexpr uint32_t idesc_dw(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

template <int C>
__global__ void __launch_bounds__(256, DwShape<C>::PERSM) k_dw_tc(DwTcArgs A) {
  const ConvArgs& a = A.src;
  using S = ConvShape<16>;                          // ZT = 8: the whole tile's halo of one slice
  using D = DwShape<C>;
  constexpr int HX = S::HX, HY = S::HY, KSTR = S::KSTR;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ uint8_t s_act[27];
  __shared__ float s_bias[8][64];
  const int cin = a.c0 + a.c1, nsl = cin >> 4, cout = A.cout;
  const int nT = *a.nTiles;
  const long long nItems = (long long)nT * nsl;
  const int lo = (int)(nItems * blockIdx.x / gridDim.x), hi = (int)(nItems * (blockIdx.x + 1) / gridDim.x);
  if (lo >= hi) return;                             // uniform over the CTA
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t zbase = smem_u32(smem), hbase = zbase + (uint32_t)(D::NPLANE * D::PLANE);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&s_tmem)), "r"((uint32_t)D::TCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) { mbar_init(&mbar, 3); s_abort = 0; }
  // the zero planes, the rows co >= cout and the spare bytes
  for (int i = threadIdx.x; i < D::SMEM / 16; i += blockDim.x) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s_tmem;
  const uint64_t ad0 = smem_desc(zbase, 128, 128 * 16), bd0 = smem_desc(hbase, HX * 16, 16);
  uint32_t phase = 0;
  bool pending = false, fresh = true;
  float bs[8] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };   // bias gradient of chunk (thread % CH)
  for (int item = lo; item < hi; item++) {
    const int kk = item / nT, tile = a.tiles[item - kk * nT];
    const int tx = tile % a.ntx, ty = (tile / a.ntx) % a.nty, tz = tile / (a.ntx * a.nty);
    const int X0 = tx * kTX, Y0 = ty * kTY, Z0 = tz * kTZ;
    stage_halo<16>(a, X0, Y0, Z0, kk, hbase, s_act);
    {
      // dZ: thread m of a 128-thread half takes voxel m of planes half, half + 2, ...
      const int m = threadIdx.x & 127, gx = X0 + (m & 7), gy = Y0 + (m >> 3);
      const bool inXY = gx < a.nx && gy < a.ny;
      const bf16* col = A.dz + ((size_t)gy * a.nx + gx) * A.dzStride + A.coOff;
      const size_t plane = (size_t)a.ny * a.nx * A.dzStride;
#pragma unroll
      for (int z = 0; z < kTZ; z += 2) {
        const int zz = z + (int)(threadIdx.x >> 7);
        const bool in = inXY && Z0 + zz < a.nz;
        const bf16* src = in ? col + plane * (size_t)(Z0 + zz) : A.dz;
#pragma unroll
        for (int c = 0; c < D::CH; c++)
          if (c * 8 < cout)
            cp_async16(zbase + (uint32_t)((zz + D::ZPAD) * D::PLANE + c * 2048 + m * 16), in ? src + c * 8 : src, in ? 16u : 0u);
      }
    }
    cp_async_wait_all();
    fence_proxy_async();
    __syncthreads();
    // One thread keeps the tensor pipe about half busy with MMAs this small,
    // so three issue: warp w the accumulators of y tap w.
    if (lane == 0 && warp < 3) {
      fence_after();
      const uint32_t dcol = tmem + (uint32_t)(warp * 64);
      const uint64_t bw = bd0 + (uint64_t)(warp * HX);
      // halo plane p (voxel z = p - 1) against the dZ planes p - 2 .. p (taps dz = 2 .. 0)
#pragma unroll 1
      for (int p = 0; p < kTZ + 2; p++) {
        const uint64_t bp = bw + (uint64_t)(p * HY * HX), ap = ad0 + (uint64_t)((p * D::PLANE) >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ks++) {
          const uint64_t bk = bp + (uint64_t)(2 * ks * HX), ak = ap + (uint64_t)(ks * 16);
          const uint32_t first = (fresh && p == 0 && ks == 0) ? 0u : 1u;
          if (C != 64) {                             // plane p - 2 up, two zero planes below
            mma_bf16(dcol, ak, bk, idesc_dw(D::ROWS, D::NCOL), first);
            mma_bf16(dcol + 32, ak, bk + (uint64_t)(KSTR >> 4), idesc_dw(D::ROWS, D::NCOL), first);
          } else {
            if (p < kTZ + 1) {                       // planes p - 1, p (one zero plane below)
              mma_bf16(dcol, ak, bk, idesc_dw(128, 32), first);
              mma_bf16(dcol + 32, ak, bk + (uint64_t)(KSTR >> 4), idesc_dw(128, 32), first);
            }
            if (p >= 2) {                            // plane p - 2
              const uint32_t first2 = (fresh && p == 2 && ks == 0) ? 0u : 1u;
              const uint64_t am = ak - (uint64_t)(D::PLANE >> 4);
              mma_bf16(dcol + 192, am, bk, idesc_dw(64, 24), first2);
              mma_bf16(dcol + 224, am, bk + (uint64_t)(KSTR >> 4), idesc_dw(64, 24), first2);
            }
          }
        }
      }
      mma_commit(&mbar);
    }
    pending = true;
    fresh = false;
    if (kk == 0) {                                   // bias gradient while the MMAs run
      const int c = threadIdx.x % D::CH;
#pragma unroll 4
      for (int v = threadIdx.x / D::CH; v < kTZ * 128; v += kConvThreads / D::CH) {
        const uint4 u = *reinterpret_cast<const uint4*>(smem + ((v >> 7) + D::ZPAD) * D::PLANE + c * 2048 + (v & 127) * 16);
        const bf16* e = reinterpret_cast<const bf16*>(&u);
#pragma unroll
        for (int q = 0; q < 8; q++) bs[q] += __bfloat162float(e[q]);
      }
    }
    const bool ok = mbar_wait(&mbar, phase);
    if (!ok) { s_abort = 1; atomicOr(a.err, WS_DERR_TIMEOUT); }
    __syncthreads();
    if (s_abort) break;
    pending = false;
    phase ^= 1u;
    if (item + 1 < hi && (item + 1) / nT == kk) continue;   // the run goes on: the accumulators stay
    fence_after();
    // Accumulator columns dx * 8 + (input channel of the half); rows: see
    // above. One channel half at a time goes to shared memory (over the halo,
    // which the next item stages anew) in the order of dW, a row of 8 x 27 per
    // output channel padded to an odd stride, and from there to global memory
    // with neighbouring lanes on neighbouring addresses: an atomic per lane on
    // a sector of its own cost 8 us more at 16 channels, where 296 CTAs add to
    // the same 27 KB.
    const int q = warp & 3;
    float* st = reinterpret_cast<float*>(smem + D::NPLANE * D::PLANE);
    constexpr int ROW = 8 * 27 + 1;
    static_assert(C * ROW * 4 <= D::HALO, "one channel half of dW fits the halo's place");
    for (int half = 0; half < 2; half++) {
      for (int jj = warp >> 2; jj < (C == 64 ? 6 : 3); jj += 2) {
        const int dy = jj % 3, j = 2 * dy + half + (jj >= 3 ? 6 : 0);
        int co, dz;
        if (C == 16) { co = lane < 16 ? lane : 64; dz = 2 - q; }
        else if (C == 32) { co = lane; dz = 2 - q; }
        else if (j < 6) { co = (q & 1) * 32 + lane; dz = 1 - (q >> 1); }
        else { co = lane < 16 ? q * 16 + lane : 64; dz = 2; }
        uint32_t r0[16], r1[16];                     // taps dx = 0, 1 and dx = 2 (upper half of r1 unused)
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(j * 32);
        tmem_ld16(at, r0);
        tmem_ld16(at + 16, r1);
        if (co >= cout || dz < 0) continue;
        float* dst = st + co * ROW + dz * 9 + dy * 3;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          dst[i * 27] = __uint_as_float(r0[i]);
          dst[i * 27 + 1] = __uint_as_float(r0[8 + i]);
          dst[i * 27 + 2] = __uint_as_float(r1[i]);
        }
      }
      __syncthreads();
      for (int co = warp; co < cout; co += 8) {
        float* dst = A.dw + ((size_t)(A.coOff + co) * cin + kk * 16 + half * 8) * 27;
#pragma unroll
        for (int r = 0; r < 7; r++)
          if (r * 32 + lane < 8 * 27) atomicAdd(dst + r * 32 + lane, st[co * ROW + r * 32 + lane]);
      }
      __syncthreads();
    }
    if (kk == 0) {
#pragma unroll
      for (int e = 0; e < 8; e++) {
        float v = bs[e];
        for (int o = 16; o >= D::CH; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane < D::CH) s_bias[warp][lane * 8 + e] = v;
        bs[e] = 0.f;
      }
      __syncthreads();
      if ((int)threadIdx.x < cout) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) v += s_bias[w][threadIdx.x];
        atomicAdd(A.db + A.coOff + threadIdx.x, v);
      }
    }
    fresh = true;
    fence_before();
    __syncthreads();                                 // accumulators free for the next run
  }
  if (s_abort && pending) mbar_wait(&mbar, phase);
  cp_async_wait_all();
  fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)D::TCOLS) : "memory");
}
cudaError_t launch_dw_tc(const ConvArgs& src, const bf16* dz, int cout, float* dw, float* db, int maxItems,
                         cudaStream_t s) {
  if (((src.c0 + src.c1) & 15) || (cout & 7) || cout > 128) return cudaErrorInvalidValue;
  static int smCount = 0;
  if (!smCount) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&smCount, cudaDevAttrMultiProcessorCount, dev); }
  if (maxItems <= 0) return cudaSuccess;
  for (int off = 0; off < cout; off += 64) {       // the A operand holds 64 output channels per pass
    DwTcArgs A{src, dz, std::min(64, cout - off), cout, off, dw, db};
    // the narrowest shape that holds the pass's channels: fewer rows are fewer bytes per MMA
    if (A.cout <= 16) k_dw_tc<16><<<std::min(maxItems, smCount * DwShape<16>::PERSM), 256, DwShape<16>::SMEM, s>>>(A);
    else if (A.cout <= 32) k_dw_tc<32><<<std::min(maxItems, smCount), 256, DwShape<32>::SMEM, s>>>(A);
    else k_dw_tc<64><<<std::min(maxItems, smCount), 256, DwShape<64>::SMEM, s>>>(A);
  }
  return cudaGetLastError();
}

template <int COUT> static cudaError_t set_smem() {
  return cudaFuncSetAttribute(k_conv3<COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, ConvShape<COUT>::SMEM);
}
cudaError_t conv3_init() {
  cudaError_t e;
  if ((e = set_smem<16>()) != cudaSuccess) return e;
  if ((e = set_smem<32>()) != cudaSuccess) return e;
  if ((e = set_smem<48>()) != cudaSuccess) return e;
  if ((e = set_smem<64>()) != cudaSuccess) return e;
  if ((e = set_smem<96>()) != cudaSuccess) return e;
  if ((e = set_smem<128>()) != cudaSuccess) return e;
  if ((e = set_smem<192>()) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_dw_tc<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, DwShape<16>::SMEM)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_dw_tc<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, DwShape<32>::SMEM)) != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_dw_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, DwShape<64>::SMEM);
}
int conv3_zt(int cout) {
  switch (cout) {
    case 16: return ConvShape<16>::ZT; case 32: return ConvShape<32>::ZT; case 48: return ConvShape<48>::ZT;
    case 64: return ConvShape<64>::ZT; case 96: return ConvShape<96>::ZT; case 128: return ConvShape<128>::ZT;
    case 192: return ConvShape<192>::ZT; default: return 0;
  }
}
size_t conv3_smem_bytes(int cout) {
  switch (cout) {
    case 16: return ConvShape<16>::SMEM; case 32: return ConvShape<32>::SMEM; case 48: return ConvShape<48>::SMEM;
    case 64: return ConvShape<64>::SMEM; case 96: return ConvShape<96>::SMEM; case 128: return ConvShape<128>::SMEM;
    case 192: return ConvShape<192>::SMEM; default: return 0;
  }
}
cudaError_t launch_conv3(const ConvArgs& a, int cout, int maxTiles, cudaStream_t s) {
  // the halo staging takes both 8-channel chunks of a slice from one source: splits are multiples of 16
  if (((a.c0 + a.c1) & 15) || (a.c0 & 15) || a.c0 + a.c1 <= 0 || (a.split & 15)) return cudaErrorInvalidValue;
  const int zt = conv3_zt(cout);
  if (!zt) return cudaErrorInvalidValue;
  // persistent: at most the CTAs the device holds at once, never more than the work items
  static int smCount = 0;
  if (!smCount) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&smCount, cudaDevAttrMultiProcessorCount, dev); }
  const size_t smb = conv3_smem_bytes(cout);
  const int perSM = (int)(233472 / (smb + 1024 + 256));
  const long long items = (long long)maxTiles * (kTZ / zt);
  const dim3 grid((unsigned)std::min<long long>(items, (long long)smCount * std::max(perSM, 1)));
  if (grid.x == 0) return cudaSuccess;
  const size_t sm = conv3_smem_bytes(cout);
  switch (cout) {
    case 16: k_conv3<16><<<grid, 256, sm, s>>>(a); break;
    case 32: k_conv3<32><<<grid, 256, sm, s>>>(a); break;
    case 48: k_conv3<48><<<grid, 256, sm, s>>>(a); break;
    case 64: k_conv3<64><<<grid, 256, sm, s>>>(a); break;
    case 96: k_conv3<96><<<grid, 256, sm, s>>>(a); break;
    case 128: k_conv3<128><<<grid, 256, sm, s>>>(a); break;
    case 192: k_conv3<192><<<grid, 256, sm, s>>>(a); break;
  }
  return cudaGetLastError();
}

}  // namespace unet
