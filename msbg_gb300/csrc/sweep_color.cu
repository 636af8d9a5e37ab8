// In-place colored sweeps (8-color / red-black) of applyChannelPdeFast, the
// streaming kernel.  Same schedule and arithmetic as sweep.cu (which keeps the
// generic gather kernel for the ping-pong schedule and FP64); this kernel is the
// one the in-place schedules use for FP32 / FP16 / uint16 storage.
//
// Per CTA one block.  Warp 0 stages the whole block and every halo piece it
// needs into shared memory with TMA bulk copies (cp.async.bulk) in chunks of 8
// planes, each chunk completing on its own mbarrier, so a CTA has the whole
// block (~77 KB for FP16 32^3) in flight at once and starts computing when the
// first chunk has landed.  Each thread owns a 4-voxel x-strip of every plane and
// marches through the block in z with a register window of three planes (rows
// y-1..y+1, columns x-1..x+4 of planes z-1, z, z+1; the three windows rotate
// roles, so no register moves).  It reads its strips straight from the staged
// data, so after the staging the warps never wait for each other.  Results go
// straight to global memory; the block is in shared memory before its first
// store, so the update is in place.
//
// Halo traffic.  The block payload is x-fastest (src/sbg.h:1816-1820), so the
// y- and z-neighbour rows/planes are contiguous but an x-neighbour column is one
// element per row.  Each channel therefore keeps, per value block, a cache of
// its two x-faces ([z][y]) and four z-parallel corner columns, written by the
// kernel whenever it updates a block and built once per applyChannelPdeFast
// call.  Same-color blocks are never 26-neighbours, so in a pass no block reads
// a cache entry that the pass writes.  Every piece is a multiple of 16 bytes at
// a 16-byte aligned address, as cp.async.bulk requires.
#include <stddef.h>
#include <string.h>

#include <type_traits>

#include "internal.cuh"
#include "sweep_common.cuh"

namespace msbg {

template <typename T> struct Vec4T;
template <> struct Vec4T<float> { using V = float4; };
template <> struct Vec4T<__half> { using V = uint2; };
template <> struct Vec4T<uint16_t> { using V = uint2; };

template <typename T>
__device__ __forceinline__ typename Vec4T<T>::V pack4(const float o[4]) {
  typename Vec4T<T>::V v;
  if constexpr (sizeof(T) == 4) {
    v.x = o[0]; v.y = o[1]; v.z = o[2]; v.w = o[3];
  } else if constexpr (std::is_same<T, __half>::value) {
    // two round-to-nearest-even conversions of a pair each (the same rounding as
    // __float2half_rn per value)
    const __half2 lo = __floats2half2_rn(o[0], o[1]), hi = __floats2half2_rn(o[2], o[3]);
    v.x = *reinterpret_cast<const uint32_t *>(&lo);
    v.y = *reinterpret_cast<const uint32_t *>(&hi);
  } else {
    T *e = reinterpret_cast<T *>(&v);
#pragma unroll
    for (int k = 0; k < 4; k++) Store<T>::storeRNE(e + k, o[k]);
  }
  return v;
}

template <typename T, int BS>
struct ColorSweep {
  static constexpr int NT = BS * BS / 4;     // threads: one 4-voxel x-strip of every plane each
  static constexpr int SPR = BS / 4;         // strips per row
  static constexpr int64_t VPB = (int64_t)BS * BS * BS;
  static constexpr int FACE = BS * BS;       // per x-face
  static constexpr int CORN = BS;            // per corner column
  static constexpr int CZ = 8;               // planes per TMA chunk (corner pieces >= 16 B)
  static constexpr int NCH = BS / CZ;        // chunks (one mbarrier each)
  static constexpr int NCC = 1 + 2 + 2 * CZ + 4 + 5;  // copy slots per chunk (<= 32)
};

// Raw (storage-type) staging of one block and its halo in shared memory.
template <typename T, int BS>
struct RawTile {
  T blk[BS * BS * BS];   // own block [z][y][x]
  T xf[2][BS * BS];      // column x=-1 (0) and x=BS (1), [z][y]
  T yr[2][BS * BS];      // row y=-1 (0) and y=BS (1), [z][x]
  alignas(16) T er[16];  // the empty value (source of every fill from an empty block)
  // from here on not staged by the fast 7-point form (facesOnly)
  T zpl[2][BS * BS];     // plane z=-1 (0) and z=BS (1), [y][x]
  T cn[4][BS];           // corner columns (x=-1|BS, y=-1|BS), k = (dx>0) + 2*(dy>0), [z]
  T zh[2][4][BS];        // planes -1 / BS: x=-1 row, x=BS row (over y), y=-1 row, y=BS row (over x)
};

__device__ __forceinline__ uint32_t smemAddr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbarInit(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarExpectTx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbarTryWait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// 1-D TMA bulk copy global -> shared, completion counted in bytes on `bar`.
__device__ __forceinline__ void bulkG2S(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smemAddr(dst)),
      "l"(src), "r"(bytes), "r"(smemAddr(bar))
      : "memory");
}

// Bounded wait on phase 0 of a chunk barrier.  Returns false after the limit.
__device__ __forceinline__ bool waitChunk(uint64_t *bar) {
  for (int it = 0; it < (1 << 22); it++)
    if (mbarTryWait(bar, 0)) return true;
  return false;
}

struct ColorArgs {
  const int32_t *bids;
  const int32_t *slot;
  void *payload;
  void *faces;    // [slot][2][BS(z)][BS(y)]  x=0 face, x=BS-1 face
  void *corners;  // [slot][4][BS(z)]  k = (x==BS-1) + 2*(y==BS-1)
  int nbx, nby, nbz;
  float emptyValue;
  int *status;    // bit 0: a chunk wait timed out
  SweepParams p;
};

// The fast 7-point form: a thread needs its own four voxels of the planes z=-1 and z=BS, which
// it reads from global memory, and no corner.  Without those pieces (4.9 KB) three CTAs of a
// 32^3 block share an SM (72 registers): FP16, 514 M voxels, 10 iterations, 6.12 -> 4.92 ms.
// The same for MCF (80 registers, planes from global memory) was slower at every size: 216 / 512 /
// 4096 blocks a pass 19.7 -> 26.6, 38.2 -> 45.5, 241 -> 252 us.
template <typename T, int FK>
constexpr bool facesOnly() { return sizeof(T) == 2 && (FK & ~FK_CLAMP) == K_JACOBI; }

// Copy slot c of chunk k (planes k*CZ .. k*CZ+CZ-1) of a block's tile: fills
// (dst, src, bytes) and returns true when the piece exists (its source block is a
// value block).  Chunk 0 also carries plane z=-1, the last chunk plane z=BS.
template <typename T, int BS, int FK>
__device__ __forceinline__ bool tileCopy(int k, int c, const int *nbs, const ColorArgs &a,
                                         RawTile<T, BS> &t, void *&dst, const void *&src,
                                         uint32_t &bytes) {
  using C = ColorSweep<T, BS>;
  constexpr int CZ = C::CZ;
  const T *pay = (const T *)a.payload;
  const T *faces = (const T *)a.faces;
  const T *corn = (const T *)a.corners;
  auto NB = [&](int dx, int dy, int dz) { return nbs[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)]; };
  auto blkp = [&](int s) { return pay + (int64_t)s * C::VPB; };
  const int z0 = k * CZ;
  if (c == 0) {  // own planes of the chunk
    dst = t.blk + (int64_t)z0 * BS * BS;
    src = blkp(NB(0, 0, 0)) + (int64_t)z0 * BS * BS;
    bytes = CZ * BS * BS * sizeof(T);
    return true;
  }
  c -= 1;
  if (c < 2) {  // x-neighbour face rows from the cache: its x=BS-1 face for dx=-1, x=0 for dx=+1
    const int s = NB(c ? 1 : -1, 0, 0);
    if (s < 0) return false;
    dst = t.xf[c] + z0 * BS;
    src = faces + ((int64_t)s * 2 + (c ? 0 : 1)) * C::FACE + z0 * BS;
    bytes = CZ * BS * sizeof(T);
    return true;
  }
  c -= 2;
  if (c < 2 * CZ) {  // y-neighbour rows, one per plane
    const int side = c / CZ, z = z0 + c % CZ;
    const int s = NB(0, side ? 1 : -1, 0);
    if (s < 0) return false;
    dst = t.yr[side] + z * BS;
    src = blkp(s) + ((int64_t)z * BS + (side ? 0 : BS - 1)) * BS;
    bytes = BS * sizeof(T);
    return true;
  }
  c -= 2 * CZ;
  if constexpr (facesOnly<T, FK>()) return false;
  if (c < 4) {  // corner-column segments of the 4 diagonal neighbours in the block's z-layer
    const int dx = (c & 1) ? 1 : -1, dy = (c & 2) ? 1 : -1;
    const int s = NB(dx, dy, 0);
    if (s < 0) return false;
    const int kSrc = (dx < 0 ? 1 : 0) + 2 * (dy < 0 ? 1 : 0);
    dst = t.cn[c] + z0;
    src = corn + ((int64_t)s * 4 + kSrc) * C::CORN + z0;
    bytes = CZ * sizeof(T);
    return true;
  }
  c -= 4;
  // z-halo plane pieces: first chunk -> plane -1, last chunk -> plane BS
  const bool first = k == 0, last = k == C::NCH - 1;
  if (!first && !last) return false;
  const int zi = first ? 0 : 1;
  if (first && last) return false;  // (single-chunk blocks are not instantiated)
  const int dz = zi ? 1 : -1;
  const int zSrc = zi ? 0 : BS - 1;
  if (c == 0) {
    const int s = NB(0, 0, dz);
    if (s < 0) return false;
    dst = t.zpl[zi];
    src = blkp(s) + (int64_t)zSrc * BS * BS;
    bytes = BS * BS * sizeof(T);
    return true;
  }
  const int j = c - 1;  // 0 x=-1, 1 x=BS (over y), 2 y=-1, 3 y=BS (over x)
  dst = t.zh[zi][j];
  bytes = BS * sizeof(T);
  if (j < 2) {
    const int dx = j ? 1 : -1;
    const int s = NB(dx, 0, dz);
    if (s < 0) return false;
    src = faces + ((int64_t)s * 2 + (dx < 0 ? 1 : 0)) * C::FACE + zSrc * BS;
  } else {
    const int dy = j == 3 ? 1 : -1;
    const int s = NB(0, dy, dz);
    if (s < 0) return false;
    src = blkp(s) + ((int64_t)zSrc * BS + (dy < 0 ? BS - 1 : 0)) * BS;
  }
  return true;
}

template <typename T, int BS>
constexpr size_t rawTileBytes() {
  return (sizeof(RawTile<T, BS>) + 15) & ~size_t(15);
}

template <typename T, int BS, int FK>
constexpr size_t colorSmemBytes() {
  using Tile = RawTile<T, BS>;
  if (facesOnly<T, FK>()) return offsetof(Tile, zpl);
  return rawTileBytes<T, BS>();
}

// FK: the stencil, fixed at compile time.  0 = any kind in the reference's
// operation order (computeStrip); K_MCF / K_JACOBI = the fast forms, plus
// FK_CLAMP when the result is clamped to [0,1]; K_MCF | FK_EXACT = MCF in the
// reference's order on packed operations (mcfExactStrip).
//
// ZG z-groups of NT threads share the staged block, each marching BS / ZG of its planes
// (zGroups has the rule and its measurements).  A small pass is bound by the latency of one
// block, not by bandwidth or issue: with one group, 64 threads march a 16^3 block.
//
// The passes of a call are launched with programmatic serialization: a pass's CTAs look up
// their blocks and neighbours and prepare their copies while the previous pass drains, and
// wait for its writes (griddepcontrol.wait) before the first copy.  Only warp 0 waits (all warps
// where facesOnly reads planes directly): what the other warps read arrives through its copies,
// and what they write comes after.  The
// trigger stands at the end of a CTA: at its start, the next pass's CTAs took places on the
// SMs early and unevenly (216 blocks: 13.4 -> 16.9 us; at the end 11.2 us).
template <typename T, int BS, int FK, int ZG>
constexpr int sweepCtas() {  // resident CTAs to leave registers for
  constexpr int nt = ColorSweep<T, BS>::NT * ZG;
  if ((FK & ~FK_CLAMP) == K_JACOBI && BS == 16 && ZG == 4) return 4;
  return facesOnly<T, FK>() && BS == 32 ? 3 : nt <= 256 ? 512 / nt : 1;
}

template <typename T, int BS, int FK, int ZG>
__global__ void __launch_bounds__(ColorSweep<T, BS>::NT *ZG, sweepCtas<T, BS, FK, ZG>()) kSweepColor(ColorArgs a) {
  using C = ColorSweep<T, BS>;
  using V4 = typename Vec4T<T>::V;
  constexpr int CZ = C::CZ, NCH = C::NCH;
  constexpr int PZ = BS / ZG;  // planes of a z-group
  extern __shared__ __align__(128) unsigned char dynSmem[];
  RawTile<T, BS> &t = *reinterpret_cast<RawTile<T, BS> *>(dynSmem);
  __shared__ int nbs[27];
  __shared__ __align__(8) uint64_t bar[NCH];

  const int tid = threadIdx.x;
  const int bid = a.bids[blockIdx.x];
  const int64_t nxy = (int64_t)a.nbx * a.nby;
  const int bz = (int)(bid / nxy), by = (int)((bid / a.nbx) % a.nby), bx = (int)(bid % a.nbx);
  if (tid < 27) {
    const int dx = tid % 3 - 1, dy = (tid / 3) % 3 - 1, dz = tid / 9 - 1;
    const int x = bx + dx, y = by + dy, z = bz + dz;
    int s = -2;  // outside the domain
    if (x >= 0 && y >= 0 && z >= 0 && x < a.nbx && y < a.nby && z < a.nbz)
      s = a.slot[(int64_t)z * nxy + (int64_t)y * a.nbx + x];
    nbs[tid] = (s < 0 && s != -2) ? -1 : s;  // -1: constant empty block
  }
  if (tid < NCH) mbarInit(&bar[tid], 1);
  if (tid == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (tid < 16) {
    T e;
    if constexpr (sizeof(T) == 4) e = a.emptyValue; else Store<T>::storeRNE(&e, a.emptyValue);
    t.er[tid] = e;
  }
  __syncthreads();
  if (tid < 32) {
    // warp 0, lane-parallel over a chunk's copies: announce the chunk's bytes, then issue.
    // A small pass prepares all chunks while the previous pass drains; a 32^3 block, whose
    // passes are bound by throughput, issues each chunk as soon as it is known (preparing
    // all four first costs Jacobi 1.4% on 498 M voxels).
    constexpr bool PRE = BS == 16;
    void *d[NCH];
    const void *src[NCH];
    uint32_t b[NCH];
    auto prepare = [&](int k) {
      const bool has = tid < C::NCC && tileCopy<T, BS, FK>(k, tid, nbs, a, t, d[k], src[k], b[k]);
      if (!has) b[k] = 0;
      const uint32_t tot = __reduce_add_sync(0xffffffffu, b[k]);
      if (tid == 0) mbarExpectTx(&bar[k], tot);
      __syncwarp();
    };
    if constexpr (PRE) {
#pragma unroll
      for (int k = 0; k < NCH; k++) prepare(k);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int k = 0; k < NCH; k++) {
      if constexpr (!PRE) prepare(k);
      if (b[k]) bulkG2S(d[k], src[k], b[k], &bar[k]);
    }
  }

  const int ownSlot = nbs[13];
  const int zg = tid / C::NT, gt = tid % C::NT;
  const int zFirst = zg * PZ;                            // first plane of the z-group
  const int ty = gt / C::SPR, tx = (gt % C::SPR) * 4;    // this thread's strip
  // planes are consumed in increasing order (plane -1 needs chunk 0, plane BS comes after
  // plane BS-1), so one counter of the planes known to have landed
  // replaces per-chunk flags
  int readyPlanes = 0;
  bool timedOut = false;
  auto need = [&](int p) {
    if (p >= readyPlanes) {
      if (!waitChunk(&bar[p / CZ])) timedOut = true;
      readyPlanes = (p / CZ + 1) * CZ;
    }
  };

  constexpr int FKK = FK & ~FK_CLAMP;
  using PW = std::conditional_t<
      FKK == K_MCF, PlaneMcf,
      std::conditional_t<FKK == K_JACOBI, PlaneJac, std::conditional_t<FKK == (K_MCF | FK_EXACT), PlaneMcfX, PlaneRaw>>>;
  T *outp = (T *)a.payload + (int64_t)ownSlot * C::VPB + ty * BS + tx;
  // x-face / corner cache entries this thread maintains (x = 0 or BS-1 strips)
  const bool faceThread = tx == 0 || tx == BS - 4;
  const int kx = tx == 0 ? 0 : 1;
  T *facep = (T *)a.faces + ((int64_t)ownSlot * 2 + kx) * C::FACE + ty;
  const bool cornThread = faceThread && (ty == 0 || ty == BS - 1);
  T *cornp = (T *)a.corners + ((int64_t)ownSlot * 4 + kx + 2 * (ty == 0 ? 0 : 1)) * C::CORN;
  PW Wa, Wb, Wc;

  auto emit = [&](int z, const PW &Wm, const PW &W0, const PW &Wp) {
    float out[4];
    constexpr bool CL = (FK & FK_CLAMP) != 0;
    if constexpr (FKK == K_MCF) mcfFastStrip<CL>(Wm, W0, Wp, a.p.dt, out);
    else if constexpr (FKK == (K_MCF | FK_EXACT)) mcfExactStrip(Wm, W0, Wp, a.p.dt, a.p.negZero, a.p.constr01, out);
    else if constexpr (FKK == K_JACOBI) jacobiFastStrip<CL>(Wm, W0, Wp, a.p.dt, out);
    else computeStrip(Wm.w, W0.w, Wp.w, a.p, out);
    const V4 pk = pack4<T>(out);
    *reinterpret_cast<V4 *>(outp + z * BS * BS) = pk;
    T v;
    if constexpr (sizeof(T) == 4) {
      v = kx ? pk.w : pk.x;
    } else {
      const uint16_t bits = kx ? (uint16_t)(pk.y >> 16) : (uint16_t)(pk.x & 0xffffu);
      v = *reinterpret_cast<const T *>(&bits);
    }
    if (faceThread) facep[z * BS] = v;
    if (cornThread) cornp[z] = v;
  };
  // Rows are read where they are staged: a thread reads its own strip of rows y-1, y, y+1 as
  // one 8- or 16-byte load each, widens them (exactly), and takes the values beside the strip
  // from the neighbouring lanes (block sides: one narrow load more).  A ring of FP32 rows in
  // shared memory, converted once per warp, costs 26 wavefronts a plane and warp where FP16
  // takes 8 to 11 here and FP32 14 to 17, and a barrier and a round trip per plane.  The march
  // is unrolled by three, which saves the moves of the rotating windows.  Measured against the
  // ring, us a pass: FP16 32^3 blocks, 512 a pass, exact MCF 66.9 -> 52.2, fast MCF 41.6 ->
  // 37.9, Jacobi 32.1 -> 22.6; 16^3 blocks, 1000 a pass, exact MCF (FP32) 22.8 -> 18.8, fast
  // MCF 22.5 -> 14.4, Jacobi 15.0 -> 10.8; 64 blocks 6.2 -> 5.3, 5.6 -> 4.7, 4.9 -> 4.2.
  //
  // The thread's rows y-1, y, y+1 of plane p at (byte offset in shared memory) rowX + p *
  // stepX, and the value beyond the block's side, in the lanes that need one, at edgeX.
  // Offsets rather than pointers: a source is a 32-bit word, a step another.
  const bool atFirst = tx == 0, atLast = tx == BS - 4;
  const uint32_t tb = smemAddr(&t);
  auto offOf = [&](const void *q) { return smemAddr(q) - tb; };
  struct Walk {
    uint32_t at, step;
  };
  // row y of the own block, its y-neighbour, the empty row, or (domain boundary) the nearest own row
  auto rowSrc = [&](int y) -> Walk {
    if (y >= 0 && y < BS) return {offOf(t.blk + y * BS + tx), BS * BS * sizeof(T)};
    const int side = y < 0 ? 0 : 1, s = nbs[9 + (side ? 2 : 0) * 3 + 1];
    if (s >= 0) return {offOf(t.yr[side] + tx), BS * sizeof(T)};
    if (s == -1) return {offOf(t.er), 0u};
    return {offOf(t.blk + (side ? BS - 1 : 0) * BS + tx), BS * BS * sizeof(T)};
  };
  auto edgeSrc = [&](int y) -> Walk {
    if (!atFirst && !atLast) return {offOf(t.er), 0u};
    const int side = atFirst ? 0 : 1, dx = side ? 1 : -1, xc = side ? BS - 1 : 0;
    if (y >= 0 && y < BS) {
      const int s = nbs[9 + 3 + (dx + 1)];
      if (s >= 0) return {offOf(t.xf[side] + y), BS * sizeof(T)};
      if (s == -1) return {offOf(t.er), 0u};
      return {offOf(t.blk + y * BS + xc), BS * BS * sizeof(T)};
    }
    const int dy = y < 0 ? -1 : 1, yc = dy < 0 ? 0 : BS - 1, s = nbs[9 + (dy + 1) * 3 + (dx + 1)];
    if (s >= 0) return {offOf(t.cn[(dx > 0 ? 1 : 0) + 2 * (dy > 0 ? 1 : 0)]), (uint32_t)sizeof(T)};
    if (s == -1) return {offOf(t.er), 0u};
    return {offOf(t.blk + yc * BS + xc), BS * BS * sizeof(T)};
  };
  constexpr bool kCorners = FKK != K_JACOBI;  // the 7-point form reads no edge of rows y-1, y+1
  const Walk wm = rowSrc(ty - 1), wp = rowSrc(ty + 1), ec = edgeSrc(ty);
  const Walk em = kCorners ? edgeSrc(ty - 1) : Walk{0, 0}, ep = kCorners ? edgeSrc(ty + 1) : Walk{0, 0};
  const uint32_t rowC = offOf(t.blk + ty * BS + tx);
  using E = std::conditional_t<sizeof(T) == 4, float, uint16_t>;  // an edge value's bits
  auto ldsRow = [&](uint32_t off) {
    V4 v;
    if constexpr (sizeof(T) == 4)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(tb + off));
    else
      asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(tb + off));
    return v;
  };
  auto ldsEdge = [&](uint32_t off) {
    E v;
    if constexpr (sizeof(T) == 4) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(tb + off));
    else asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(tb + off));
    return v;
  };
  struct Raw {
    V4 m, c, p;
    E em, ec, ep;
  };
  auto fetchIn = [&](int p, Raw &r) {  // plane 0 .. BS-1
    need(p);
    r.m = ldsRow(wm.at + p * wm.step);
    r.c = ldsRow(rowC + p * (uint32_t)(BS * BS * sizeof(T)));
    r.p = ldsRow(wp.at + p * wp.step);
    r.ec = ldsEdge(ec.at + p * ec.step);
    if constexpr (kCorners) {
      r.em = ldsEdge(em.at + p * em.step);
      r.ep = ldsEdge(ep.at + p * ep.step);
    }
  };
  V4 zOut[2];  // facesOnly: the strip's voxels of planes -1 and BS, from the blocks below and above
  if constexpr (facesOnly<T, FK>()) {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous pass wrote them
#pragma unroll
    for (int zi = 0; zi < 2; zi++) {
      const int s = nbs[zi * 18 + 4];
      if (s >= 0)
        zOut[zi] = __ldcg(reinterpret_cast<const V4 *>((const T *)a.payload + (int64_t)s * C::VPB +
                                                          ((zi ? 0 : BS - 1) * BS + ty) * BS + tx));
      else if (s == -1) zOut[zi] = ldsRow(offOf(t.er));
    }
  }
  auto fetchOut = [&](int p, Raw &r) {  // z-halo plane -1 or BS; the stencils read no edge of its rows y-1, y+1
    if constexpr (facesOnly<T, FK>()) {  // and the 7-point form only the strip itself
      const int zi = p < 0 ? 0 : 1, pc = zi ? BS - 1 : 0;
      need(pc);
      r.c = nbs[zi * 18 + 4] == -2 ? ldsRow(offOf(t.blk + (pc * BS + ty) * BS + tx)) : zOut[zi];
      r.m = r.p = r.c;
      r.em = r.ec = r.ep = 0;
      return;
    }
    const int zi = p < 0 ? 0 : 1, dzb = zi ? 1 : -1, pc = zi ? BS - 1 : 0;
    need(pc);
    auto row = [&](int y) -> V4 {
      const T *q;
      if (y >= 0 && y < BS) {
        const int s = nbs[(dzb + 1) * 9 + 4];
        q = s >= 0 ? t.zpl[zi] + y * BS + tx : s == -1 ? t.er : t.blk + (pc * BS + y) * BS + tx;
      } else {
        const int dy = y < 0 ? -1 : 1, yc = dy < 0 ? 0 : BS - 1, s = nbs[(dzb + 1) * 9 + (dy + 1) * 3 + 1];
        q = s >= 0 ? t.zh[zi][dy < 0 ? 2 : 3] + tx : s == -1 ? t.er : t.blk + (pc * BS + yc) * BS + tx;
      }
      return ldsRow(offOf(q));
    };
    r.m = row(ty - 1);
    r.c = row(ty);
    r.p = row(ty + 1);
    const int side = atFirst ? 0 : 1, s = nbs[(dzb + 1) * 9 + 3 + (side ? 2 : 0)];
    r.ec = ldsEdge(offOf(s >= 0 ? t.zh[zi][side] + ty : s == -1 ? t.er : t.blk + (pc * BS + ty) * BS + (side ? BS - 1 : 0)));
    r.em = r.ep = 0;
  };
  // u16 to float without the slow conversion pipe: u under the exponent of 2^23 is 2^23 + u
  auto u16Val = [](uint32_t w, uint32_t sel) {
    return __fmul_rn(__fsub_rn(__uint_as_float(__byte_perm(w, 0x4b000000u, sel)), 8388608.0f), kU16ToF);
  };
  auto unpackRow = [&](const V4 &v, float o[4]) {
    if constexpr (sizeof(T) == 4) {
      o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else if constexpr (std::is_same<T, uint16_t>::value) {
      o[0] = u16Val(v.x, 0x7610); o[1] = u16Val(v.x, 0x7632);
      o[2] = u16Val(v.y, 0x7610); o[3] = u16Val(v.y, 0x7632);
    } else {
      const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
      const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
      o[0] = lo.x; o[1] = lo.y; o[2] = hi.x; o[3] = hi.y;
    }
  };
  auto edgeVal = [&](E v) {
    if constexpr (sizeof(T) == 4) return v;
    else if constexpr (std::is_same<T, uint16_t>::value) return u16Val(v, 0x7610);
    else return __half2float(__ushort_as_half(v));
  };
  auto plane = [&](const Raw &r, PW &W) {
    StripRows s;
    unpackRow(r.m, s.m);
    unpackRow(r.c, s.c);
    unpackRow(r.p, s.p);
    s.ec = edgeVal(r.ec);
    s.em = s.ep = 0.0f;
    if constexpr (kCorners) { s.em = edgeVal(r.em); s.ep = edgeVal(r.ep); }
    planeOf(s, atFirst, atLast, W);
  };
  auto fetch = [&](int p, Raw &r) {
    if (p < 0 || p >= BS) fetchOut(p, r);
    else fetchIn(p, r);
  };
  Raw r;
  fetch(zFirst - 1, r);
  plane(r, Wa);
  fetchIn(zFirst, r);
  plane(r, Wb);
  fetch(zFirst + 1, r);
  plane(r, Wc);
  // the rows of plane z+2 are read while plane z is computed, and become the window that
  // plane z-1 leaves
  auto step = [&](int z, PW &A, PW &B, PW &Cw) {
    const bool more = z + 1 < zFirst + PZ;
    if (more) fetch(z + 2, r);
    emit(z, A, B, Cw);
    if (more) plane(r, A);
  };
  // the window roles rotate every plane: (a,b,c) -> (b,c,a)
#pragma unroll 1
  for (int z = zFirst; z + 3 <= zFirst + PZ; z += 3) {
    step(z, Wa, Wb, Wc);
    step(z + 1, Wb, Wc, Wa);
    step(z + 2, Wc, Wa, Wb);
  }
  constexpr int PT = PZ - PZ % 3;
  if constexpr (PZ % 3 > 0) step(zFirst + PT, Wa, Wb, Wc);
  if constexpr (PZ % 3 > 1) step(zFirst + PT + 1, Wb, Wc, Wa);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // let the next pass in
  if (timedOut) {
    atomicOr(a.status, 1);
    for (int k = 0; k < NCH; k++) waitChunk(&bar[k]);  // no copy may land after exit
  }
}

// Builds the x-face and corner caches of every value block from the payload.
template <typename T, int BS>
__global__ void kExtractFaces(const T *__restrict__ pay, int64_t nAct, T *__restrict__ faces,
                              T *__restrict__ corners) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // (slot, z, y)
  if (i >= nAct * BS * BS) return;
  const int64_t s = i / (BS * BS);
  const int z = (int)((i / BS) % BS), y = (int)(i % BS);
  const T *row = pay + s * (int64_t)BS * BS * BS + ((int64_t)z * BS + y) * BS;
  faces[(s * 2 + 0) * BS * BS + z * BS + y] = row[0];
  faces[(s * 2 + 1) * BS * BS + z * BS + y] = row[BS - 1];
  if (y == 0 || y == BS - 1) {
    const int ky = y == 0 ? 0 : 1;
    corners[(s * 4 + 0 + 2 * ky) * BS + z] = row[0];
    corners[(s * 4 + 1 + 2 * ky) * BS + z] = row[BS - 1];
  }
}

// the stencil forms of kSweepColor: any kind in the reference's operation order, the fast
// forms with and without the clamp, and MCF in the reference's order
enum { kKernGeneric, kKernMcf, kKernMcfClamp, kKernJacobi, kKernJacobiClamp, kKernMcfExact };

// z-groups per CTA of a pass of n blocks.  A pass is as long as one block takes while its
// CTAs fit the chip at once (152 SMs), and more groups shorten a block; they cost every
// group two more planes to read, so a pass of several waves takes fewer.  Two 4-group or four
// 2-group CTAs (registers) share an SM, four 4-group ones of the fast Jacobi.  Measured, us a
// pass for 1 / 2 / 4 groups (FP32, 16^3 blocks): exact MCF 9.4 / 7.3 / 5.2 at 64 blocks, 10.2 /
// 7.9 / 6.2 at 216, 12.5 / 10.6 / 12.6 at 512, 14.9 / 17.1 / 18.5 at 729; fast MCF 6.8 / 5.7 /
// 4.6 at 64, 9.3 / 8.6 / 11.0 at 512, 11.2 / 14.4 / 16.9 at 729; fast Jacobi for 1 / 4: 5.3 /
// 4.1 at 64, 6.7 / 5.6 at 512, 8.2 / 10.5 at 729.  On 32^3 blocks the exact form takes two
// groups up to one block per SM (FP16, 64 blocks: 18.4 -> 15.7; 216 blocks: 26.7 against 32.0)
// and, with FP32 storage, whose 145 KB of staging leave one CTA per SM, always (76.3 -> 67.9 at
// 512 blocks).
template <typename T, int BS>
static int zGroups(int n, int ki) {
  constexpr int kSm = 152;
  if constexpr (BS == 16) {
    if (n <= 2 * kSm) return 4;
    if (n > 4 * kSm || ki == kKernGeneric) return 1;
    return ki == kKernJacobi || ki == kKernJacobiClamp ? 4 : 2;
  } else {
    return ki == kKernMcfExact && (sizeof(T) == 4 || n <= kSm) ? 2 : 1;
  }
}

template <typename T, int BS, int FK, int ZG>
static cudaError_t launchPassT(const ColorArgs &a, unsigned blocks, cudaStream_t st) {
  const auto kern = kSweepColor<T, BS, FK, ZG>;
  constexpr size_t smem = colorSmemBytes<T, BS, FK>();
  static SmemOptIn optIn;
  const cudaError_t e = optIn((const void *)kern, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(ColorSweep<T, BS>::NT * ZG);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

template <typename T, int BS>
static cudaError_t launchPass(const ColorArgs &a, int ki, int zg, unsigned blocks, cudaStream_t st) {
  constexpr int ZS = BS == 16 ? 4 : 1;  // the small passes' groups (generic and fast forms)
  switch (ki) {
    case kKernMcf:
      if constexpr (ZS > 1) if (zg == 2) return launchPassT<T, BS, K_MCF, 2>(a, blocks, st);
      return zg > 1 ? launchPassT<T, BS, K_MCF, ZS>(a, blocks, st) : launchPassT<T, BS, K_MCF, 1>(a, blocks, st);
    case kKernMcfClamp:
      if constexpr (ZS > 1) if (zg == 2) return launchPassT<T, BS, K_MCF | FK_CLAMP, 2>(a, blocks, st);
      return zg > 1 ? launchPassT<T, BS, K_MCF | FK_CLAMP, ZS>(a, blocks, st)
                    : launchPassT<T, BS, K_MCF | FK_CLAMP, 1>(a, blocks, st);
    case kKernJacobi:
      return zg > 1 ? launchPassT<T, BS, K_JACOBI, ZS>(a, blocks, st) : launchPassT<T, BS, K_JACOBI, 1>(a, blocks, st);
    case kKernJacobiClamp:
      return zg > 1 ? launchPassT<T, BS, K_JACOBI | FK_CLAMP, ZS>(a, blocks, st)
                    : launchPassT<T, BS, K_JACOBI | FK_CLAMP, 1>(a, blocks, st);
    case kKernMcfExact:
      if (zg == ZS && ZS > 1) return launchPassT<T, BS, K_MCF | FK_EXACT, ZS>(a, blocks, st);
      return zg == 2 ? launchPassT<T, BS, K_MCF | FK_EXACT, 2>(a, blocks, st)
                     : launchPassT<T, BS, K_MCF | FK_EXACT, 1>(a, blocks, st);
    default: return zg > 1 ? launchPassT<T, BS, 0, ZS>(a, blocks, st) : launchPassT<T, BS, 0, 1>(a, blocks, st);
  }
}

template <typename T, int BS>
static int runColorT(msbg_gpu_ctx *ctx, Channel &c, bool exact, bool color8, int nIter,
                     const SweepParams &p, const int32_t *bids, const int *cs) {
  const int64_t nAct = ctx->nActive;
  if (nAct == 0) return MSBG_GPU_OK;
  const size_t faceBytes = (size_t)nAct * (2 * BS * BS + 4 * BS) * sizeof(T);
  if (c.cacheBytes < faceBytes) {
    if (c.cache) MSBG_CUDA(ctx, cudaFree(c.cache));
    c.cache = nullptr;
    c.cacheBytes = 0;
    MSBG_CUDA(ctx, cudaMalloc(&c.cache, faceBytes));
    c.cacheBytes = faceBytes;
  }
  T *faces = (T *)c.cache;
  T *corners = faces + (size_t)nAct * 2 * BS * BS;
  const int64_t n = nAct * BS * BS;
  MSBG_LAUNCH(ctx, (kExtractFaces<T, BS>), gridFor(n, 256), 256, 0, (const T *)c.d, nAct, faces, corners);
  ColorArgs a;
  a.slot = ctx->dSlot;
  a.payload = c.d;
  a.faces = faces;
  a.corners = corners;
  a.nbx = ctx->nbx; a.nby = ctx->nby; a.nbz = ctx->nbz;
  a.emptyValue = 0.0f;
  a.status = ctx->dStatus;
  a.p = p;
  int ki = kKernGeneric;
  if (p.kind == K_MCF) ki = exact ? kKernMcfExact : p.constr01 ? kKernMcfClamp : kKernMcf;
  else if (p.kind == K_JACOBI && !exact) ki = p.constr01 ? kKernJacobiClamp : kKernJacobi;
  static const int rbOrder[2][4] = {{1, 2, 4, 7}, {0, 3, 5, 6}};
  int zgOf[8];
  for (int c8 = 0; c8 < 8; c8++) zgOf[c8] = zGroups<T, BS>(cs[c8 + 1] - cs[c8], ki);
  int nLaunch = 0;
  for (int pass = 0; pass < 8; pass++) nLaunch += cs[pass + 1] > cs[pass];
  nLaunch *= nIter;
  if (nLaunch == 0) return MSBG_GPU_OK;
  auto launchAll = [&](cudaStream_t st) -> int {
    for (int it = 0; it < nIter; it++) {
      for (int pass = 0; pass < 8; pass++) {
        const int col = color8 ? pass : rbOrder[pass / 4][pass % 4];
        const int cnt = cs[col + 1] - cs[col];
        if (cnt <= 0) continue;
        a.bids = bids + cs[col];
        if (launchPass<T, BS>(a, ki, zgOf[col], (unsigned)cnt, st) != cudaSuccess) return MSBG_GPU_ERR_CUDA;
      }
    }
    return MSBG_GPU_OK;
  };
  // The colour passes go out as one CUDA graph, captured the first time a call
  // presents these launches (kernel, arguments, grids) and replayed after that: a
  // small layout's passes (a few hundred blocks each) are otherwise bound by the
  // launches themselves.  A context whose stream is being captured by its caller
  // launches them directly.
  cudaStreamCaptureStatus outer = cudaStreamCaptureStatusNone;
  MSBG_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &outer));
  if (outer != cudaStreamCaptureStatusNone) {
    if (launchAll(ctx->stream)) return fail(ctx, MSBG_GPU_ERR_CUDA, "sweep: launch failed");
    ctx->launches += nLaunch;
    return MSBG_GPU_OK;
  }
  std::vector<unsigned char> key;
  auto put = [&key](const auto &v) {
    const unsigned char *b = reinterpret_cast<const unsigned char *>(&v);
    key.insert(key.end(), b, b + sizeof(v));
  };
  put(reinterpret_cast<const void *>(&runColorT<T, BS>)); put(ki); put(bids); put(a.slot); put(a.payload); put(a.faces); put(a.corners);
  put(a.nbx); put(a.nby); put(a.nbz); put(a.emptyValue); put(a.status);
  put(p.kind); put(p.constr01); put(p.dt); put(p.anisAlpha); put(nIter); put(color8);
  for (int i = 0; i < 9; i++) put(cs[i]);
  cudaGraphExec_t exec = nullptr;
  for (size_t i = 0; i < c.sweepGraphs.size(); i++)
    if (c.sweepGraphs[i].key == key) {
      CachedGraph hit = std::move(c.sweepGraphs[i]);
      c.sweepGraphs.erase(c.sweepGraphs.begin() + i);
      c.sweepGraphs.push_back(std::move(hit));
      exec = c.sweepGraphs.back().exec;
      break;
    }
  if (!exec) {
    if (!ctx->captureStream) MSBG_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->captureStream, cudaStreamNonBlocking));
    MSBG_CUDA(ctx, cudaStreamBeginCapture(ctx->captureStream, cudaStreamCaptureModeThreadLocal));
    const int lrc = launchAll(ctx->captureStream);
    cudaGraph_t graph = nullptr;
    const cudaError_t ee = cudaStreamEndCapture(ctx->captureStream, &graph);
    if (lrc || ee != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      return fail(ctx, MSBG_GPU_ERR_CUDA, "sweep: capturing the colour passes failed");
    }
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return cudaFail(ctx, ie, "cudaGraphInstantiate");
    if (c.sweepGraphs.size() >= 4) {  // keep the four most recent
      cudaGraphExecDestroy(c.sweepGraphs.front().exec);
      c.sweepGraphs.erase(c.sweepGraphs.begin());
    }
    c.sweepGraphs.push_back(CachedGraph{std::move(key), exec});
  }
  MSBG_CUDA(ctx, cudaGraphLaunch(exec, ctx->stream));
  ctx->launches += nLaunch;
  return MSBG_GPU_OK;
}

int colorSweepRun(msbg_gpu_ctx *ctx, Channel &c, bool exact, bool color8, int nIter, const SweepParams &p,
                  const int32_t *bids, const int *cs) {
  if (ctx->bsx == 32) {
    switch (c.storage) {
      case MSBG_GPU_F32: return runColorT<float, 32>(ctx, c, exact, color8, nIter, p, bids, cs);
      case MSBG_GPU_F16: return runColorT<__half, 32>(ctx, c, exact, color8, nIter, p, bids, cs);
      case MSBG_GPU_U16: return runColorT<uint16_t, 32>(ctx, c, exact, color8, nIter, p, bids, cs);
    }
  } else if (ctx->bsx == 16) {
    switch (c.storage) {
      case MSBG_GPU_F32: return runColorT<float, 16>(ctx, c, exact, color8, nIter, p, bids, cs);
      case MSBG_GPU_F16: return runColorT<__half, 16>(ctx, c, exact, color8, nIter, p, bids, cs);
      case MSBG_GPU_U16: return runColorT<uint16_t, 16>(ctx, c, exact, color8, nIter, p, bids, cs);
    }
  }
  return 1;  // not handled: caller uses the gather kernel
}

}  // namespace msbg
