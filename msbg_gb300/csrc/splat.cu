// Particle splat and distance-to-density finalize (channel 0).
//
// Reference: the demo's 8-color lockless splat (src/msbg_demo.cpp:527-636) and
// finalize (src/msbg_demo.cpp:655-680).  The CPU code walks per-block particle
// lists in 8 colors so that threads never write the same block concurrently.
// Here the particles are sorted by the value blocks their splat boxes touch (a
// counting sort: count, scan, scatter), and one CTA per value block takes the
// minimum of its particles' values in shared memory (atomicMin on the float's bit
// pattern: distances are non-negative, so their bit patterns order like the
// floats) and writes the block once.  The minimum is order-independent, so this
// gives the same field as the colored passes.
//
// The minimum is taken in FP32.  For uint16 / FP16 storage the splat runs into an
// FP32 staging slab and the finalize quantizes the minimum to the storage type
// first: rounding is monotonic, so quantize(min) == min(quantize) and the result
// equals the demo's min over quantized values (src/msbg_demo.cpp:624-628).
#include <algorithm>
#include <type_traits>

#include "internal.cuh"

namespace msbg {

// Every voxel of a slab <- v (the demo fills value blocks with 1.0 before splatting).
// Eight voxels per thread and step, stored as 16-byte vectors.
template <typename T>
__global__ void kFill(T *__restrict__ p, int64_t n, float v, double vd) {
  T e;
  if constexpr (sizeof(T) == 8) e = vd; else Store<T>::storeRHA(&e, v);
  T q[8];
#pragma unroll
  for (int k = 0; k < 8; k++) q[k] = e;
  const int64_t n8 = n / 8;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
    uint4 *dst = reinterpret_cast<uint4 *>(p + 8 * i);
#pragma unroll
    for (int k = 0; k < (int)(8 * sizeof(T) / 16); k++) dst[k] = reinterpret_cast<const uint4 *>(q)[k];
  }
  for (int64_t i = 8 * n8 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = e;
}

static unsigned gridVec(int64_t n) {  // 8 elements per thread, grid-stride
  const int64_t t = (n / 8 + 255) / 256;
  return (unsigned)(t < 1 ? 1 : t > 152 * 64 ? 152 * 64 : t);
}

int fillChannel(msbg_gpu_ctx *ctx, int chan, double v) {
  Channel &c = ctx->ch[chan];
  const int64_t n = ctx->nActive * ctx->voxPerBlock;
  if (n == 0) return MSBG_GPU_OK;
  switch (c.storage) {
    case MSBG_GPU_F32: MSBG_LAUNCH(ctx, kFill<float>, gridVec(n), 256, 0, (float *)c.d, n, (float)v, v); break;
    case MSBG_GPU_U16: MSBG_LAUNCH(ctx, kFill<uint16_t>, gridVec(n), 256, 0, (uint16_t *)c.d, n, (float)v, v); break;
    case MSBG_GPU_F16: MSBG_LAUNCH(ctx, kFill<__half>, gridVec(n), 256, 0, (__half *)c.d, n, (float)v, v); break;
    default: MSBG_LAUNCH(ctx, kFill<double>, gridVec(n), 256, 0, (double *)c.d, n, (float)v, v); break;
  }
  return MSBG_GPU_OK;
}

struct SplatGeom {
  int sx, sy, sz, nbx, nby, log2bs;
  float domMin[3], domMax[3];
  float rScan, distSqMax, distSqMaxInv;
  float negZero = -0.0f;  // see splatEntries
};

// A particle's splat box (src/msbg_demo.cpp:571-592): voxels [i1, i2] per axis,
// the voxel centres within rScan of the particle, clamped to the grid.
struct SplatBox {
  int ix1, iy1, iz1, ix2, iy2, iz2;
  float x0, y0, z0;  // particle position - 0.5 (voxel centre offsets)
};

__device__ __forceinline__ bool splatBox(const SplatGeom &g, float px, float py, float pz, SplatBox &b) {
  const float r = g.rScan;
  b.ix1 = max((int)ceilf(__fsub_rn(__fsub_rn(px, r), 0.5f)), 0);
  b.iy1 = max((int)ceilf(__fsub_rn(__fsub_rn(py, r), 0.5f)), 0);
  b.iz1 = max((int)ceilf(__fsub_rn(__fsub_rn(pz, r), 0.5f)), 0);
  b.ix2 = min((int)floorf(__fsub_rn(__fadd_rn(px, r), 0.5f)), g.sx - 1);
  b.iy2 = min((int)floorf(__fsub_rn(__fadd_rn(py, r), 0.5f)), g.sy - 1);
  b.iz2 = min((int)floorf(__fsub_rn(__fadd_rn(pz, r), 0.5f)), g.sz - 1);
  b.x0 = __fsub_rn(px, 0.5f); b.y0 = __fsub_rn(py, 0.5f); b.z0 = __fsub_rn(pz, 0.5f);
  return b.ix2 >= b.ix1 && b.iy2 >= b.iy1 && b.iz2 >= b.iz1;
}

// The lists' counters are shared by the particles near each other: a surface's particles
// come one after another, so thousands of atomics at a time met on the same few hundred
// addresses (2.05 M particles of the 512^3 workload: 346 us to count, 357 us to scatter).
// A CTA therefore sums its particles' blocks in a hash table in shared memory and goes to
// the global counters once per block (35 and 65 us).  Places are never given back.  Once a
// block finds none within kHashProbes, the CTA goes on without the table (full): most of its
// blocks come once (particles in no order on many blocks).  Giving up at half the places was
// slower: 1 M particles in a ball, 1,000 blocks of 16^3, 643 us against 510.
constexpr int kListThreads = 512, kHashSize = 2048, kHashProbes = 16;
constexpr int kDirectThreads = 256;  // of the forms without the table
struct BlockHash {
  int key[kHashSize], val[kHashSize];
  int full;
  __device__ __forceinline__ bool isFull() const { return *(const volatile int *)&full; }
};
__device__ __forceinline__ void hashClear(BlockHash &h) {
  if (threadIdx.x == 0) h.full = 0;
  for (int i = threadIdx.x; i < kHashSize; i += kListThreads) { h.key[i] = -1; h.val[i] = 0; }
}
// place of slot sl, claimed if INSERT; -1: none
template <bool INSERT>
__device__ __forceinline__ int hashPlace(BlockHash &h, int sl) {
  unsigned p = ((unsigned)sl * 2654435761u) >> 21;
  static_assert(kHashSize == 2048, "11 hash bits");
  for (int k = 0; k < kHashProbes; k++, p = (p + 1) & (kHashSize - 1)) {
    int at = *(volatile int *)&h.key[p];
    if (INSERT && at == -1) {
      at = atomicCAS(&h.key[p], -1, sl);
      if (at == -1) return (int)p;
    }
    if (at == sl) return (int)p;
    if (!INSERT && at == -1) return -1;
  }
  return -1;
}

// The slots of the value blocks a box touches (at most two per axis), each once, -1 elsewhere.
__device__ __forceinline__ bool boxSlots(const SplatGeom &g, const SplatBox &b, const int32_t *__restrict__ slot,
                                         int32_t sl[8]) {
  const int s = g.log2bs;
  const int64_t nxy = (int64_t)g.nbx * g.nby;
  const int bx[2] = {b.ix1 >> s, b.ix2 >> s}, by[2] = {b.iy1 >> s, b.iy2 >> s}, bz[2] = {b.iz1 >> s, b.iz2 >> s};
  bool allValue = true;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const bool dup = ((k & 1) && bx[1] == bx[0]) || ((k & 2) && by[1] == by[0]) || ((k & 4) && bz[1] == bz[0]);
    sl[k] = -1;
    if (!dup) {
      sl[k] = slot[(int64_t)bz[k >> 2] * nxy + (int64_t)by[(k >> 1) & 1] * g.nbx + bx[k & 1]];
      allValue = allValue && sl[k] >= 0;
    }
  }
  return allValue;
}

// List entries that a CTA of the third pass takes: an eighth of an even share of all entries
// over the CTAs that the chip holds (places), and at least 32 bs.  Without the share, 3 M
// particles in no order split every list in two (32^3 blocks, radius 4: 2.99 ms, 2.37 so).  Four
// times as many at least costs scenes whose particles crowd into a few blocks more (172 k on 56
// spheres, 1805 blocks of 16^3: 492 us, 280 so) than it saves where the lists are even (100 k in
// a ball, 32^3 blocks, radius 4: 175 us, 220 so; radius 10 907 and 1085).  whole: so few particles
// over so many blocks that the second launch is left out.
struct ChunkRule {
  int least, places, nz;
  bool whole;
  ChunkRule(int bs, int64_t nAct, int64_t n)
      : least(32 * bs), places(152 * 1536 / (16 * bs)), nz(bs == 32 ? 2 : 1),
        whole(n <= least || (n <= 4 * least && nz * nAct > places / 2)) {}
  __device__ int of(int64_t total) const {
    return whole ? 4 * least : (int)max((int64_t)least, total * nz / (8 * places));
  }
};

// Pass 1.  Valid particles (the marking loop's domain tests, src/msbg_demo.cpp:358-360, and
// an owning value block: the demo walks the particle lists of value blocks only,
// src/msbg_demo.cpp:541-566) get their abort index: the scan position (z, y, x order over
// the box) of the first in-sphere voxel whose block is not a value block
// (src/msbg_demo.cpp:613-618), or the box size.  Voxels from that position on are not
// written.  Every value block the box touches counts the particle once.  abortAt = 0 marks
// a particle that writes nothing.  A thread takes ppt particles, NT apart; HASH: counted through
// the table.
template <int NT, bool HASH>
__global__ void __launch_bounds__(NT) kSplatCount(const float *__restrict__ pts, int64_t n, int ppt, SplatGeom g,
                                                            const int32_t *__restrict__ slot,
                                                            int32_t *__restrict__ abortAt, int32_t *__restrict__ cnt,
                                                            unsigned long long *__restrict__ nAborted) {
  __shared__ BlockHash h;
  if (HASH) {
    hashClear(h);
    __syncthreads();
  }
  const int s = g.log2bs;
  const int64_t nxy = (int64_t)g.nbx * g.nby;
  const int64_t first = (int64_t)blockIdx.x * ppt * NT + threadIdx.x;
  for (int q = 0; q < ppt; q++) {
    const int64_t i = first + (int64_t)q * NT;
    if (i >= n) break;
    const float px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
    int abortIdx = 0;
    SplatBox b;
    int32_t sl[8];
    bool valid = !(px < g.domMin[0] || px > g.domMax[0] || py < g.domMin[1] || py > g.domMax[1] ||
                   pz < g.domMin[2] || pz > g.domMax[2]);
    if (valid) {
      const int ix = (int)px, iy = (int)py, iz = (int)pz;
      valid = ix >= 0 && ix < g.sx && iy >= 0 && iy < g.sy && iz >= 0 && iz < g.sz &&
              slot[(int64_t)(iz >> s) * nxy + (int64_t)(iy >> s) * g.nbx + (ix >> s)] >= 0;
    }
    if (valid && splatBox(g, px, py, pz, b)) {
      const int nx = b.ix2 - b.ix1 + 1, ny = b.iy2 - b.iy1 + 1, nz = b.iz2 - b.iz1 + 1;
      const int total = nx * ny * nz;
      abortIdx = total;
      if (!boxSlots(g, b, slot, sl)) {
        for (int t = 0; t < total; t++) {
          const int lx = t % nx, rest = t / nx, ly = rest % ny, lz = rest / ny;
          const int ix = b.ix1 + lx, iy = b.iy1 + ly, iz = b.iz1 + lz;
          const float dz = __fsub_rn((float)iz, b.z0), dy = __fsub_rn((float)iy, b.y0), dx = __fsub_rn((float)ix, b.x0);
          const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dz, dz), __fmul_rn(dy, dy)), __fmul_rn(dx, dx));
          if (d2 > g.distSqMax) continue;
          if (slot[(int64_t)(iz >> s) * nxy + (int64_t)(iy >> s) * g.nbx + (ix >> s)] < 0) {
            abortIdx = t;
            break;
          }
        }
        if (abortIdx < total) atomicAdd(nAborted, 1ull);
      }
    }
    abortAt[i] = abortIdx;
    if (abortIdx == 0) continue;
    bool hashed = HASH && !h.isFull();
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if (sl[k] < 0) continue;
      const int p = hashed ? hashPlace<true>(h, sl[k]) : -1;
      if (p >= 0) {
        atomicAdd(&h.val[p], 1);
      } else {
        if (hashed) h.full = 1;
        hashed = false;
        atomicAdd(&cnt[sl[k]], 1);
      }
    }
  }
  if (!HASH) return;
  __syncthreads();
  for (int i = threadIdx.x; i < kHashSize; i += NT)
    if (h.key[i] >= 0) atomicAdd(&cnt[h.key[i]], h.val[i]);
}

// Pass 2: the particle's index into the list of every value block it touches
// (list of slot s: entries[off[s] .. off[s+1]-1], in no particular order).  The CTA counts
// its particles per block, reserves a run of each list, and fills it (HASH), or takes every
// position by itself.  *chunk: the list entries that a CTA of the third pass takes.
template <int NT, bool HASH>
__global__ void __launch_bounds__(NT) kSplatScatter(const float *__restrict__ pts, int64_t n, int ppt,
                                                              SplatGeom g, const int32_t *__restrict__ slot,
                                                              const int32_t *__restrict__ abortAt,
                                                              const int64_t *__restrict__ off,
                                                              int32_t *__restrict__ cursor,
                                                              int32_t *__restrict__ entries, int64_t nAct, ChunkRule rule,
                                                              int *__restrict__ chunk) {
  __shared__ BlockHash h;
  __shared__ int run[kHashSize];  // the CTA's first position in a block's list
  if (blockIdx.x == 0 && threadIdx.x == 0) *chunk = rule.of(off[nAct]);
  const int64_t first = (int64_t)blockIdx.x * ppt * NT + threadIdx.x;
  auto forBlocks = [&](auto go, auto f) {
    for (int q = 0; q < ppt && go(); q++) {
      const int64_t i = first + (int64_t)q * NT;
      if (i >= n) break;
      if (abortAt[i] == 0) continue;
      SplatBox b;
      splatBox(g, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], b);
      int32_t sl[8];
      boxSlots(g, b, slot, sl);
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (sl[k] >= 0) f(sl[k], (int32_t)i);
    }
  };
  const auto always = [] { return true; };
  if (HASH) {
    hashClear(h);
    __syncthreads();
    forBlocks([&] { return !h.isFull(); }, [&](int sl, int32_t) {
      const int p = hashPlace<true>(h, sl);
      if (p >= 0) atomicAdd(&h.val[p], 1);
      else h.full = 1;
    });
    __syncthreads();
  }
  if (!HASH || h.isFull()) {
    forBlocks(always, [&](int sl, int32_t i) { entries[off[sl] + atomicAdd(&cursor[sl], 1)] = i; });
    return;
  }
  for (int i = threadIdx.x; i < kHashSize; i += NT)
    if (h.key[i] >= 0) {
      run[i] = atomicAdd(&cursor[h.key[i]], h.val[i]);
      h.val[i] = 0;
    }
  __syncthreads();
  forBlocks(always, [&](int sl, int32_t i) {  // every block has its place
    const int p = hashPlace<false>(h, sl);
    entries[off[sl] + run[p] + atomicAdd(&h.val[p], 1)] = i;
  });
}

// Pass 3, one CTA per value block (slot = blockIdx.x): the minimum of the splat
// values of the block's particles in shared memory, starting from the block's
// current values (init: FP32 channels, where the demo's splat takes the minimum
// with what the channel holds) or from 1.0 (the FP32 staging of other storage
// types, which the demo fills with 1.0 first), then one coalesced write of the
// block.  Half a warp or a warp (LANES) takes one particle at a time; its
// lanes take the (y, z) rows of the box clipped to the block, skip rows already
// outside the sphere (dz*dz + dy*dy exceeds it, and adding dx*dx >= 0 cannot lower
// a float sum), and keep the voxels before the particle's abort index.
// The block's minima in shared memory use a row stride of BS + 1 words: the lanes
// of a warp take different rows, which then fall into different banks.  NZ CTAs
// share a block, each taking BS/NZ of its z-planes (and clipping the boxes to
// them): for BS = 32 two halves of 68 KB let three CTAs share an SM where a whole
// block's 135 KB allowed one.
template <int BS, int NZ>
constexpr int splatSmemWords() { return BS * (BS / NZ) * (BS + 1); }
// threads per CTA (512, 256, 128 for BS 32, 16, 8), and CTAs per SM to keep the registers
// for: 1536 threads
template <int BS>
constexpr int splatThreads() { return 16 * BS; }
template <int BS>
constexpr int splatMinCtas() { return 1536 / splatThreads<BS>(); }

// LANES share a particle (the rule is at the launch).  A box has 81 rows at the demo's radius, fewer where the block
// clips it, and every lane of a group works out the whole box: 8 / 16 / 32 lanes take 940 / 901
// / 937 us for the splat of 768 k particles on 32^3 blocks, 4.07 / 4.05 / 4.26 ms for the 512^3
// pipeline (smaller groups of a warp wait for its longest box).
// Entries e0 .. e1-1 of a block's list into the minima of its planes Z0 .. Z0+PZ-1.
// Bound: issue (80% of the slots).
template <int BS, int NZ, int LANES>
__device__ __forceinline__ void splatEntries(int *smin, const float *__restrict__ pts, const SplatGeom &g, int X0, int Y0,
                                             int Z0, const int32_t *__restrict__ abortAt,
                                             const int32_t *__restrict__ entries, int64_t e0, int64_t e1) {
  constexpr int RS = BS + 1, PZ = BS / NZ;
  const int lane = threadIdx.x % LANES, group = threadIdx.x / LANES, nGroups = blockDim.x / LANES;
  for (int64_t e = e0 + group; e < e1; e += nGroups) {
    const int i = entries[e];
    const float px = pts[3 * (int64_t)i], py = pts[3 * (int64_t)i + 1], pz = pts[3 * (int64_t)i + 2];
    const int ab = abortAt[i];
    SplatBox b;
    splatBox(g, px, py, pz, b);
    const int nx = b.ix2 - b.ix1 + 1, ny = b.iy2 - b.iy1 + 1;
    const int cx1 = max(b.ix1, X0), cx2 = min(b.ix2, X0 + BS - 1);
    const int cy1 = max(b.iy1, Y0), cy2 = min(b.iy2, Y0 + BS - 1);
    const int cz1 = max(b.iz1, Z0), cz2 = min(b.iz2, Z0 + PZ - 1);
    const int cny = cy2 - cy1 + 1, cnz = cz2 - cz1 + 1;
    if (cx2 < cx1 || cny <= 0 || cnz <= 0) continue;
    // the lane's rows: row = lane + LANES k, decoded as (row % cny, row / cny) through an
    // approximate reciprocal (row < 34^2 and cny <= 33: the quotient's fraction stays
    // at least 1/(2 cny) away from an integer, so the truncation is exact)
    const float rcny = __frcp_rn((float)cny);
    for (int row = lane; row < cny * cnz; row += LANES) {
      const int qz = (int)(((float)row + 0.5f) * rcny);
      const int iy = cy1 + row - qz * cny, iz = cz1 + qz;
      const float dz = __fsub_rn((float)iz, b.z0), dy = __fsub_rn((float)iy, b.y0);
      const float dzy = __fadd_rn(__fmul_rn(dz, dz), __fmul_rn(dy, dy));
      if (dzy > g.distSqMax) continue;
      const int rowScan = ((iz - b.iz1) * ny + (iy - b.iy1)) * nx - b.ix1;  // + ix: the scan index
      int *rowMin = smin + ((iz - Z0) * BS + (iy - Y0)) * RS - X0;
      // The scan index grows with ix along the row, so the abort rule cuts the row at
      // ab - rowScan.  Two voxels a step on packed operations (splat of 768 k particles on
      // 32^3 blocks: 960 -> 935 us), x as floats (exact for these integers); distSq exactly
      // as the demo forms it, (dz*dz + dy*dy) + dx*dx: the square as fma(dx, dx, -0) with a
      // run-time -0, or the compiler would fuse it into the sum.
      const int xEnd = min(cx2, ab - 1 - rowScan);
      float2 fx = make_float2((float)cx1, (float)(cx1 + 1));
      const float2 nx0 = make_float2(-b.x0, -b.x0), nz = make_float2(g.negZero, g.negZero);
      const float2 dzy2 = make_float2(dzy, dzy), inv = make_float2(g.distSqMaxInv, g.distSqMaxInv);
#pragma unroll 1
      for (int ix = cx1; ix <= xEnd; ix += 2) {
        const float2 dx = __fadd2_rn(fx, nx0);
        const float2 d2 = __fadd2_rn(dzy2, __ffma2_rn(dx, dx, nz));
        const float2 v = __fmul2_rn(d2, inv);
        if (d2.x <= g.distSqMax) atomicMin(rowMin + ix, __float_as_int(v.x));
        if (d2.y <= g.distSqMax && ix < xEnd) atomicMin(rowMin + ix + 1, __float_as_int(v.y));
        fx = __fadd2_rn(fx, make_float2(2.0f, 2.0f));
      }
    }
  }
}

// A value block's first chunk, and the write of the block.  Blocks hold very different
// numbers of particles (a small sphere's 32,000 particles lie in a few dozen blocks), and a
// CTA that took the longest list alone ran while the other SMs had finished: the SMs were
// active 40% of the launch on the 512^3 workload (4.36 ms).  A longer list's other chunks
// are queued for kSplatRest (0.43 + 1.27 ms).
template <int BS, int NZ, int LANES>
__global__ void __launch_bounds__(splatThreads<BS>(), splatMinCtas<BS>()) kSplatBlock(const float *__restrict__ pts, SplatGeom g,
                                                   const int32_t *__restrict__ active,
                                                   const int32_t *__restrict__ abortAt,
                                                   const int64_t *__restrict__ off,
                                                   const int32_t *__restrict__ entries, const float *init,
                                                   float *dst, const int *__restrict__ chunk,
                                                   int *__restrict__ nRest, int2 *__restrict__ rest) {
  constexpr int VPB = BS * BS * BS, RS = BS + 1, PZ = BS / NZ, VPP = BS * BS * PZ;
  extern __shared__ __align__(16) int smin[];
  __shared__ int restAt;
  const int sl = blockIdx.x / NZ, zp = blockIdx.x % NZ;
  const int bid = active[sl];
  const int X0 = (bid % g.nbx) * BS, Y0 = ((bid / g.nbx) % g.nby) * BS,
            Z0 = (int)(bid / ((int64_t)g.nbx * g.nby)) * BS + zp * PZ;  // this CTA's first plane
  const int64_t e0 = off[sl];
  const int cnt = (int)(off[sl + 1] - e0), ch = *chunk;
  const int one = __float_as_int(1.0f);
  if (cnt == 0) {  // no particle: the block keeps its values, or is 1
    if (init) return;
    int4 *o = reinterpret_cast<int4 *>(dst + (int64_t)sl * VPB + zp * VPP);
    for (int v = threadIdx.x; v < VPP / 4; v += blockDim.x) o[v] = make_int4(one, one, one, one);
    return;
  }
  const float *in = init ? init + (int64_t)sl * VPB + zp * VPP : nullptr;
  for (int v = threadIdx.x; v < VPP; v += blockDim.x)
    smin[(v / BS) * RS + v % BS] = in ? __float_as_int(in[v]) : one;
  const int more = zp == 0 && cnt > ch ? (cnt - 1) / ch : 0;
  if (more && threadIdx.x == 0) restAt = atomicAdd(nRest, more);
  __syncthreads();
  for (int k = threadIdx.x; k < more; k += blockDim.x) rest[restAt + k] = make_int2(sl, k + 1);
  splatEntries<BS, NZ, LANES>(smin, pts, g, X0, Y0, Z0, abortAt, entries, e0, e0 + min(cnt, ch));
  __syncthreads();
  float *out = dst + (int64_t)sl * VPB + zp * VPP;
  for (int v = threadIdx.x * 4; v < VPP; v += blockDim.x * 4) {
    const int *row = smin + (v / BS) * RS + v % BS;
    *reinterpret_cast<int4 *>(out + v) = make_int4(row[0], row[1], row[2], row[3]);
  }
}

// The queued chunks: their minima are merged into the blocks that kSplatBlock has written
// (integer minima of the bit patterns, as there).
template <int BS, int NZ, int LANES>
__global__ void __launch_bounds__(splatThreads<BS>(), splatMinCtas<BS>()) kSplatRest(const float *__restrict__ pts, SplatGeom g,
                                                   const int32_t *__restrict__ active,
                                                   const int32_t *__restrict__ abortAt,
                                                   const int64_t *__restrict__ off,
                                                   const int32_t *__restrict__ entries, int *dst,
                                                   const int *__restrict__ chunk, const int *__restrict__ nRest, const int2 *__restrict__ rest) {
  constexpr int VPB = BS * BS * BS, RS = BS + 1, PZ = BS / NZ, VPP = BS * BS * PZ;
  extern __shared__ __align__(16) int smin[];
  const int n = *nRest * NZ, ch = *chunk;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int2 r = rest[w / NZ];
    const int sl = r.x, zp = w % NZ, bid = active[sl];
    const int X0 = (bid % g.nbx) * BS, Y0 = ((bid / g.nbx) % g.nby) * BS,
              Z0 = (int)(bid / ((int64_t)g.nbx * g.nby)) * BS + zp * PZ;
    for (int v = threadIdx.x; v < VPP; v += blockDim.x) smin[(v / BS) * RS + v % BS] = 0x7fffffff;
    __syncthreads();
    const int64_t e0 = off[sl] + (int64_t)r.y * ch;
    splatEntries<BS, NZ, LANES>(smin, pts, g, X0, Y0, Z0, abortAt, entries, e0, min(e0 + ch, off[sl + 1]));
    __syncthreads();
    int *out = dst + (int64_t)sl * VPB + zp * VPP;
    for (int v = threadIdx.x; v < VPP; v += blockDim.x) {
      const int m = smin[(v / BS) * RS + v % BS];
      if (m != 0x7fffffff && m < __ldcg(out + v)) atomicMin(out + v, m);
    }
    __syncthreads();
  }
}

// The demo's particlesPerBlock (src/msbg_demo.cpp:349-390): the containing block
// of every point that passes the marking loop's domain tests.
__device__ __forceinline__ int64_t ownerBlock(const SplatGeom &g, int nbz, const float *pts, int64_t i) {
  const float px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  if (px < g.domMin[0] || px > g.domMax[0] || py < g.domMin[1] || py > g.domMax[1] || pz < g.domMin[2] ||
      pz > g.domMax[2])
    return -1;
  const int ix = (int)px, iy = (int)py, iz = (int)pz;
  if (ix < 0 || ix >= g.sx || iy < 0 || iy >= g.sy || iz < 0 || iz >= g.sz) return -1;
  const int s = g.log2bs;
  return ((int64_t)(iz >> s) * g.nby + (iy >> s)) * g.nbx + (ix >> s);
}

__global__ void kOwnerCount(const float *__restrict__ pts, int64_t n, SplatGeom g, int nbz, int32_t *__restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t b = ownerBlock(g, nbz, pts, i);
  if (b >= 0) atomicAdd(&cnt[b], 1);
}

__global__ void kOwnerScatter(const float *__restrict__ pts, int64_t n, SplatGeom g, int nbz,
                              const int64_t *__restrict__ off, int32_t *__restrict__ cursor,
                              int32_t *__restrict__ index) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t b = ownerBlock(g, nbz, pts, i);
  if (b >= 0) index[off[b] + atomicAdd(&cursor[b], 1)] = (int32_t)i;
}

// distance -> density of one voxel (q: the quantized minimum splat value)
__device__ __forceinline__ float finalizeValue(float d, float rParticle, float nbDist, float distSqMax) {
  float f = 0.0f;
  if (d < 0.999f) {
    d = __fmul_rn(d, distSqMax);
    const float dist = __fsub_rn(__fsqrt_rn(d), rParticle);
    // 1 - MT_LINSTEPF(-rParticle, rParticle + nbDist, dist) (src/mtool.h:400-408);
    // the reference's -ffast-math build divides by the constant span through its
    // rounded reciprocal.
    const float a = -rParticle, b = __fadd_rn(rParticle, nbDist);
    float lin;
    if (dist < a) lin = 0.0f;
    else if (dist >= b) lin = 1.0f;
    else lin = __fmul_rn(__fsub_rn(dist, a), __frcp_rn(__fsub_rn(b, a)));
    f = __fsub_rn(1.0f, lin);
  }
  return f;
}

// Eight voxels per thread and step: two 16-byte reads of the FP32 minimum, one
// 16-byte (2-byte storage) or two (FP32) writes.
template <typename T>
__global__ void kFinalize(const float *__restrict__ splat, T *__restrict__ out, int64_t n, float rParticle,
                          float nbDist, float distSqMax) {
  const int64_t n8 = n / 8;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 a = reinterpret_cast<const float4 *>(splat)[2 * i], b = reinterpret_cast<const float4 *>(splat)[2 * i + 1];
    const float in[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    T q[8];
#pragma unroll
    for (int k = 0; k < 8; k++)  // the demo reads back the quantized minimum (renderDensToFloat_)
      Store<T>::storeRHA(&q[k], finalizeValue(Store<T>::quant(in[k]), rParticle, nbDist, distSqMax));
    uint4 *dst = reinterpret_cast<uint4 *>(out + 8 * i);
#pragma unroll
    for (int k = 0; k < (int)(8 * sizeof(T) / 16); k++) dst[k] = reinterpret_cast<const uint4 *>(q)[k];
  }
  for (int64_t i = 8 * n8 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    Store<T>::storeRHA(out + i, finalizeValue(Store<T>::quant(splat[i]), rParticle, nbDist, distSqMax));
}

template <>
__global__ void kFinalize<double>(const float *__restrict__ splat, double *__restrict__ out, int64_t n,
                                  float rParticle, float nbDist, float distSqMax) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = (double)finalizeValue(splat[i], rParticle, nbDist, distSqMax);
}

int splatRun(msbg_gpu_ctx *ctx, const float *dPts, int64_t n, float rParticle, float nbDist) {
  Channel &c = ctx->ch[0];
  const int64_t nAct = ctx->nActive;
  const int64_t nVox = nAct * ctx->voxPerBlock;
  float *dst;
  if (c.storage == MSBG_GPU_F32) {
    dst = (float *)c.d;
  } else {
    int rc = ensureTmpSlab(ctx, (size_t)(nVox > 0 ? nVox : 1) * 4);
    if (rc) return rc;
    dst = (float *)ctx->dTmpSlab;
  }
  MSBG_CUDA(ctx, cudaMemsetAsync(ctx->dCounters + 1, 0, 8, ctx->stream));
  if (nVox == 0) return MSBG_GPU_OK;
  SplatGeom g;
  g.sx = ctx->sx; g.sy = ctx->sy; g.sz = ctx->sz; g.nbx = ctx->nbx; g.nby = ctx->nby;
  g.log2bs = ctx->log2bs;
  for (int k = 0; k < 3; k++) { g.domMin[k] = ctx->domMin[k]; g.domMax[k] = ctx->domMax[k]; }
  g.rScan = rParticle + nbDist;
  g.distSqMax = g.rScan * g.rScan;
  g.distSqMaxInv = 1.0f / g.distSqMax;
  // scratch (stream-ordered): abort indices [n], counts / cursors [nAct], offsets
  // [nAct + 1], list entries [8 n] (a box touches at most 8 blocks)
  const int64_t nn = n > 0 ? n : 1;
  const size_t bAbort = (size_t)nn * 4, bCnt = ((size_t)nAct * 4 + 15) & ~size_t(15),
               bOff = (size_t)(nAct + 1) * 8, bEnt = (size_t)nn * 8 * 4;
  // queued chunks: fewer than the entries / the chunk length (32 bs); their count beside
  // the list counts, which are zeroed
  const size_t bRest = ((size_t)nn * 8 / (32 * ctx->bsx) + 1) * sizeof(int2);
  char *scratch = nullptr;
  MSBG_CUDA(ctx, cudaMallocAsync((void **)&scratch, bAbort + 2 * bCnt + bOff + bEnt + bRest + 128, ctx->stream));
  int32_t *abortAt = (int32_t *)scratch;
  int32_t *cnt = (int32_t *)(scratch + ((bAbort + 15) & ~size_t(15)));
  int32_t *cursor = (int32_t *)((char *)cnt + bCnt);
  int *nRest = (int *)((char *)cursor + bCnt), *chunk = nRest + 1;
  int64_t *off = (int64_t *)((char *)nRest + 16);
  int2 *rest = (int2 *)((char *)off + ((bOff + 15) & ~size_t(15)));
  int32_t *entries = (int32_t *)((char *)rest + ((bRest + 15) & ~size_t(15)));
  // particles per thread of the list passes: more per CTA share its table, while the CTAs
  // still fill the chip.  Splat on 2,100 blocks of 16^3 in us, 1 / 4 / 8 a thread: 300 k particles
  // 108 / 114 / 127, 700 k 193 / 195 / 205, 1.5 M 305 / 297 / 304, 3 M 536 / 517 / 520, 10 M 1674 / 1596 / 1596.
  const int ppt = n >= (int64_t)152 * 4 * kListThreads * 8 ? 8 : n >= (int64_t)152 * 4 * kListThreads * 2 ? 4 : 1;
  // The table pays where a block has many particles; with few, and for the smallest calls, its
  // set-up and flush cost more than they save.  Splat of FP16 blocks in us, table / none: 1 M
  // particles on shells in 32^3 blocks (radius 4) 1040 / 1532, 100 k so 157 / 191, 10 k (33 a
  // block) 69 / 66, 1 k 51 / 45; 1 M in no order on 262 k blocks of 8^3 (radius 1) 670 / 627.
  const bool hash = n >= 2048 && n >= 48 * nAct;
  const unsigned listGrid = hash ? gridFor(n, ppt * kListThreads) : gridFor(n, kDirectThreads);
  const ChunkRule rule(ctx->bsx, nAct, n);
  int rc = MSBG_GPU_OK;
  auto run = [&]() -> int {
    MSBG_CUDA(ctx, cudaMemsetAsync(cnt, 0, 2 * bCnt + 16, ctx->stream));
    if (n > 0) {
      unsigned long long *aborted = (unsigned long long *)(ctx->dCounters + 1);
      if (hash)
        MSBG_LAUNCH(ctx, (kSplatCount<kListThreads, true>), listGrid, kListThreads, 0, dPts, n, ppt, g, ctx->dSlot, abortAt,
                    cnt, aborted);
      else
        MSBG_LAUNCH(ctx, (kSplatCount<kDirectThreads, false>), listGrid, kDirectThreads, 0, dPts, n, 1, g, ctx->dSlot,
                    abortAt, cnt, aborted);
    }
    int r = exclusiveScanCounts(ctx, cnt, nAct, off, off + nAct);
    if (r) return r;
    if (n > 0) {
      if (hash)
        MSBG_LAUNCH(ctx, (kSplatScatter<kListThreads, true>), listGrid, kListThreads, 0, dPts, n, ppt, g, ctx->dSlot, abortAt,
                    off, cursor, entries, nAct, rule, chunk);
      else
        MSBG_LAUNCH(ctx, (kSplatScatter<kDirectThreads, false>), listGrid, kDirectThreads, 0, dPts, n, 1, g, ctx->dSlot,
                    abortAt, off, cursor, entries, nAct, rule, chunk);
    }
    const float *init = c.storage == MSBG_GPU_F32 ? dst : nullptr;
    auto blocks = [&](auto bsC, auto nzC, auto lanesC) -> int {
      constexpr int BS = decltype(bsC)::value, NZ = decltype(nzC)::value, LANES = decltype(lanesC)::value;
      constexpr int smem = splatSmemWords<BS, NZ>() * 4;
      const auto block = kSplatBlock<BS, NZ, LANES>;
      const auto restKern = kSplatRest<BS, NZ, LANES>;
      if (smem > 48 * 1024) {
        static SmemOptIn optInBlock, optInRest;
        MSBG_CUDA(ctx, optInBlock((const void *)block, smem));
        MSBG_CUDA(ctx, optInRest((const void *)restKern, smem));
      }
      MSBG_LAUNCH(ctx, block, (unsigned)(NZ * nAct), splatThreads<BS>(), smem, dPts, g, ctx->dActive, abortAt, off,
                  entries, init, dst, chunk, nRest, rest);
      if (!rule.whole)
        MSBG_LAUNCH(ctx, restKern, (unsigned)std::min<int64_t>(rule.places, NZ * (8 * n / rule.least + 1)),
                    splatThreads<BS>(), smem, dPts, g, ctx->dActive, abortAt, off, entries, (int *)dst, chunk, nRest, rest);
      return MSBG_GPU_OK;
    };
    using std::integral_constant;
    const int edge = (int)(2.0f * g.rScan) + 1;
    // Whole warps for boxes of 128 rows and more (the half warps of a warp wait for the longer
    // of two clipped boxes) and where a block has fewer particles than warps.  32^3 blocks, half /
    // whole warps, us: 1 M particles on shells, radius 2.5 557 / 667, radius 4 1038 / 1066; 100 k,
    // radius 4 156 / 163, radius 6 313 / 291, radius 10 971 / 766; 10 k in no order, radius 4 169 /
    // 159, radius 2.5 152 / 150.
    const bool wide = edge * edge >= 128 || n <= nAct * (ctx->bsx / 2);
    auto sized = [&](auto lanesC) -> int {
      if (ctx->bsx == 32) return blocks(integral_constant<int, 32>{}, integral_constant<int, 2>{}, lanesC);
      if (ctx->bsx == 16) return blocks(integral_constant<int, 16>{}, integral_constant<int, 1>{}, lanesC);
      return blocks(integral_constant<int, 8>{}, integral_constant<int, 1>{}, lanesC);
    };
    return wide ? sized(integral_constant<int, 32>{}) : sized(integral_constant<int, 16>{});
  };
  rc = run();
  cudaFreeAsync(scratch, ctx->stream);
  return rc;
}

int splatFinalizeRun(msbg_gpu_ctx *ctx, float rParticle, float nbDist) {
  Channel &c = ctx->ch[0];
  const int64_t n = ctx->nActive * ctx->voxPerBlock;
  if (n == 0) return MSBG_GPU_OK;
  const float rScan = rParticle + nbDist, distSqMax = rScan * rScan;
  const float *src = c.storage == MSBG_GPU_F32 ? (const float *)c.d : (const float *)ctx->dTmpSlab;
  if (c.storage != MSBG_GPU_F32 && ctx->tmpSlabBytes < (size_t)n * 4)
    return fail(ctx, MSBG_GPU_ERR_STATE, "finalize without a splat");
  switch (c.storage) {
    case MSBG_GPU_F32: MSBG_LAUNCH(ctx, kFinalize<float>, gridVec(n), 256, 0, src, (float *)c.d, n, rParticle, nbDist, distSqMax); break;
    case MSBG_GPU_U16: MSBG_LAUNCH(ctx, kFinalize<uint16_t>, gridVec(n), 256, 0, src, (uint16_t *)c.d, n, rParticle, nbDist, distSqMax); break;
    case MSBG_GPU_F16: MSBG_LAUNCH(ctx, kFinalize<__half>, gridVec(n), 256, 0, src, (__half *)c.d, n, rParticle, nbDist, distSqMax); break;
    default: MSBG_LAUNCH(ctx, kFinalize<double>, gridFor(n, 256), 256, 0, src, (double *)c.d, n, rParticle, nbDist, distSqMax); break;
  }
  return MSBG_GPU_OK;
}

int particlesPerBlockRun(msbg_gpu_ctx *ctx, const float *dPts, int64_t n, int64_t *dOff, int32_t *dIndex,
                         int64_t *count) {
  const int64_t nB = ctx->nBlocks;
  SplatGeom g;
  g.sx = ctx->sx; g.sy = ctx->sy; g.sz = ctx->sz; g.nbx = ctx->nbx; g.nby = ctx->nby;
  g.log2bs = ctx->log2bs;
  for (int k = 0; k < 3; k++) { g.domMin[k] = ctx->domMin[k]; g.domMax[k] = ctx->domMax[k]; }
  const size_t bCnt = ((size_t)nB * 4 + 15) & ~size_t(15);
  int32_t *cnt = nullptr;
  MSBG_CUDA(ctx, cudaMallocAsync((void **)&cnt, 2 * bCnt, ctx->stream));
  int32_t *cursor = (int32_t *)((char *)cnt + bCnt);
  auto run = [&]() -> int {
    MSBG_CUDA(ctx, cudaMemsetAsync(cnt, 0, 2 * bCnt, ctx->stream));
    if (n > 0) MSBG_LAUNCH(ctx, kOwnerCount, gridFor(n, 256), 256, 0, dPts, n, g, ctx->nbz, cnt);
    int r = exclusiveScanCounts(ctx, cnt, nB, dOff, dOff + nB);
    if (r) return r;
    if (n > 0) MSBG_LAUNCH(ctx, kOwnerScatter, gridFor(n, 256), 256, 0, dPts, n, g, ctx->nbz, dOff, cursor, dIndex);
    MSBG_CUDA(ctx, cudaMemcpyAsync(count, dOff + nB, 8, cudaMemcpyDeviceToHost, ctx->stream));
    return MSBG_GPU_OK;
  };
  int rc = run();
  cudaFreeAsync(cnt, ctx->stream);
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess && !rc) rc = fail(ctx, MSBG_GPU_ERR_CUDA, "particles_per_block");
  return rc;
}

}  // namespace msbg
