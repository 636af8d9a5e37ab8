// Block-structured Poisson kernels for the multigrid levels that keep level 0's
// block set (block edge bs = 32, 16, 8, 4 on a bs-32 layout): every cell finds
// its neighbours by offset inside its block and through a per-block table of the
// six face-neighbour slots across block faces, so no cell decodes a block id.
//
//   kApplyRows    y = A x, or r = b - A x, 4 cells along x per thread; with a
//                 fused FP64 dot (x . A x, the CG step length) or a fused
//                 restriction (the 8 children of a coarse cell sit in one
//                 4-lane group: lanes differ in the y and z parity bits).
//   kTileSmooth   one tile colour of the smoother: tiles of edge T (16 or 8) of
//                 one colour ((gx/T + gy/T + gz/T) & 1) are staged in shared
//                 memory with their one-cell halo by TMA, relaxed k times by
//                 red-black Gauss-Seidel inside the tile, and written back once.  The
//                 first pre-smoothing pass of a V-cycle starts from zero without
//                 reading x; the first post-smoothing pass adds the coarse
//                 correction (constant prolongation) while it loads.
//
// The reference relaxes red-black ordered blocks with block-local in-place
// iterations (src/msbg3.cpp:2170-2369, _mgSmBlockIter src/msbg.cpp:814-843) and
// evaluates the operator per block with a halo (src/msbg3.cpp:1281-1296); these
// kernels keep that structure with tiles as the GPU's unit of shared memory.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "internal.cuh"
#include "poisson.cuh"

namespace msbg {

__device__ __forceinline__ uint32_t smemAddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
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

// Index of the cell at block-local (lx, ly, lz) of slot s, where at most one
// coordinate may lie one block outside ([-bs, 2bs)); -1 when that block is absent.
__device__ __forceinline__ int64_t cellAt(const BlkGeom &g, int s, int lx, int ly, int lz) {
  const int bs = g.bs, L = g.log2bs;
  int dir = -1;
  if (lx < 0) { dir = 0; lx += bs; }
  else if (lx >= bs) { dir = 1; lx -= bs; }
  else if (ly < 0) { dir = 2; ly += bs; }
  else if (ly >= bs) { dir = 3; ly -= bs; }
  else if (lz < 0) { dir = 4; lz += bs; }
  else if (lz >= bs) { dir = 5; lz -= bs; }
  if (dir >= 0) {
    s = g.nbr[(int64_t)s * 6 + dir];
    if (s < 0) return -1;
  }
  return ((int64_t)s << (3 * L)) + ((int64_t)((lz << L) + ly) << L) + lx;
}

// Index on the coarse level (same blocks, edge bs/2) of the parent of fine cell j.
__device__ __forceinline__ int64_t parentOf(int64_t j, int L) {
  const int64_t s = j >> (3 * L);
  const int v = (int)(j & ((1 << (3 * L)) - 1));
  const int m = (1 << L) - 1;
  const int lx = v & m, ly = (v >> L) & m, lz = v >> (2 * L);
  const int Lc = L - 1;
  return (s << (3 * Lc)) + ((int64_t)(((lz >> 1) << Lc) + (ly >> 1)) << Lc) + (lx >> 1);
}

// ---------------------------------------------------------------------------------
// operator rows
// ---------------------------------------------------------------------------------
// Row segment q of a block (CPT cells along x: 4 for FP32 storage, 8 for FP16 on
// levels with bs >= 8, so that a thread moves 16 bytes per row load) -> block-local
// origin.  Bits of q from the bottom: x segment (log2(bs/CPT) bits), y parity,
// z parity, y pair, z pair; so the 8 children of the coarse cells over a segment
// pair are the 4 lanes {q, q^xq, q^2xq, q^3xq}.
template <typename V, int MODE, int CPT = 4>
__global__ void __launch_bounds__(256, CPT == 4 || sizeof(V) == 2 ? 3 : 2)
    kApplyRows(BlkGeom g, const V *__restrict__ x, const V *__restrict__ b, const V *__restrict__ cx,
               const V *__restrict__ cy, const V *__restrict__ cz, const V *__restrict__ d, V *__restrict__ y,
               double *__restrict__ dotPartial, V *__restrict__ bc, V *__restrict__ xc,
               __half *__restrict__ rhOut, float rhScale) {
  constexpr int LC = CPT == 4 ? 2 : 3;
  const int L = g.log2bs, bs = g.bs;
  const int xb = L - LC;
  const int qPerBlockLog = 3 * L - LC;
  const int64_t nQuad = g.nAct << qPerBlockLog;
  const int64_t nQuadPad = (nQuad + 31) & ~int64_t(31);
  const int64_t sy = bs, sz = (int64_t)bs * bs;
  double dot = 0.0, dot2 = 0.0;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nQuadPad;
       q += (int64_t)gridDim.x * blockDim.x) {
    const bool act = q < nQuad;
    const int64_t qq = act ? q : 0;
    const int s = (int)(qq >> qPerBlockLog);
    const int qb = (int)(qq & ((int64_t(1) << qPerBlockLog) - 1));
    const int qx = qb & ((1 << xb) - 1);
    const int yp = (qb >> xb) & 1, zp = (qb >> (xb + 1)) & 1;
    const int rest = qb >> (xb + 2);
    const int yh = rest & ((bs >> 1) - 1), zh = rest >> (L - 1);
    const int lx = qx << LC, ly = 2 * yh + yp, lz = 2 * zh + zp;
    const int64_t base = (int64_t)s << (3 * L);
    const int64_t c = base + ((int64_t)((lz << L) + ly) << L) + lx;

    // All loads as stored, the conversions after the last one (a conversion waits for its
    // load).  FP16: the x neighbours, which may need a block's table entry first, come last, and
    // the right-hand side early; FP32 rows leave no registers for that.
    constexpr bool H = sizeof(V) == 2;
    RawRow<V, CPT> xv, dv, cxv, cyv, czv, ym, yq, zm, zq, cyu, czu, bRow;
    xv.ld(x + c);
    dv.ld(d + c);
    cxv.ld(cx + c);
    cyv.ld(cy + c);
    czv.ld(cz + c);
    if constexpr (MODE > 0 && H) bRow.ld(b + c);
    V xlV = V(0.f), xrV = V(0.f), cxrV = V(0.f);
    auto xSides = [&]() {
      const int64_t j = lx > 0 ? c - 1 : cellAt(g, s, lx - 1, ly, lz);
      if (j >= 0) xlV = x[j];
      const int64_t k = lx + CPT < bs ? c + CPT : cellAt(g, s, lx + CPT, ly, lz);
      if (k >= 0) { xrV = x[k]; cxrV = cx[k]; }
    };
    if constexpr (!H) xSides();
    {
      const int64_t j = ly > 0 ? c - sy : cellAt(g, s, lx, ly - 1, lz);
      if (j >= 0) ym.ld(x + j); else ym.zero();
      const int64_t k = ly + 1 < bs ? c + sy : cellAt(g, s, lx, ly + 1, lz);
      if (k >= 0) { yq.ld(x + k); cyu.ld(cy + k); }
      else { yq.zero(); cyu.zero(); }
    }
    {
      const int64_t j = lz > 0 ? c - sz : cellAt(g, s, lx, ly, lz - 1);
      if (j >= 0) zm.ld(x + j); else zm.zero();
      const int64_t k = lz + 1 < bs ? c + sz : cellAt(g, s, lx, ly, lz + 1);
      if (k >= 0) { zq.ld(x + k); czu.ld(cz + k); }
      else { zq.zero(); czu.zero(); }
    }
    if constexpr (H) xSides();
    const float xl = ldv(&xlV), xr = ldv(&xrV), cxr = ldv(&cxrV);
    float r[CPT];
    if constexpr (MODE == 2) {
      static_assert(MODE != 2 || CPT == 4, "the checked residual runs on FP32 storage");
      // r = b - A x in double-float arithmetic: every product split exactly into
      // a rounded part and its error (fma), the running sum kept exact with
      // TwoSum and the errors gathered in a second float; then sum r^2, b^2.
      if constexpr (!H) bRow.ld(b + c);
      float rq = 0.f, bq = 0.f;
#pragma unroll
      for (int i = 0; i < CPT; i++) {
        const float xm1 = i == 0 ? xl : xv[i - 1];
        const float xp1 = i == CPT - 1 ? xr : xv[i + 1];
        const float cxp = i == CPT - 1 ? cxr : cxv[i + 1];
        const float fa[7] = {-dv[i], cxv[i], cxp, cyv[i], cyu[i], czv[i], czu[i]};
        const float fb[7] = {xv[i], xm1, xp1, ym[i], yq[i], zm[i], zq[i]};
        float S = bRow[i], E = 0.f;
#pragma unroll
        for (int t = 0; t < 7; t++) {
          const float h = __fmul_rn(fa[t], fb[t]);
          const float l = __fmaf_rn(fa[t], fb[t], -h);
          const float sn = __fadd_rn(S, h);
          const float bb2 = __fsub_rn(sn, S);
          const float e = __fadd_rn(__fsub_rn(S, __fsub_rn(sn, bb2)), __fsub_rn(h, bb2));
          S = sn;
          E = __fadd_rn(E, __fadd_rn(e, l));
        }
        r[i] = __fadd_rn(S, E);
        rq = fmaf(r[i], r[i], rq);
        bq = fmaf(bRow[i], bRow[i], bq);
      }
      if (act) {
        dot += (double)rq;
        dot2 += (double)bq;
        if (rhOut) {  // the scaled residual in FP16 (right-hand side of a correction solve)
          float sc[CPT];
#pragma unroll
          for (int i = 0; i < CPT; i++) sc[i] = r[i] * rhScale;
          stRow<CPT>(rhOut + c, sc);
        }
      }
    } else {
#pragma unroll
    for (int i = 0; i < CPT; i++) {
      const float xm1 = i == 0 ? xl : xv[i - 1];
      const float xp1 = i == CPT - 1 ? xr : xv[i + 1];
      const float cxp = i == CPT - 1 ? cxr : cxv[i + 1];
      float a = dv[i] * xv[i];
      a -= cxv[i] * xm1;
      a -= cxp * xp1;
      a -= cyv[i] * ym[i];
      a -= cyu[i] * yq[i];
      a -= czv[i] * zm[i];
      a -= czu[i] * zq[i];
      r[i] = a;
    }
    if constexpr (MODE == 1) {
      if constexpr (!H) bRow.ld(b + c);
#pragma unroll
      for (int i = 0; i < CPT; i++) r[i] = bRow[i] - r[i];
    }
    if (dotPartial && act) {
      float qd = 0.f;  // four products in FP32, then FP64 accumulation
#pragma unroll
      for (int i = 0; i < CPT; i += 4) {
        float q4 = 0.f;
#pragma unroll
        for (int k = i; k < i + 4; k++) q4 = fmaf(xv[k], r[k], q4);
        qd += q4;
      }
      dot += (double)qd;
    }
    if (bc) {
      // sum the 8 children: x pairs in-thread, y and z parities across lanes
      float p[CPT / 2];
#pragma unroll
      for (int i = 0; i < CPT / 2; i++) {
        p[i] = r[2 * i] + r[2 * i + 1];
        p[i] += __shfl_xor_sync(0xffffffffu, p[i], 1 << xb);
        p[i] += __shfl_xor_sync(0xffffffffu, p[i], 2 << xb);
      }
      if (act && yp == 0 && zp == 0) {
        const int Lc = L - 1;
        const int64_t ci = ((int64_t)s << (3 * Lc)) + ((int64_t)((zh << Lc) + yh) << Lc) + (lx >> 1);
        float zz[CPT / 2];
#pragma unroll
        for (int i = 0; i < CPT / 2; i++) zz[i] = 0.f;
        stRow<CPT / 2>(bc + ci, p);
        stRow<CPT / 2>(xc + ci, zz);
      }
    } else if (act && y) {
      stRow<CPT>(y + c, r);
    }
    }
  }
  if (dotPartial) {
    dot = blockSum(dot);
    if constexpr (MODE == 2) {
      dot2 = blockSum(dot2);
      if (threadIdx.x == 0) {
        dotPartial[2 * blockIdx.x] = dot;
        dotPartial[2 * blockIdx.x + 1] = dot2;
      }
    } else if (threadIdx.x == 0) {
      dotPartial[blockIdx.x] = dot;
    }
  }
}

// ---------------------------------------------------------------------------------
// tile smoother
// ---------------------------------------------------------------------------------
// Tiles: 32x16x8 cells on bs-32 levels (full 128-byte block rows, 8 tiles per
// block), the whole block on bs-16 and bs-8 levels.  Tile colour =
// (gx/TX + gy/TY + gz/TZ) & 1.  A CTA relaxes NT tiles; each thread owns one
// column of cells (cx, cy, 0..TZ-1) of a tile, whose x (with the two z-halo
// cells), b, 1/d and z-face coefficients it keeps in registers; the x values of
// the whole tile are mirrored in shared memory with an x / y halo ring, where the
// x and y neighbours are read.  The columns of a warp all have the same parity of
// cx + cy (every other x of whole rows), so in a red-black half step a warp
// updates the same z cells in every lane: no divergence, and since the padded row
// stride is even, the two half rows of a warp use the even and the odd banks.
//
// Loading: one thread per tile issues 3-D TMA boxes (cp.async.bulk.tensor) for the
// tile's x, b, d, cx, cy, cz, for the y and z halo faces of x and for the upper
// y / z faces of cy / cz, all completing on one mbarrier.  A face whose neighbour
// block is absent is requested at a coordinate outside the tensor and arrives as
// zeros.  The x halo columns (x = -1, x = TX) and cx at x = TX start at an x not
// aligned to 16 bytes and are loaded with plain loads while the boxes fly.
struct TileMaps {
  CUtensorMap xM, xY, xZ, b, d, cx, cy, cyY, cz, czZ;
};

template <int BS> struct TileShape;
template <> struct TileShape<32> { static constexpr int TX = 32, TY = 16, TZ = 8, NT = 1; };
template <> struct TileShape<16> { static constexpr int TX = 16, TY = 16, TZ = 16, NT = 1; };
template <> struct TileShape<8> { static constexpr int TX = 8, TY = 8, TZ = 8, NT = 4; };

__device__ __forceinline__ void tmaLoad3(void *dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smemAddr(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smemAddr(bar))
      : "memory");
}

// Byte offsets of one tile's buffers (each 128-byte aligned).
template <typename V, int BS>
struct TileSmem {
  using Sh = TileShape<BS>;
  static constexpr int TX = Sh::TX, TY = Sh::TY, TZ = Sh::TZ;
  static constexpr int E = (int)sizeof(V);
  static constexpr bool H = E != 4;  // FP16 storage: cx, cy read from the staged boxes
  static constexpr int C3 = TX * TY * TZ, CY2 = TX * TZ, CZ2 = TX * TY, CX2 = TY * TZ;
  static constexpr int al(int b) { return (b + 127) & ~127; }
  // FP32 x of the tile with its x and y halo: [TZ][TY + 2][TX + 2], cell (x, y, z)
  // at z*XPS + (y+1)*XRS + x+1 (even row stride)
  static constexpr int XRS = TX + 2, XPS = (TY + 2) * XRS, XSB = al(TZ * XPS * 4);
  static constexpr int X = 0;                       // TMA boxes [z][y][x] (V)
  static constexpr int B = X + al(C3 * E);
  static constexpr int D = B + al(C3 * E);
  static constexpr int CZ = D + al(C3 * E);
  static constexpr int CX = CZ + al(C3 * E);
  static constexpr int CY = CX + al(C3 * E);
  static constexpr int XYLO = CY + al(C3 * E);      // x at y = -1, y = TY ([z][x], V)
  static constexpr int XYHI = XYLO + al(CY2 * E);
  static constexpr int XZLO = XYHI + al(CY2 * E);   // x at z = -1, z = TZ ([y][x], V)
  static constexpr int XZHI = XZLO + al(CZ2 * E);
  static constexpr int CYHI = XZHI + al(CZ2 * E);   // cy at y = TY ([z][x], V)
  static constexpr int CZHI = CYHI + al(CY2 * E);   // cz at z = TZ ([y][x], V)
  static constexpr int CXHI = CZHI + al(CZ2 * E);   // cx at x = TX ([z][y], float; V on FP16 storage)
  static constexpr int END0 = CXHI + al(CX2 * 4);
  // the padded x array: over the x/b/d/cz boxes once they sit in registers when
  // it fits there (FP32), else after everything
  static constexpr bool XS_OVER = XSB <= CX;
  static constexpr int XS = XS_OVER ? 0 : END0;
  // FP32 tiles of edge 16: copies of cx and cy with the padded array's row stride and with
  // their upper faces as one more column / row, behind it over the same boxes.  In the boxes
  // themselves, rows two apart lie in the same banks and a warp holds four: conflicts were
  // more than half of the kernel's shared-memory wavefronts, which kept that pipe 75% busy
  // (solve of 14.2 M cells, copies and the warps' rows together: 7.47 -> 6.94 ms).
  static constexpr bool PADC = E == 4 && BS == 16;
  static constexpr int CXP = XSB, CXPS = TY * XRS, CYP = CXP + al(TZ * CXPS * 4), CYPS = (TY + 1) * XRS;
  static_assert(!PADC || CYP + TZ * CYPS * 4 <= CX, "the padded copies fit over the consumed boxes");
  static constexpr int END1 = XS_OVER ? END0 : END0 + XSB;
  static constexpr int BYTES = END1;
};
template <int BS>
constexpr int tileThreads() {
  using Sh = TileShape<BS>;
  return Sh::NT * Sh::TX * Sh::TY;
}
template <typename V, int BS>
constexpr size_t tileSmemBytes() {
  return (size_t)TileShape<BS>::NT * TileSmem<V, BS>::BYTES + 128;  // + mbarrier
}

// One red-black half step of a column: cells z = P, P+2, ... (all lanes of a warp
// share P).  xp points at the cell (tx, ty, 0) of the padded x array; the upper
// x / y face coefficients come from (pointer, stride per z).
template <int TZ, int TXY, int XRS, int XPS, int P>
__device__ __forceinline__ void colStep(float *xr, const float *bb, const float *rd, const float *czr, float *xp,
                                        const float *cxs, const float *pcxu, int scxu, const float *cys,
                                        const float *pcyu, int scyu) {
#pragma unroll
  for (int z = P; z < TZ; z += 2) {
    float *q = xp + z * XPS;
    float acc = bb[z];
    acc += cxs[z * TXY] * q[-1];
    acc += pcxu[z * scxu] * q[1];
    acc += cys[z * TXY] * q[-XRS];
    acc += pcyu[z * scyu] * q[XRS];
    acc += czr[z] * xr[z];
    acc += czr[z + 1] * xr[z + 2];
    const float v = acc * rd[z];
    xr[z + 1] = v;
    q[0] = v;
  }
}

// The same half step on padded coefficient copies (TileSmem::PADC): all strides are known.
template <int TZ, int XRS, int XPS, int CXPS, int CYPS, int P>
__device__ __forceinline__ void colStepP(float *xr, const float *bb, const float *rd, const float *czr, float *xp,
                                         const float *cxs, const float *cys) {
#pragma unroll
  for (int z = P; z < TZ; z += 2) {
    float *q = xp + z * XPS;
    float acc = bb[z];
    acc += cxs[z * CXPS] * q[-1];
    acc += cxs[z * CXPS + 1] * q[1];
    acc += cys[z * CYPS] * q[-XRS];
    acc += cys[z * CYPS + XRS] * q[XRS];
    acc += czr[z] * xr[z];
    acc += czr[z + 1] * xr[z + 2];
    const float v = acc * rd[z];
    xr[z + 1] = v;
    q[0] = v;
  }
}

// The same half step on FP16 storage.  The column's own lower-face coefficients
// (cx, cy of cell z) sit in registers as one packed FP16 pair per cell; the upper
// ones (the x+1 / y+1 neighbour's cx / cy) are read from the staged FP16 boxes
// (pointer, stride per z).  FP16 to FP32 is exact, so the sums are those of the
// FP32-copy form, in the same order.
template <int TZ, int TXY, int XRS, int XPS, int P>
__device__ __forceinline__ void colStepH(float *xr, const float *bb, const float *rd, const float *czr, float *xp,
                                         const uint32_t *cpk, const __half *pcxu, int scxu, const __half *pcyu,
                                         int scyu) {
#pragma unroll
  for (int z = P; z < TZ; z += 2) {
    float *q = xp + z * XPS;
    const uint32_t w = cpk[z];
    const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&w));
    float acc = bb[z];
    acc += c.x * q[-1];
    acc += __half2float(pcxu[z * scxu]) * q[1];
    acc += c.y * q[-XRS];
    acc += __half2float(pcyu[z * scyu]) * q[XRS];
    acc += czr[z] * xr[z];
    acc += czr[z + 1] * xr[z + 2];
    const float v = acc * rd[z];
    xr[z + 1] = v;
    q[0] = v;
  }
}

template <typename V, int BS>
__global__ void __launch_bounds__(tileThreads<BS>(), 2)
    kTileSmooth(const __grid_constant__ TileMaps maps, BlkGeom g, V *__restrict__ x, const V *__restrict__ cxg,
                const V *__restrict__ xc, int tc, int k, int reverse, int flags, int *__restrict__ status) {
  using S = TileSmem<V, BS>;
  using Sh = TileShape<BS>;
  constexpr int TX = Sh::TX, TY = Sh::TY, TZ = Sh::TZ, NT = Sh::NT, TXY = TX * TY;
  constexpr int HX = TX / 2, RW = 64 / TX;  // lanes per half row, rows per warp
  extern __shared__ __align__(128) unsigned char smem[];
  const int tIn = threadIdx.x / TXY, r = threadIdx.x % TXY;
  // column of this thread: warp w of the tile takes rows RW*(w/2).. with
  // (x + y) & 1 == w & 1
  const int wq = r >> 5, lane = r & 31;
  const int P = wq & 1;
  // rows of the warp: with 16-cell rows, two pairs eight rows apart, which a row stride of 18
  // words puts into different banks (consecutive rows meet in a third of them)
  const int lr = lane / HX;
  const int ty = BS == 16 ? 2 * (wq >> 1) + (lr & 1) + 8 * (lr >> 1) : (wq >> 1) * RW + lr;
  const int tx = 2 * (lane % HX) + ((P + ty) & 1);
  unsigned char *tb = smem + tIn * S::BYTES;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + NT * S::BYTES);

  const int L = g.log2bs;
  const int64_t unit = (int64_t)blockIdx.x * NT + tIn;
  int s = 0, ox = 0, oy = 0, oz = 0;
  bool valid;
  if (BS == 32) {  // 4 tiles of each colour per block: z tile j, y tile from the colour
    valid = unit < g.nAct * 4;
    if (valid) {
      s = (int)(unit >> 2);
      const int j = (int)(unit & 3);
      const int bxp = g.bpar[s] & 1;
      oz = j * TZ;
      oy = ((tc + bxp + j) & 1) * TY;
    }
  } else {         // the tile is the block: block parity lists
    const int64_t nUnits = tc == 0 ? g.nEven : g.nAct - g.nEven;
    valid = unit < nUnits;
    if (valid) s = g.parList[tc == 0 ? unit : g.nEven + unit];
  }
  const bool ownZero = flags & kOwnZero, haloZero = flags & kHaloZero;
  const bool ownCorr = flags & kOwnCorr, haloCorr = flags & kHaloCorr;
  const int zb = s * BS;

  if (threadIdx.x == 0) {
    mbarInit(bar, NT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (r == 0) {
    if (valid) {
      constexpr uint32_t B3 = S::C3 * S::E, BY = S::CY2 * S::E, BZ = S::CZ2 * S::E;
      const uint32_t bytes = (ownZero ? 5 : 6) * B3 + (haloZero ? 0 : 2 * (BY + BZ)) + BY + BZ;
      mbarExpectTx(bar, bytes);
      if (!ownZero) tmaLoad3(tb + S::X, &maps.xM, ox, oy, zb + oz, bar);
      tmaLoad3(tb + S::B, &maps.b, ox, oy, zb + oz, bar);
      tmaLoad3(tb + S::D, &maps.d, ox, oy, zb + oz, bar);
      tmaLoad3(tb + S::CZ, &maps.cz, ox, oy, zb + oz, bar);
      tmaLoad3(tb + S::CX, &maps.cx, ox, oy, zb + oz, bar);
      tmaLoad3(tb + S::CY, &maps.cy, ox, oy, zb + oz, bar);
      const int32_t *nb = g.nbr + (int64_t)s * 6;
      // y faces (box TX x 1 x TZ), z faces (box TX x TY x 1); absent -> outside -> zeros
      int ylo, ylz, yhi, yhz, zlo, zhi;
      if (oy > 0) { ylo = oy - 1; ylz = zb + oz; }
      else { const int n = nb[2]; ylo = BS - 1; ylz = n >= 0 ? n * BS + oz : -2 * TZ; }
      if (oy + TY < BS) { yhi = oy + TY; yhz = zb + oz; }
      else { const int n = nb[3]; yhi = 0; yhz = n >= 0 ? n * BS + oz : -2 * TZ; }
      if (oz > 0) zlo = zb + oz - 1;
      else { const int n = nb[4]; zlo = n >= 0 ? n * BS + BS - 1 : -2; }
      if (oz + TZ < BS) zhi = zb + oz + TZ;
      else { const int n = nb[5]; zhi = n >= 0 ? n * BS : -2; }
      if (!haloZero) {
        tmaLoad3(tb + S::XYLO, &maps.xY, ox, ylo, ylz, bar);
        tmaLoad3(tb + S::XYHI, &maps.xY, ox, yhi, yhz, bar);
        tmaLoad3(tb + S::XZLO, &maps.xZ, ox, oy, zlo, bar);
        tmaLoad3(tb + S::XZHI, &maps.xZ, ox, oy, zhi, bar);
      }
      tmaLoad3(tb + S::CYHI, &maps.cyY, ox, yhi, yhz, bar);
      tmaLoad3(tb + S::CZHI, &maps.czZ, ox, oy, zhi, bar);
    } else {
      mbarExpectTx(bar, 0);
    }
  }
  // while the boxes fly: the x halo columns (x = -1, x = TX) and cx at x = TX by
  // plain loads (face cell (y, z) = (q % TY, q / TY)), coarse corrections
  // Values stay as stored until the boxes have landed: a conversion waits for its load, and
  // the loads behind it for the conversion.
  constexpr int NXF = (S::CX2 + TXY - 1) / TXY;
  const V zeroV = V(0.f);
  V xloV[NXF], xhiV[NXF], xloC[NXF], xhiC[NXF];  // values and coarse corrections
  using CxT = std::conditional_t<S::H, V, float>;
  CxT *cxhi = reinterpret_cast<CxT *>(tb + S::CXHI);
  V chi[NXF];
#pragma unroll
  for (int i = 0; i < NXF; i++) {
    const int q = r + i * TXY;
    xloV[i] = xhiV[i] = xloC[i] = xhiC[i] = chi[i] = zeroV;
    if (valid && q < S::CX2) {
      const int j = q % TY, kk = q / TY;
      const int64_t lo = cellAt(g, s, ox - 1, oy + j, oz + kk);
      const int64_t hi = cellAt(g, s, ox + TX, oy + j, oz + kk);
      if (hi >= 0) chi[i] = cxg[hi];
      if (!haloZero) {
        if (lo >= 0) xloV[i] = x[lo];
        if (hi >= 0) xhiV[i] = x[hi];
        if (haloCorr) {
          if (lo >= 0) xloC[i] = xc[parentOf(lo, L)];
          if (hi >= 0) xhiC[i] = xc[parentOf(hi, L)];
        }
      }
    }
  }
  V corrV[TZ / 2], czc0V = zeroV, czc1V = zeroV;
#pragma unroll
  for (int z = 0; z < TZ / 2; z++) corrV[z] = zeroV;
  if (valid && ownCorr) {
    const int Lc = L - 1;
    const int64_t pb = ((int64_t)s << (3 * Lc)) + ((ox + tx) >> 1) + ((int64_t)((oy + ty) >> 1) << Lc);
#pragma unroll
    for (int z = 0; z < TZ / 2; z++) corrV[z] = xc[pb + ((int64_t)((oz >> 1) + z) << (2 * Lc))];
  }
  if (valid && haloCorr) {  // the z-halo cells of this column
    const int64_t j2 = cellAt(g, s, ox + tx, oy + ty, oz - 1), j3 = cellAt(g, s, ox + tx, oy + ty, oz + TZ);
    if (j2 >= 0) czc0V = xc[parentOf(j2, L)];
    if (j3 >= 0) czc1V = xc[parentOf(j3, L)];
  }
#pragma unroll
  for (int i = 0; i < NXF; i++) {
    const int q = r + i * TXY;
    if (q < S::CX2) cxhi[q] = (CxT)chi[i];
  }
  // wait for the boxes (bounded): one warp polls the barrier, the others sleep in
  // __syncthreads, which also publishes the landed data to them; the decision is
  // CTA-uniform
  bool ok = true;
  if (threadIdx.x < 32) {
    int it = 0;
    while (!mbarTryWait(bar, 0))
      if (++it >= (1 << 22)) { ok = false; break; }
  }
  ok = __syncthreads_and(ok);
  if (!ok) {
    if (threadIdx.x == 0) atomicOr(status, 2);
    for (int it = 0; it < (1 << 22); it++)
      if (mbarTryWait(bar, 0)) break;  // no copy may land after exit
    return;
  }
  float xlo[NXF], xhi[NXF], corr[TZ / 2];
#pragma unroll
  for (int i = 0; i < NXF; i++) {
    xlo[i] = ldv(&xloV[i]) + ldv(&xloC[i]);
    xhi[i] = ldv(&xhiV[i]) + ldv(&xhiC[i]);
  }
#pragma unroll
  for (int z = 0; z < TZ / 2; z++) corr[z] = ldv(&corrV[z]);
  const float czc0 = ldv(&czc0V), czc1 = ldv(&czc1V);
  // the column into registers
  const int own = ty * TX + tx;
  float xr[TZ + 2], bb[TZ], rd[TZ], czr[TZ + 1];
  {
    const V *sx = reinterpret_cast<const V *>(tb + S::X), *sb = reinterpret_cast<const V *>(tb + S::B);
    const V *sd = reinterpret_cast<const V *>(tb + S::D), *scz = reinterpret_cast<const V *>(tb + S::CZ);
#pragma unroll
    for (int z = 0; z < TZ; z++) {
      xr[z + 1] = (ownZero ? 0.f : ldv(sx + own + z * TXY)) + corr[z >> 1];
      bb[z] = ldv(sb + own + z * TXY);
      rd[z] = __frcp_rn(ldv(sd + own + z * TXY));
      czr[z] = ldv(scz + own + z * TXY);
    }
    czr[TZ] = ldv(reinterpret_cast<const V *>(tb + S::CZHI) + own);
    const V *fz0 = reinterpret_cast<const V *>(tb + S::XZLO), *fz1 = reinterpret_cast<const V *>(tb + S::XZHI);
    xr[0] = haloZero ? 0.f : ldv(fz0 + own) + czc0;
    xr[TZ + 1] = haloZero ? 0.f : ldv(fz1 + own) + czc1;
  }
  // y faces (+ coarse correction) and the FP32 coefficient copies, read before
  // the padded x array may overwrite the staged boxes
  constexpr int NYF = (S::CY2 + TXY - 1) / TXY;
  float ya[NYF], yb[NYF];
  {
    const V *fy0 = reinterpret_cast<const V *>(tb + S::XYLO), *fy1 = reinterpret_cast<const V *>(tb + S::XYHI);
#pragma unroll
    for (int i = 0; i < NYF; i++) {
      const int q = r + i * TXY;
      ya[i] = yb[i] = 0.f;
      if (valid && !haloZero && q < S::CY2) {
        ya[i] = ldv(fy0 + q);
        yb[i] = ldv(fy1 + q);
        if (haloCorr) {
          const int fx = q % TX, fz = q / TX;
          const int64_t j0 = cellAt(g, s, ox + fx, oy - 1, oz + fz), j1 = cellAt(g, s, ox + fx, oy + TY, oz + fz);
          if (j0 >= 0) ya[i] += ldv(xc + parentOf(j0, L));
          if (j1 >= 0) yb[i] += ldv(xc + parentOf(j1, L));
        }
      }
    }
  }
  // FP16 storage: the column's own (cx, cy) pairs into registers
  uint32_t cpk[S::H ? TZ : 1];
  if constexpr (S::H) {
    const uint16_t *scx = reinterpret_cast<const uint16_t *>(tb + S::CX);
    const uint16_t *scy = reinterpret_cast<const uint16_t *>(tb + S::CY);
#pragma unroll
    for (int z = 0; z < TZ; z++) cpk[z] = (uint32_t)scx[own + z * TXY] | ((uint32_t)scy[own + z * TXY] << 16);
  }
  if (S::XS_OVER) __syncthreads();  // the boxes under the padded array are read
  float *xs = reinterpret_cast<float *>(tb + S::XS);
  float *xp = xs + (ty + 1) * S::XRS + tx + 1;
#pragma unroll
  for (int z = 0; z < TZ; z++) xp[z * S::XPS] = xr[z + 1];
#pragma unroll
  for (int i = 0; i < NXF; i++) {
    const int q = r + i * TXY;
    if (q < S::CX2) {
      const int j = q % TY, kk = q / TY;
      xs[kk * S::XPS + (j + 1) * S::XRS] = xlo[i];
      xs[kk * S::XPS + (j + 1) * S::XRS + TX + 1] = xhi[i];
    }
  }
#pragma unroll
  for (int i = 0; i < NYF; i++) {
    const int q = r + i * TXY;
    if (q < S::CY2) {
      const int fx = q % TX, fz = q / TX;
      xs[fz * S::XPS + fx + 1] = ya[i];                      // y = -1
      xs[fz * S::XPS + (TY + 1) * S::XRS + fx + 1] = yb[i];  // y = TY
    }
  }
  float *cxP = reinterpret_cast<float *>(tb + S::CXP), *cyP = reinterpret_cast<float *>(tb + S::CYP);
  if constexpr (S::PADC) {
    const float *bx = reinterpret_cast<const float *>(tb + S::CX) + own, *by = reinterpret_cast<const float *>(tb + S::CY) + own;
#pragma unroll
    for (int z = 0; z < TZ; z++) {
      cxP[z * S::CXPS + ty * S::XRS + tx] = bx[z * TXY];
      cyP[z * S::CYPS + ty * S::XRS + tx] = by[z * TXY];
    }
#pragma unroll
    for (int i = 0; i < NXF; i++) {  // cx at x = TX, as this thread loaded it
      const int q = r + i * TXY;
      if (q < S::CX2) cxP[(q / TY) * S::CXPS + (q % TY) * S::XRS + TX] = ldv(cxhi + q);
    }
    const float *fy = reinterpret_cast<const float *>(tb + S::CYHI);
#pragma unroll
    for (int i = 0; i < NYF; i++) {
      const int q = r + i * TXY;
      if (q < S::CY2) cyP[(q / TX) * S::CYPS + TY * S::XRS + q % TX] = fy[q];
    }
  }
  __syncthreads();
  // upper-face coefficients inside the tile or on a face (pointer, stride per z)
  using CT = std::conditional_t<S::H, V, float>;  // type of the staged cx, cy boxes and faces
  const CT *cxs = reinterpret_cast<const CT *>(tb + S::CX) + own;
  const CT *cys = reinterpret_cast<const CT *>(tb + S::CY) + own;
  const CT *pcxu = tx < TX - 1 ? cxs + 1 : cxhi + ty;
  const int scxu = tx < TX - 1 ? TXY : TY;
  const CT *pcyu = ty < TY - 1 ? cys + TX : reinterpret_cast<const CT *>(tb + S::CYHI) + tx;
  const int scyu = ty < TY - 1 ? TXY : TX;
  for (int it = 0; it < k; it++) {
    for (int ci = 0; ci < 2; ci++) {
      const int cc = reverse ? 1 - ci : ci;
      if (valid) {  // cells z with (tx + ty + z) & 1 == cc: z = ((cc - P) & 1) + 2m
        if constexpr (S::H) {
          if (((cc - P) & 1) == 0)
            colStepH<TZ, TXY, S::XRS, S::XPS, 0>(xr, bb, rd, czr, xp, cpk, pcxu, scxu, pcyu, scyu);
          else
            colStepH<TZ, TXY, S::XRS, S::XPS, 1>(xr, bb, rd, czr, xp, cpk, pcxu, scxu, pcyu, scyu);
        } else if constexpr (S::PADC) {
          const float *px = cxP + ty * S::XRS + tx, *py = cyP + ty * S::XRS + tx;
          if (((cc - P) & 1) == 0)
            colStepP<TZ, S::XRS, S::XPS, S::CXPS, S::CYPS, 0>(xr, bb, rd, czr, xp, px, py);
          else
            colStepP<TZ, S::XRS, S::XPS, S::CXPS, S::CYPS, 1>(xr, bb, rd, czr, xp, px, py);
        } else {
          if (((cc - P) & 1) == 0)
            colStep<TZ, TXY, S::XRS, S::XPS, 0>(xr, bb, rd, czr, xp, cxs, pcxu, scxu, cys, pcyu, scyu);
          else
            colStep<TZ, TXY, S::XRS, S::XPS, 1>(xr, bb, rd, czr, xp, cxs, pcxu, scxu, cys, pcyu, scyu);
        }
      }
      // the write-back reads registers only: no barrier after the last half step
      if (ci == 0 || it + 1 < k) __syncthreads();
    }
  }
  if (valid) {
    const int64_t base = ((int64_t)s << (3 * L)) + ((int64_t)(oy + ty) << L) + ox + tx;
#pragma unroll
    for (int z = 0; z < TZ; z++) stv(x + base + ((int64_t)(oz + z) << (2 * L)), xr[z + 1]);
  }
}

static __global__ void kSumPartialsBlk(const double *__restrict__ partial, int n, double *__restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  s = blockSum(s);
  if (threadIdx.x == 0) *out = s;
}
static __global__ void kSumPartialsBlk2(const double *__restrict__ partial, int n, double *__restrict__ out) {
  double s0 = 0.0, s1 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    s0 += partial[2 * i];
    s1 += partial[2 * i + 1];
  }
  s0 = blockSum(s0);
  s1 = blockSum(s1);
  if (threadIdx.x == 0) { out[0] = s0; out[1] = s1; }
}

// ---------------------------------------------------------------------------------
// CG vector kernels on level 0 (n a multiple of 4), 4 values per thread; FP32
// products summed per group of 4, then accumulated in FP64.
// ---------------------------------------------------------------------------------
#define QUAD_STRIDE(q, nq) \
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < (nq); q += (int64_t)gridDim.x * blockDim.x)

// W cells per thread and step: 4 (FP32, 16-byte loads) or 8 (FP16, 16-byte loads)
template <typename V, int W>
__global__ void __launch_bounds__(256) kDotQuad(const V *__restrict__ a, const V *__restrict__ b, int64_t nq,
                                                double *__restrict__ partial) {
  double s = 0.0;
  QUAD_STRIDE(q, nq) {
    float av[W], bv[W];
    ldRow<W>(a + W * q, av);
    ldRow<W>(b + W * q, bv);
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < W; i++) t = fmaf(av[i], bv[i], t);
    s += (double)t;
  }
  s = blockSum(s);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
// alpha = sc[0] / sc[1]; x += alpha p; r -= alpha q; partial = sum r^2 (stored r)
template <typename V, int W>
__global__ void __launch_bounds__(256) kUpdateXRQuad(const double *__restrict__ sc, const V *__restrict__ p,
                                                     const V *__restrict__ q, V *__restrict__ x, V *__restrict__ r,
                                                     int64_t nq, double *__restrict__ partial) {
  const float alpha = sc[1] != 0.0 ? (float)(sc[0] / sc[1]) : 0.0f;
  double rr = 0.0;
  QUAD_STRIDE(k, nq) {
    float pv[W], qv[W], xv[W], rv[W];
    ldRow<W>(p + W * k, pv);
    ldRow<W>(q + W * k, qv);
    ldRow<W>(x + W * k, xv);
    ldRow<W>(r + W * k, rv);
#pragma unroll
    for (int i = 0; i < W; i++) {
      xv[i] = fmaf(alpha, pv[i], xv[i]);
      rv[i] = fmaf(-alpha, qv[i], rv[i]);
    }
    stRow<W>(x + W * k, xv);
    stRow<W>(r + W * k, rv);
    float rs[W];
    ldRow<W>(r + W * k, rs);  // the values as stored
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < W; i++) t = fmaf(rs[i], rs[i], t);
    rr += (double)t;
  }
  rr = blockSum(rr);
  if (threadIdx.x == 0) partial[blockIdx.x] = rr;
}
// x += scale * e (FP32 x, FP16 correction), 8 cells per step
__global__ void __launch_bounds__(256) kAddScaledQuad(const __half *__restrict__ e, float scale, float *__restrict__ x,
                                                      int64_t nq) {
  QUAD_STRIDE(k, nq) {
    float ev[8], xv[8];
    ldRow<8>(e + 8 * k, ev);
    ldRow<8>(x + 8 * k, xv);
#pragma unroll
    for (int i = 0; i < 8; i++) xv[i] = fmaf(scale, ev[i], xv[i]);
    stRow<8>(x + 8 * k, xv);
  }
}
// beta = sc[2] / sc[0]; p = z + beta p
template <typename V, int W>
__global__ void __launch_bounds__(256) kUpdatePQuad(const double *__restrict__ sc, const V *__restrict__ z,
                                                    V *__restrict__ p, int64_t nq) {
  const float beta = sc[0] != 0.0 ? (float)(sc[2] / sc[0]) : 0.0f;
  QUAD_STRIDE(k, nq) {
    float zv[W], pv[W];
    ldRow<W>(z + W * k, zv);
    ldRow<W>(p + W * k, pv);
#pragma unroll
    for (int i = 0; i < W; i++) pv[i] = fmaf(beta, pv[i], zv[i]);
    stRow<W>(p + W * k, pv);
  }
}

// ---------------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------------
__global__ void kNbrTable(const int32_t *__restrict__ active, int64_t nAct, int nbx, int nby, int nbz,
                          const int32_t *__restrict__ slot, int32_t *__restrict__ nbr, int32_t *__restrict__ even,
                          uint8_t *__restrict__ bpar) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nAct) return;
  const int bid = active[s];
  const int bx = bid % nbx, by = (bid / nbx) % nby, bz = bid / (nbx * nby);
  const int dx[6] = {-1, 1, 0, 0, 0, 0}, dy[6] = {0, 0, -1, 1, 0, 0}, dz[6] = {0, 0, 0, 0, -1, 1};
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int x = bx + dx[k], y = by + dy[k], z = bz + dz[k];
    int v = -1;
    if (x >= 0 && y >= 0 && z >= 0 && x < nbx && y < nby && z < nbz) v = slot[((int64_t)z * nby + y) * nbx + x];
    nbr[s * 6 + k] = v;
  }
  if (even) even[s] = ((bx + by + bz) & 1) == 0;
  bpar[s] = (uint8_t)((bx & 1) | ((by & 1) << 1) | ((bz & 1) << 2));
}
__global__ void kParityList(const int32_t *__restrict__ even, const int64_t *__restrict__ off, int64_t nAct,
                            const int64_t *__restrict__ nEvenPtr, int32_t *__restrict__ list) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nAct) return;
  const int64_t nEven = *nEvenPtr;
  list[even[s] ? off[s] : nEven + (s - off[s])] = (int32_t)s;
}

int blkBuildTables(msbg_gpu_ctx *ctx, PoissonState *ps) {
  const MgLevel &L0 = ps->levels[0];
  const int64_t n = L0.nAct;
  MSBG_CUDA(ctx, cudaMalloc(&ps->dNbr, (size_t)(n > 0 ? n : 1) * 6 * 4));
  MSBG_CUDA(ctx, cudaMalloc(&ps->dParList, (size_t)(n > 0 ? n : 1) * 4));
  MSBG_CUDA(ctx, cudaMalloc(&ps->dBpar, (size_t)(n > 0 ? n : 1)));
  int rc;
  if ((rc = ensureTmpSlab(ctx, (size_t)(n + 1) * 12 + 64))) return rc;
  int32_t *even = (int32_t *)ctx->dTmpSlab;
  int64_t *off = (int64_t *)((char *)ctx->dTmpSlab + (((size_t)(n + 1) * 4 + 15) & ~size_t(15)));
  if (n > 0) {
    MSBG_LAUNCH(ctx, kNbrTable, gridFor(n, 256), 256, 0, L0.active, n, L0.nbx, L0.nby, L0.nbz, L0.slot, ps->dNbr,
                even, ps->dBpar);
  }
  if ((rc = exclusiveScanFlags(ctx, even, n, off, ctx->dCounters + 6))) return rc;
  if (n > 0) MSBG_LAUNCH(ctx, kParityList, gridFor(n, 256), 256, 0, even, off, n, ctx->dCounters + 6, ps->dParList);
  int64_t ne = 0;
  MSBG_CUDA(ctx, cudaMemcpyAsync(&ne, ctx->dCounters + 6, 8, cudaMemcpyDeviceToHost, ctx->stream));
  MSBG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ps->nEven = ne;
  return MSBG_GPU_OK;
}

int blkNbrTable(msbg_gpu_ctx *ctx, const MgLevel &L, int32_t *nbr, uint8_t *bpar) {
  if (L.nAct > 0)
    MSBG_LAUNCH(ctx, kNbrTable, gridFor(L.nAct, 256), 256, 0, L.active, L.nAct, L.nbx, L.nby, L.nbz, L.slot, nbr,
                (int32_t *)nullptr, bpar);
  return MSBG_GPU_OK;
}

BlkGeom blkOf(const PoissonState *ps, const MgLevel &L) {
  BlkGeom g;
  g.bs = L.bs; g.log2bs = L.log2bs; g.nAct = L.nAct;
  g.nbr = ps->dNbr; g.parList = ps->dParList; g.nEven = ps->nEven; g.bpar = ps->dBpar;
  return g;
}

// ---------------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------------
template <typename V, int CPT>
static int applyLaunch(msbg_gpu_ctx *ctx, PoissonState *ps, const MgLevel &Lv, const PrecSet &P, size_t l,
                       const V *x, const V *b, V *y, int mode, double *dotOut, V *bc, V *xc, __half *rhOut,
                       float rhScale, int gridCap) {
  const int64_t nSeg = Lv.nCell / CPT;
  int64_t grid = (nSeg + 255) / 256;
  if (grid > gridCap) grid = gridCap;
  if (grid < 1) grid = 1;
  const BlkGeom gg = blkOf(ps, Lv);
  const V *cx = (const V *)P.cx[l], *cy = (const V *)P.cy[l], *cz = (const V *)P.cz[l], *d = (const V *)P.d[l];
  double *part = dotOut ? ps->dPartial : nullptr;
  if (mode == 0)
    MSBG_LAUNCH(ctx, (kApplyRows<V, 0, CPT>), (unsigned)grid, 256, 0, gg, x, b, cx, cy, cz, d, y, part, bc, xc,
                rhOut, rhScale);
  else if (mode == 1)
    MSBG_LAUNCH(ctx, (kApplyRows<V, 1, CPT>), (unsigned)grid, 256, 0, gg, x, b, cx, cy, cz, d, y, part, bc, xc,
                rhOut, rhScale);
  else if constexpr (CPT == 4)
    MSBG_LAUNCH(ctx, (kApplyRows<V, 2, 4>), (unsigned)grid, 256, 0, gg, x, b, cx, cy, cz, d, y, part, bc, xc,
                rhOut, rhScale);
  else
    return fail(ctx, MSBG_GPU_ERR_UNSUPPORTED, "checked residual on FP16 storage");
  if (dotOut && mode == 2) MSBG_LAUNCH(ctx, kSumPartialsBlk2, 1, kRedThreads, 0, ps->dPartial, (int)grid, dotOut);
  else if (dotOut) MSBG_LAUNCH(ctx, kSumPartialsBlk, 1, kRedThreads, 0, ps->dPartial, (int)grid, dotOut);
  return MSBG_GPU_OK;
}

// Launch-shape autotuner of the operator kernel.  The shape is the block-to-thread
// mapping (cells per thread: 4, or 8 with 16-byte (FP16) / 32-byte (FP32) row loads
// on levels with bs >= 8) and the grid (CTAs of the grid-stride loop).  On the
// first call of a (level, precision, mode) on a level of at least 2^21 cells, each
// candidate runs on the call's own data (every candidate computes the same cells,
// so the repeated launches leave the same outputs) and the fastest is kept for the
// layout; smaller levels, calls during a stream capture, and a context with tuning
// switched off use the static rule (8 cells for FP16 on bs >= 8, else 4; the
// largest grid).  The FP64 dot products of different shapes sum in different
// orders, so they can differ in their last bits, as the reference's thread-local
// reductions do between runs.
template <typename V>
int blkApply(msbg_gpu_ctx *ctx, PoissonState *ps, size_t l, const PrecSet &P, const V *x, const V *b, V *y,
             int mode, double *dotOut, V *bc, V *xc, __half *rhOut, float rhScale) {
  const MgLevel &Lv = ps->levels[l];
  auto launch = [&](int cpt, int cap) -> int {
    if (cpt == 8) return applyLaunch<V, 8>(ctx, ps, Lv, P, l, x, b, y, mode, dotOut, bc, xc, rhOut, rhScale, cap);
    return applyLaunch<V, 4>(ctx, ps, Lv, P, l, x, b, y, mode, dotOut, bc, xc, rhOut, rhScale, cap);
  };
  const bool can8 = Lv.bs >= 8 && mode != 2;
  int cpt = (sizeof(V) == 2 && can8) ? 8 : 4, cap = ps->nPartial;
  const auto key = std::make_tuple((int)l, (int)sizeof(V), mode);
  auto it = ps->applyShape.find(key);
  if (it != ps->applyShape.end()) {
    cpt = it->second >> 16;
    cap = it->second & 0xffff;
  } else if (ps->autotune && Lv.nCell >= (int64_t(1) << 21)) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    MSBG_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cs));
    if (cs == cudaStreamCaptureStatusNone) {
      cudaEvent_t e[2];
      MSBG_CUDA(ctx, cudaEventCreate(&e[0]));
      MSBG_CUDA(ctx, cudaEventCreate(&e[1]));
      float best = 1e30f;
      int rc = MSBG_GPU_OK;
      for (int c : {4, 8}) {
        if (c == 8 && !can8) continue;
        for (int g : {152 * 4, 152 * 8, ps->nPartial}) {
          if ((rc = launch(c, g))) break;  // warm
          cudaEventRecord(e[0], ctx->stream);
          for (int k = 0; k < 2 && !rc; k++) rc = launch(c, g);
          cudaEventRecord(e[1], ctx->stream);
          if (rc) break;
          cudaEventSynchronize(e[1]);
          float ms = 0.f;
          cudaEventElapsedTime(&ms, e[0], e[1]);
          if (ms < best) { best = ms; cpt = c; cap = g; }
        }
        if (rc) break;
      }
      cudaEventDestroy(e[0]);
      cudaEventDestroy(e[1]);
      if (rc) return rc;
      ps->applyShape[key] = (cpt << 16) | cap;
    }
  }
  return launch(cpt, cap);
}

static unsigned quadGrid(const PoissonState *ps, int64_t nq) {
  int64_t g = (nq + 255) / 256;
  if (g > ps->nPartial) g = ps->nPartial;
  return (unsigned)(g < 1 ? 1 : g);
}

// cells per thread and step of the vector kernels: 8 for FP16 (16-byte loads) when n
// allows, else 4
template <typename V>
static int vecWidth(int64_t n) {
  return (sizeof(V) == 2 && n % 8 == 0) ? 8 : 4;
}

template <typename V>
int blkDot(msbg_gpu_ctx *ctx, PoissonState *ps, const V *a, const V *b, int64_t n, double *dOut) {
  const int w = vecWidth<V>(n);
  const unsigned g = quadGrid(ps, n / w);
  if (w == 8) MSBG_LAUNCH(ctx, (kDotQuad<V, 8>), g, 256, 0, a, b, n / 8, ps->dPartial);
  else MSBG_LAUNCH(ctx, (kDotQuad<V, 4>), g, 256, 0, a, b, n / 4, ps->dPartial);
  MSBG_LAUNCH(ctx, kSumPartialsBlk, 1, kRedThreads, 0, ps->dPartial, (int)g, dOut);
  return MSBG_GPU_OK;
}
template <typename V>
int blkUpdateXR(msbg_gpu_ctx *ctx, PoissonState *ps, const double *sc, const V *p, const V *q, V *x, V *r, int64_t n,
                double *rrOut) {
  const int w = vecWidth<V>(n);
  const unsigned g = quadGrid(ps, n / w);
  if (w == 8) MSBG_LAUNCH(ctx, (kUpdateXRQuad<V, 8>), g, 256, 0, sc, p, q, x, r, n / 8, ps->dPartial);
  else MSBG_LAUNCH(ctx, (kUpdateXRQuad<V, 4>), g, 256, 0, sc, p, q, x, r, n / 4, ps->dPartial);
  MSBG_LAUNCH(ctx, kSumPartialsBlk, 1, kRedThreads, 0, ps->dPartial, (int)g, rrOut);
  return MSBG_GPU_OK;
}
int blkAddScaled(msbg_gpu_ctx *ctx, PoissonState *ps, const __half *e, float scale, float *x, int64_t n) {
  if (n % 8) return fail(ctx, MSBG_GPU_ERR_ARG, "add_scaled: %lld cells are not a multiple of 8", (long long)n);
  MSBG_LAUNCH(ctx, kAddScaledQuad, quadGrid(ps, n / 8), 256, 0, e, scale, x, n / 8);
  return MSBG_GPU_OK;
}
template <typename V>
int blkUpdateP(msbg_gpu_ctx *ctx, PoissonState *ps, const double *sc, const V *z, V *p, int64_t n) {
  const int w = vecWidth<V>(n);
  if (w == 8) MSBG_LAUNCH(ctx, (kUpdatePQuad<V, 8>), quadGrid(ps, n / 8), 256, 0, sc, z, p, n / 8);
  else MSBG_LAUNCH(ctx, (kUpdatePQuad<V, 4>), quadGrid(ps, n / 4), 256, 0, sc, z, p, n / 4);
  return MSBG_GPU_OK;
}

// cuTensorMapEncodeTiled from the driver (no link against libcuda)
static PFN_cuTensorMapEncodeTiled_v12000 encodeTiled() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

// Tensor map of a level array viewed as [bs * nAct][bs][bs] with box (bx, by, bz),
// cached per (address, level, box kind).
static int tileMap(msbg_gpu_ctx *ctx, PoissonState *ps, size_t l, const void *ptr, int elem, int kind,
                   const int *T, CUtensorMap *out) {
  const auto key = std::make_tuple(ptr, (int)l, (kind * 8 + elem) * 64 + T[2]);
  auto it = ps->tmaMaps.find(key);
  if (it != ps->tmaMaps.end()) { *out = it->second; return MSBG_GPU_OK; }
  auto fn = encodeTiled();
  if (!fn) return fail(ctx, MSBG_GPU_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const MgLevel &Lv = ps->levels[l];
  const cuuint64_t bs = (cuuint64_t)Lv.bs;
  cuuint64_t dims[3] = {bs, bs, bs * (cuuint64_t)Lv.nAct};
  cuuint64_t strides[2] = {bs * elem, bs * bs * elem};
  cuuint32_t box[3] = {(cuuint32_t)T[0], kind == 1 ? 1u : (cuuint32_t)T[1], kind == 2 ? 1u : (cuuint32_t)T[2]};
  cuuint32_t es[3] = {1, 1, 1};
  CUtensorMap m;
  const CUresult r = fn(&m, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                        const_cast<void *>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, MSBG_GPU_ERR_CUDA, "tensor map encode failed (%d)", (int)r);
  ps->tmaMaps.emplace(key, m);
  *out = m;
  return MSBG_GPU_OK;
}

template <typename V, int BS>
static int smoothLaunch(msbg_gpu_ctx *ctx, PoissonState *ps, const MgLevel &Lv, const PrecSet &P, size_t l, V *x,
                        const V *b, const V *xc, int tc, int k, int reverse, int flags) {
  using Sh = TileShape<BS>;
  constexpr int NT = Sh::NT;
  constexpr size_t smem = tileSmemBytes<V, BS>();
  static SmemOptIn optIn;
  MSBG_CUDA(ctx, optIn((const void *)kTileSmooth<V, BS>, (int)smem));
  const int64_t nUnits = BS == 32 ? Lv.nAct * 4 : (tc == 0 ? ps->nEven : Lv.nAct - ps->nEven);
  if (nUnits <= 0) return MSBG_GPU_OK;
  constexpr int E = (int)sizeof(V);
  const int bx[3] = {Sh::TX, Sh::TY, Sh::TZ};
  TileMaps maps;
  int rc;
  if ((rc = tileMap(ctx, ps, l, x, E, 0, bx, &maps.xM)) || (rc = tileMap(ctx, ps, l, x, E, 1, bx, &maps.xY)) ||
      (rc = tileMap(ctx, ps, l, x, E, 2, bx, &maps.xZ)) || (rc = tileMap(ctx, ps, l, b, E, 0, bx, &maps.b)) ||
      (rc = tileMap(ctx, ps, l, P.d[l], E, 0, bx, &maps.d)) ||
      (rc = tileMap(ctx, ps, l, P.cx[l], E, 0, bx, &maps.cx)) ||
      (rc = tileMap(ctx, ps, l, P.cy[l], E, 0, bx, &maps.cy)) ||
      (rc = tileMap(ctx, ps, l, P.cy[l], E, 1, bx, &maps.cyY)) ||
      (rc = tileMap(ctx, ps, l, P.cz[l], E, 0, bx, &maps.cz)) ||
      (rc = tileMap(ctx, ps, l, P.cz[l], E, 2, bx, &maps.czZ)))
    return rc;
  const int64_t grid = (nUnits + NT - 1) / NT;
  MSBG_LAUNCH(ctx, (kTileSmooth<V, BS>), (unsigned)grid, tileThreads<BS>(), smem, maps, blkOf(ps, Lv), x,
              (const V *)P.cx[l], xc, tc, k, reverse, flags, ctx->dStatus);
  return MSBG_GPU_OK;
}

template <typename V>
int blkSmoothColor(msbg_gpu_ctx *ctx, PoissonState *ps, size_t l, const PrecSet &P, V *x, const V *b,
                   const V *xc, int tileColor, int k, int reverse, int flags) {
  const MgLevel &Lv = ps->levels[l];
  if (Lv.tile == 32) return smoothLaunch<V, 32>(ctx, ps, Lv, P, l, x, b, xc, tileColor, k, reverse, flags);
  if (Lv.tile == 16) return smoothLaunch<V, 16>(ctx, ps, Lv, P, l, x, b, xc, tileColor, k, reverse, flags);
  if (Lv.tile == 8) return smoothLaunch<V, 8>(ctx, ps, Lv, P, l, x, b, xc, tileColor, k, reverse, flags);
  return fail(ctx, MSBG_GPU_ERR_STATE, "level %zu has no tile smoother", l);
}

template int blkApply<float>(msbg_gpu_ctx *, PoissonState *, size_t, const PrecSet &, const float *, const float *,
                             float *, int, double *, float *, float *, __half *, float);
template int blkApply<__half>(msbg_gpu_ctx *, PoissonState *, size_t, const PrecSet &, const __half *,
                              const __half *, __half *, int, double *, __half *, __half *, __half *, float);
#define INST_VEC(V)                                                                                         \
  template int blkDot<V>(msbg_gpu_ctx *, PoissonState *, const V *, const V *, int64_t, double *);                 \
  template int blkUpdateXR<V>(msbg_gpu_ctx *, PoissonState *, const double *, const V *, const V *, V *, V *,     \
                              int64_t, double *);                                                                  \
  template int blkUpdateP<V>(msbg_gpu_ctx *, PoissonState *, const double *, const V *, V *, int64_t);
INST_VEC(float)
INST_VEC(__half)
template int blkSmoothColor<float>(msbg_gpu_ctx *, PoissonState *, size_t, const PrecSet &, float *, const float *,
                                   const float *, int, int, int, int);
template int blkSmoothColor<__half>(msbg_gpu_ctx *, PoissonState *, size_t, const PrecSet &, __half *,
                                    const __half *, const __half *, int, int, int, int);

}  // namespace msbg
