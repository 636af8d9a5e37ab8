// Restriction of a channel to the next coarser multigrid level:
// downsampleFloatChannelNew (src/msbg4.cpp:1035-1379) for the value blocks, the
// case levelMg = 1 of a layout whose value blocks are the level-0 blocks.
//
// A coarse cell v (block edge bs/2) is the sum over the fine cells 2v-1 .. 2v+2
// with weights (1,3,3,1)x(1,3,3,1)x(1,3,3,1)/512 (G3D_GetGausslikeKernel4x4x4,
// src/grid.c:30-70), or with simpleAverage the mean of its 8 children
// (OPT_SIMPLE_AVERAGE).  The fine halo is that of fillHaloBlock_ with
// OPT_BC_COARSE_LEVEL (src/halo.cpp:266-479, src/halo.h:288-300): a cell outside
// the domain takes the value at the clamped position, a cell in a block without
// payload the channel's empty value (0).
//
// Summation order, shared with the CPU restatement: per x offset i and row j an
// accumulator over the 4 planes, S[j][i] = fma(w, f, S[j][i]); then per i
// T[i] = ((S0 + S1) + S2) + S3 and the value (T0 + T1) + (T2 + T3).  This is the
// reference's four 4-wide accumulators (one per row, lanes = x offsets) and its
// horizontal add.
//
// One CTA per value block, one thread per two coarse (x, y) columns (neighbours in y, which
// share two of their fine rows), marching the coarse planes in z.  Fine planes with their 1-cell x/y halo are staged as FP32
// in a 4-plane shared-memory ring ([bs+2][bs+2] each, rows coalesced along x), two
// new planes per coarse plane, so each fine plane is read from memory once; the
// loads of the next two planes are in flight while the current two are used.  Each
// thread carries the 32 partial sums of its cells of the coarse plane above in registers.
// The planes in flight are kept as stored and widened when they are put into the ring:
// a conversion at the load would wait for it.  The thread's ring cells are looked up
// once for the block's own z-layer, the sums run in column pairs on the packed FP32
// pipe (the same operations per column).  Floor: S bytes per fine cell read, 4 per
// coarse cell written (236 M FP16 cells: 85 us); measured 322 us with per-plane lookups
// and conversions at the load, 274 with the lookups and the pairs of columns alone, 199
// with planes as stored, 193 with the rows' stores in different banks, 177 with two cells
// a thread (six row reads for two cells where one takes four; the shared-memory pipe was
// 84% busy).  Five CTAs a SM instead of four (96 registers): 180.
#include "internal.cuh"

namespace msbg {

// Four consecutive values of a block row as stored (one 8- or 16-byte load; x is a multiple of
// 4), and as floats, converted as Store<T>::load does.
template <typename T> struct Quad { using V = uint2; };
template <> struct Quad<float> { using V = float4; };
__device__ __forceinline__ void quadVals(const float4 &q, float v[4], const float *) {
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void quadVals(const uint2 &q, float v[4], const __half *) {
  const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&q.x));
  const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&q.y));
  v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
}
__device__ __forceinline__ void quadVals(const uint2 &q, float v[4], const uint16_t *) {
  v[0] = __fmul_rn((float)(q.x & 0xffffu), kU16ToF);
  v[1] = __fmul_rn((float)(q.x >> 16), kU16ToF);
  v[2] = __fmul_rn((float)(q.y & 0xffffu), kU16ToF);
  v[3] = __fmul_rn((float)(q.y >> 16), kU16ToF);
}

template <int BS>
constexpr int dsThreads() {
  return BS / 2 * BS / 4 < 32 ? 32 : BS / 2 * BS / 4;
}

template <typename T, int BS, bool SIMPLE>
__global__ void __launch_bounds__(dsThreads<BS>(), 4) kDownsample(const T *__restrict__ pay,
                                                                 const int32_t *__restrict__ active,
                                                                 const int32_t *__restrict__ slot, int nbx,
                                                                 int nby, int nbz, float *__restrict__ out) {
  constexpr int NT = dsThreads<BS>(), CB = BS / 2, H = BS + 2, HH = H * H;
  constexpr int L = BS == 32 ? 5 : BS == 16 ? 4 : 3, m = BS - 1;
  __shared__ __align__(16) float st[4 * HH];  // fine plane p (-1..BS) in slot (p + 1) & 3
  __shared__ int nbs[27];
  const int t = blockIdx.x, tid = threadIdx.x;
  const int bid = active[t];
  const int bx = bid % nbx, by = (bid / nbx) % nby, bz = bid / (nbx * nby);
  if (tid < 27) {
    const int x = bx + tid % 3 - 1, y = by + (tid / 3) % 3 - 1, z = bz + tid / 9 - 1;
    int s = -1;  // outside the domain: never read (coordinates are clamped first)
    if (x >= 0 && y >= 0 && z >= 0 && x < nbx && y < nby && z < nbz)
      s = slot[(int64_t)z * nbx * nby + (int64_t)y * nbx + x];
    nbs[tid] = s;
  }
  __syncthreads();
  const int sx = nbx << L, sy = nby << L, sz = nbz << L;
  // Fine plane p (local z) with its x/y halo.  The plane's BS x BS interior comes
  // from one block (the own block, its z-neighbour, or the clamped own plane at the
  // domain face), 4 consecutive values per thread; the ring of 4 (BS + 1) halo cells
  // goes cell by cell.  fetch issues the loads into registers, put stores them into
  // the ring slot.
  constexpr int NI = BS * BS / 4, NR = 4 * (BS + 1), PR = (NR + NT - 1) / NT, PQ = (NI + NT - 1) / NT;
  // a plane's values as stored: a conversion here would wait for the loads it follows
  struct Plane {
    typename Quad<T>::V in[PQ];
    T ring[PR];
  };
  const T zero = T(0.0f);  // the empty value
  // ring cell e: rows 0 and H-1 (e < 2H), then columns 0 and H-1 of rows 1..H-2
  auto ringAt = [](int e, int &r, int &c) {
    if (e < 2 * H) { r = e < H ? 0 : H - 1; c = e < H ? e : e - H; }
    else { const int f = e - 2 * H; r = 1 + (f >> 1); c = (f & 1) ? H - 1 : 0; }
  };
  // the thread's ring cells in the block's own z-layer: their source in plane 0 (null: an empty
  // block) and their place in a ring slot (-1: none)
  const T *ringSrc[PR];
  int ringDst[PR];
#pragma unroll
  for (int k = 0; k < PR; k++) {
    const int e = tid + k * NT;
    ringSrc[k] = nullptr;
    ringDst[k] = -1;
    if (e < NR) {
      int r, c;
      ringAt(e, r, c);
      ringDst[k] = r * H + c;
      const int gy = min(max((by << L) + r - 1, 0), sy - 1), gx = min(max((bx << L) + c - 1, 0), sx - 1);
      const int sn = nbs[9 + 1 + ((gy >> L) - by + 1) * 3 + (gx >> L) - bx];
      if (sn >= 0) ringSrc[k] = pay + ((int64_t)sn << (3 * L)) + ((gy & m) << L) + (gx & m);
    }
  }
  const T *quadSrc = pay + ((int64_t)t << (3 * L)) + 4 * tid;
  auto fetch = [&](int p, Plane &v) {
    if (p >= 0 && p < BS) {
#pragma unroll
      for (int k = 0; k < PQ; k++)
        if (tid + k * NT < NI)
          v.in[k] = *reinterpret_cast<const typename Quad<T>::V *>(quadSrc + 4 * NT * k + (p << (2 * L)));
#pragma unroll
      for (int k = 0; k < PR; k++)
        v.ring[k] = ringSrc[k] ? ringSrc[k][p << (2 * L)] : zero;
      return;
    }
    const int gz = min(max((bz << L) + p, 0), sz - 1);
    const int nz = ((gz >> L) - bz + 1) * 9 + 1;
    const int64_t zoff = (int64_t)(gz & m) << (2 * L);
    const int sc = nbs[nz + 3];  // the block above / below (or the own block)
#pragma unroll
    for (int k = 0; k < PQ; k++) {
      v.in[k] = {};
      if (sc >= 0 && tid + k * NT < NI)
        v.in[k] = *reinterpret_cast<const typename Quad<T>::V *>(pay + ((int64_t)sc << (3 * L)) + zoff + 4 * (tid + k * NT));
    }
#pragma unroll
    for (int k = 0; k < PR; k++) {
      const int e = tid + k * NT;
      v.ring[k] = zero;
      if (e < NR) {
        int r, c;
        ringAt(e, r, c);
        const int gy = min(max((by << L) + r - 1, 0), sy - 1), gx = min(max((bx << L) + c - 1, 0), sx - 1);
        const int sn = nbs[nz + ((gy >> L) - by + 1) * 3 + (gx >> L) - bx];
        if (sn >= 0) v.ring[k] = pay[((int64_t)sn << (3 * L)) + zoff + ((gy & m) << L) + (gx & m)];
      }
    }
  };
  auto put = [&](int p, const Plane &v) {
    float *dst = st + ((p + 1) & 3) * HH;
#pragma unroll
    for (int u = 0; u < PQ; u++) {
      const int e = tid + u * NT;
      if (e >= NI) break;
      const int r = (4 * e) >> L, c = (4 * e) & m;
      float *q = dst + (r + 1) * H + c + 1;
      float in[4];
      quadVals(v.in[u], in, (const T *)nullptr);
      // 32-wide rows: two pairs of rows of a warp lie in the same banks for one k; the second
      // pair stores its values in the order 1, 0, 3, 2
      const int sw = BS == 32 ? (e >> 4) & 1 : 0;
#pragma unroll
      for (int k = 0; k < 4; k++) q[k ^ sw] = sw ? in[k ^ 1] : in[k];
    }
#pragma unroll
    for (int k = 0; k < PR; k++)
      if (ringDst[k] >= 0) dst[ringDst[k]] = Store<T>::load(&v.ring[k]);
  };
  const bool own = tid < CB * CB / 2;
  const int vx = tid & (CB - 1), vy = 2 * (tid / CB);  // coarse cells (vx, vy) and (vx, vy + 1)
  // exact weights k1[k] k1[j] k1[i] / 512 of (plane k, row j, columns i = 2h, 2h + 1)
  auto wgt = [](int k, int j, int h) {
    const float k1[4] = {1.f, 3.f, 3.f, 1.f};
    return make_float2(k1[k] * k1[j] * k1[2 * h] / 512.0f, k1[k] * k1[j] * k1[2 * h + 1] / 512.0f);
  };
  // row j (fine row 2vy-1+j, columns 2vx-1 .. 2vx+2) of fine plane p
  auto row = [&](int p, int j, float2 (&r)[2]) {
    const float *src = st + ((p + 1) & 3) * HH + (2 * vy + j) * H + 2 * vx;
    r[0] = *reinterpret_cast<const float2 *>(src);
    r[1] = *reinterpret_cast<const float2 *>(src + 2);
  };
  // Coarse plane vz reads fine planes 2vz-1 .. 2vz+2 (k = 0..3).  The accumulators of
  // plane vz over k = 0, 1 come from the previous pair of fine planes; the pair
  // (2vz+1, 2vz+2) completes them (k = 2, 3) and starts those of plane vz+1.  The
  // next pair's loads are in flight while a pair is used.
  const float2 zero2 = make_float2(0.0f, 0.0f);
  float2 acc[2][4][2];  // [cell][j][h]: columns 2h, 2h + 1 over k = 0, 1
  float part[2] = {0.0f, 0.0f};  // the children sums in plane 2vz
  // Fine-plane pairs go through two register sets (A: pairs of even coarse planes, B:
  // odd), so the loads of the next two pairs are in flight while a pair is used.
  Plane va, vb, vc, vd;
  fetch(-1, va);
  fetch(0, vb);
  put(-1, va);
  put(0, vb);
  __syncthreads();
  fetch(1, va);
  fetch(2, vb);
  fetch(3, vc);
  fetch(4, vd);
  if (own) {
#pragma unroll
    for (int j = 0; j < 6; j++) {
      float2 r0[2], r1[2];
      row(-1, j, r0);
      row(0, j, r1);
#pragma unroll
      for (int y = 0; y < 2; y++) {
        const int jy = j - 2 * y;  // row of cell vy + y
        if (jy < 0 || jy > 3) continue;
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (!SIMPLE) acc[y][jy][h] = __ffma2_rn(wgt(1, jy, h), r1[h], __ffma2_rn(wgt(0, jy, h), r0[h], zero2));
        if (SIMPLE && jy == 1) part[y] = __fadd_rn(r1[0].y, r1[1].x);
        if (SIMPLE && jy == 2) part[y] = __fadd_rn(__fadd_rn(part[y], r1[0].y), r1[1].x);
      }
    }
  }
  // one coarse plane from the pair (p, q) of fine planes 2vz+1, 2vz+2
  auto step = [&](int vz, Plane &p, Plane &q) {
    // the pair's ring slots are not the previous pair's, whose last reads were
    // before the previous barrier
    put(2 * vz + 1, p);
    put(2 * vz + 2, q);
    __syncthreads();
    if (vz + 2 < CB) {  // the pair after next into the registers just emptied
      fetch(2 * vz + 5, p);
      fetch(2 * vz + 6, q);
    }
    if (!own) return;
    float2 T2[2][2];
    float sum[2] = {part[0], part[1]};
#pragma unroll
    for (int j = 0; j < 6; j++) {
      float2 r2[2], r3[2];
      row(2 * vz + 1, j, r2);
      row(2 * vz + 2, j, r3);
#pragma unroll
      for (int y = 0; y < 2; y++) {
        const int jy = j - 2 * y;
        if (jy < 0 || jy > 3) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if (SIMPLE) break;
          const float2 S = __ffma2_rn(wgt(3, jy, h), r3[h], __ffma2_rn(wgt(2, jy, h), r2[h], acc[y][jy][h]));
          T2[y][h] = jy == 0 ? S : __fadd2_rn(T2[y][h], S);
          acc[y][jy][h] = __ffma2_rn(wgt(1, jy, h), r3[h], __ffma2_rn(wgt(0, jy, h), r2[h], zero2));
        }
        if (SIMPLE && (jy == 1 || jy == 2)) {  // children in plane 2vz+1 (this cell) and 2vz+2 (the next)
          sum[y] = __fadd_rn(__fadd_rn(sum[y], r2[0].y), r2[1].x);
          part[y] = jy == 1 ? __fadd_rn(r3[0].y, r3[1].x) : __fadd_rn(__fadd_rn(part[y], r3[0].y), r3[1].x);
        }
      }
    }
#pragma unroll
    for (int y = 0; y < 2; y++) {
      const float val = SIMPLE ? __fmul_rn(sum[y], 0.125f)
                               : __fadd_rn(__fadd_rn(T2[y][0].x, T2[y][0].y), __fadd_rn(T2[y][1].x, T2[y][1].y));
      out[(int64_t)t * CB * CB * CB + ((int64_t)vz * CB + vy + y) * CB + vx] = val;
    }
  };
  static_assert(CB % 2 == 0, "coarse planes in pairs");
#pragma unroll 1
  for (int vz = 0; vz < CB; vz += 2) {
    step(vz, va, vb);
    step(vz + 1, vc, vd);
  }
}

template <typename T, int BS>
static int downsampleT(msbg_gpu_ctx *ctx, const Channel &c, float *dDst, int simple) {
  if (simple)
    MSBG_LAUNCH(ctx, (kDownsample<T, BS, true>), (unsigned)ctx->nActive, dsThreads<BS>(), 0, (const T *)c.d,
                ctx->dActive, ctx->dSlot, ctx->nbx, ctx->nby, ctx->nbz, dDst);
  else
    MSBG_LAUNCH(ctx, (kDownsample<T, BS, false>), (unsigned)ctx->nActive, dsThreads<BS>(), 0, (const T *)c.d,
                ctx->dActive, ctx->dSlot, ctx->nbx, ctx->nby, ctx->nbz, dDst);
  return MSBG_GPU_OK;
}

template <typename T>
static int downsampleBs(msbg_gpu_ctx *ctx, const Channel &c, float *dDst, int simple) {
  switch (ctx->bsx) {
    case 8: return downsampleT<T, 8>(ctx, c, dDst, simple);
    case 16: return downsampleT<T, 16>(ctx, c, dDst, simple);
    default: return downsampleT<T, 32>(ctx, c, dDst, simple);
  }
}

}  // namespace msbg

using namespace msbg;

extern "C" int msbg_gpu_downsample_channel(msbg_gpu_ctx *ctx, int chSrc, float *dDst, int simpleAverage) {
  if (!ctx || !dDst) return MSBG_GPU_ERR_ARG;
  if (chSrc < 0 || chSrc >= kMaxChannels || !ctx->ch[chSrc].exists)
    return fail(ctx, MSBG_GPU_ERR_ARG, "channel %d does not exist", chSrc);
  if (!ctx->layoutValid) return fail(ctx, MSBG_GPU_ERR_STATE, "no block layout: call set_refinement_map");
  if (ctx->nActive == 0) return MSBG_GPU_OK;
  const Channel &c = ctx->ch[chSrc];
  switch (c.storage) {
    case MSBG_GPU_F32: return downsampleBs<float>(ctx, c, dDst, simpleAverage);
    case MSBG_GPU_F16: return downsampleBs<__half>(ctx, c, dDst, simpleAverage);
    case MSBG_GPU_U16: return downsampleBs<uint16_t>(ctx, c, dDst, simpleAverage);
    default:
      return fail(ctx, MSBG_GPU_ERR_UNSUPPORTED, "downsample: FP64 channels are not supported");
  }
}
