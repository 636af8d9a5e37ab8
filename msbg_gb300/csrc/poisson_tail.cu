// The multigrid's small levels in one launch.
//
// Below the tile-smoothed levels a V-cycle runs pointwise red-black sweeps on levels of a
// few hundred to a few hundred thousand cells (block edges 4, 2, 1 and the aggregated
// blocks), 24 half sweeps each at the default parameters, and the exact coarsest solve:
// about 100 launches whose work is a fraction of a launch's cost.  Here one cooperative
// kernel walks down and up that part of the cycle.  Its phases (a half sweep, residual and
// restriction, prolongation) are separated by a grid barrier on the levels that one CTA
// does not hold, and by __syncthreads on the rest, which CTA 0 runs alone with the level's x
// in shared memory.
//
// Every level is a set of blocks with a table of their six face neighbours (aggregated
// levels: blocks of one cell), so no cell decodes a block id; aggregated levels also have
// tables of parents and children.  Sweeps read x past L1 (ld.cg), as other SMs write it;
// the coefficients stay in L1 over the sweeps.
//
// Bound: latency, of a barrier and of one L2 read chain per phase.  Measured on the 512^3
// layout (14.2 M cells, FP32; levels of 221 k, 27.7 k and 3.5 k cells): 265 us a V-cycle in
// place of 98 launches of together 640 us; the solve 9.72 -> 7.47 ms.
#include <cuda_fp16.h>

#include "internal.cuh"
#include "poisson.cuh"

namespace msbg {

constexpr int kTailLevels = 12, kTailThreads = 1024, kTailSmall = 8192;

template <typename V>
struct TailLevel {
  int log2bs, nCell;
  const int32_t *nbr;    // [blocks][6]
  const uint8_t *bpar;   // [blocks]: parities of the block's coordinates
  V *x, *b;
  const V *cx, *cy, *cz, *d;
  const int32_t *parent, *child;  // next level's cell of a cell, a cell's children on the
                                  // previous level [8]; null: blocks of halved edge
};
template <typename V>
struct TailArgs {
  TailLevel<V> lv[kTailLevels];
  int n, firstSmall;  // levels; the first that CTA 0 runs alone
  int npre, npost;    // red-black sweeps before and after the coarser level
  const float *inv;   // inverse of the coarsest operator
  unsigned *bar;      // arrivals; zero at the launch
  int *status;
};

namespace {

template <typename V> __device__ __forceinline__ float ldcgv(const V *p);
template <> __device__ __forceinline__ float ldcgv<float>(const float *p) { return __ldcg(p); }
template <> __device__ __forceinline__ float ldcgv<__half>(const __half *p) { return __half2float(__ldcg(p)); }

// The x a phase works on: global memory, or shared memory (CTA 0's levels).
template <typename V, bool SM>
struct XRef {
  V *p;
  __device__ __forceinline__ float ld(int i) const {
    if constexpr (SM) return ldv(p + i); else return ldcgv<V>(p + i);
  }
  __device__ __forceinline__ void st(int i, float v) const { stv(p + i, v); }
};

struct Nb {
  int xm, xp, ym, yp, zm, zp;
};
// neighbours of cell (lx, ly, lz) of block s, index c; -1: none
__device__ __forceinline__ Nb nbOf(const int32_t *__restrict__ nbr, int L, int s, int lx, int ly, int lz, int c) {
  const int32_t *t = nbr + 6 * (int64_t)s;
  Nb n;
  if (L == 0) {
    n.xm = t[0]; n.xp = t[1]; n.ym = t[2]; n.yp = t[3]; n.zm = t[4]; n.zp = t[5];
    return n;
  }
  const int m = (1 << L) - 1;
  auto far = [&](int dir, int off) {  // the cell on the opposite face of the neighbour block
    const int q = t[dir];
    return q < 0 ? -1 : c + (q - s) * (1 << (3 * L)) + off;
  };
  n.xm = lx > 0 ? c - 1 : far(0, m);
  n.xp = lx < m ? c + 1 : far(1, -m);
  n.ym = ly > 0 ? c - (1 << L) : far(2, m << L);
  n.yp = ly < m ? c + (1 << L) : far(3, -(m << L));
  n.zm = lz > 0 ? c - (1 << (2 * L)) : far(4, m << (2 * L));
  n.zp = lz < m ? c + (1 << (2 * L)) : far(5, -(m << (2 * L)));
  return n;
}
__device__ __forceinline__ int parityOf(uint8_t b) { return (b ^ (b >> 1) ^ (b >> 2)) & 1; }

// sum of c_f x_nb over the faces, added to s with sign (+1: smoother, -1: operator)
template <typename V, bool SM>
__device__ __forceinline__ float faces(const TailLevel<V> &L, const XRef<V, SM> &x, int c, const Nb &n, float s,
                                       float sign) {
  if (n.xm >= 0) s += sign * ldv(L.cx + c) * x.ld(n.xm);
  if (n.xp >= 0) s += sign * ldv(L.cx + n.xp) * x.ld(n.xp);
  if (n.ym >= 0) s += sign * ldv(L.cy + c) * x.ld(n.ym);
  if (n.yp >= 0) s += sign * ldv(L.cy + n.yp) * x.ld(n.yp);
  if (n.zm >= 0) s += sign * ldv(L.cz + c) * x.ld(n.zm);
  if (n.zp >= 0) s += sign * ldv(L.cz + n.zp) * x.ld(n.zp);
  return s;
}

// One half sweep: the cells of one colour get x = (b + sum c x_nb) / d.  ZERO: x is zero on
// entry and is not read; the other colour's cells are set to zero.
template <typename V, bool SM, bool ZERO>
__device__ __forceinline__ void halfSweep(const TailLevel<V> &L, const XRef<V, SM> &x, int color, int t0, int stride) {
  const int l2 = L.log2bs;
  if (l2 == 0) {
    for (int c = t0; c < L.nCell; c += stride) {
      if (parityOf(L.bpar[c]) != color) {
        if (ZERO) x.st(c, 0.0f);
        continue;
      }
      float s = ldcgv<V>(L.b + c);
      if (!ZERO) s = faces<V, SM>(L, x, c, nbOf(L.nbr, 0, c, 0, 0, 0, c), s, 1.0f);
      x.st(c, s / ldv(L.d + c));
    }
    return;
  }
  const int m = (1 << l2) - 1;
  for (int i = t0; i < L.nCell / 2; i += stride) {  // block edges are even: the block's parity is local
    const int blk = i >> (3 * l2 - 1), h = i & ((1 << (3 * l2 - 1)) - 1);
    const int hx = h & ((1 << (l2 - 1)) - 1), ly = (h >> (l2 - 1)) & m, lz = h >> (2 * l2 - 1);
    const int lx = 2 * hx + ((ly + lz + color) & 1);
    const int c = (blk << (3 * l2)) + (((lz << l2) + ly) << l2) + lx;
    float s = ldcgv<V>(L.b + c);
    if (!ZERO) s = faces<V, SM>(L, x, c, nbOf(L.nbr, l2, blk, lx, ly, lz, c), s, 1.0f);
    x.st(c, s / ldv(L.d + c));
    if (ZERO) x.st(c ^ 1, 0.0f);
  }
}

// Child k (x, y, z bits) of cell p of the coarser level, -1: none
template <typename V>
__device__ __forceinline__ int childOf(const TailLevel<V> &F, const TailLevel<V> &C, int p, int k) {
  if (C.child) return C.child[8 * (int64_t)p + k];
  const int lc = C.log2bs, lf = F.log2bs, mc = (1 << lc) - 1;
  const int blk = p >> (3 * lc), v = p & ((1 << (3 * lc)) - 1);
  const int lx = 2 * (v & mc) + (k & 1), ly = 2 * ((v >> lc) & mc) + ((k >> 1) & 1), lz = 2 * (v >> (2 * lc)) + (k >> 2);
  return (blk << (3 * lf)) + (((lz << lf) + ly) << lf) + lx;
}

// Coarse right-hand side: the sum of the children's residuals b - A x, eight lanes a cell.
template <typename V, bool SM>
__device__ __forceinline__ void restrictResidual(const TailLevel<V> &F, const TailLevel<V> &C, const XRef<V, SM> &x,
                                                 int t0, int stride) {
  const int l2 = F.log2bs, m = (1 << l2) - 1;
  const int n = C.nCell * 8, nPad = (n + 31) & ~31;
  for (int i = t0; i < nPad; i += stride) {  // strides are whole warps
    float r = 0.0f;
    if (i < n) {
      const int c = childOf(F, C, i >> 3, i & 7);
      if (c >= 0) {
        const int blk = c >> (3 * l2), v = c & ((1 << (3 * l2)) - 1);
        const float ax = faces<V, SM>(F, x, c, nbOf(F.nbr, l2, blk, v & m, (v >> l2) & m, v >> (2 * l2), c),
                                      ldv(F.d + c) * x.ld(c), -1.0f);
        r = ldcgv<V>(F.b + c) - ax;
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (i < n && (i & 7) == 0) stv(C.b + (i >> 3), r);
  }
}

// x += the parent's value
template <typename V, bool SM>
__device__ __forceinline__ void prolong(const TailLevel<V> &F, const TailLevel<V> &C, const XRef<V, SM> &x, int t0,
                                        int stride) {
  const int lf = F.log2bs, lc = C.log2bs, mf = (1 << lf) - 1;
  for (int c = t0; c < F.nCell; c += stride) {
    int p;
    if (F.parent) {
      p = F.parent[c];
    } else {
      const int blk = c >> (3 * lf), v = c & ((1 << (3 * lf)) - 1);
      const int px = (v & mf) >> 1, py = ((v >> lf) & mf) >> 1, pz = (v >> (2 * lf)) >> 1;
      p = (blk << (3 * lc)) + (((pz << lc) + py) << lc) + px;
    }
    if (p >= 0) x.st(c, x.ld(c) + ldcgv<V>(C.x + p));
  }
}

// Barrier over the grid's CTAs (co-resident: cooperative launch); false after the limit.
__device__ __forceinline__ bool gridBarrier(unsigned *bar, unsigned target) {
  bool ok = true;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned v = 0;
    int it = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (++it >= (1 << 22)) { ok = false; break; }
    } while (v < target);
  }
  return __syncthreads_and(ok);
}

template <typename V, bool SM, typename Sync>
__device__ __forceinline__ bool smooth(const TailLevel<V> &L, const XRef<V, SM> &x, int sweeps, bool reverse, bool zero,
                                       int t0, int stride, Sync sync) {
  if (zero && sweeps == 0) {
    for (int c = t0; c < L.nCell; c += stride) x.st(c, 0.0f);
    return sync();
  }
  for (int h = 0; h < 2 * sweeps; h++) {
    const int color = reverse ? 1 - (h & 1) : h & 1;
    if (zero && h == 0) halfSweep<V, SM, true>(L, x, color, t0, stride);
    else halfSweep<V, SM, false>(L, x, color, t0, stride);
    if (!sync()) return false;
  }
  return true;
}

// CTA 0's levels l.. : x of the current level in xs
template <typename V>
__device__ void smallLevels(const TailArgs<V> &a, V *xs, int first) {
  const int tid = threadIdx.x;
  auto sync = [] { __syncthreads(); return true; };
  const XRef<V, true> x{xs};
  for (int l = first; l + 1 < a.n; l++) {
    const TailLevel<V> &L = a.lv[l];
    smooth<V, true>(L, x, a.npre, false, true, tid, kTailThreads, sync);
    restrictResidual<V, true>(L, a.lv[l + 1], x, tid, kTailThreads);
    for (int c = tid; c < L.nCell; c += kTailThreads) L.x[c] = xs[c];
    __syncthreads();
  }
  {
    const TailLevel<V> &L = a.lv[a.n - 1];  // x = inverse b, one warp per row
    const int n = L.nCell, lane = tid & 31;
    for (int c = tid; c < n; c += kTailThreads) xs[c] = L.b[c];
    __syncthreads();
    for (int row = tid >> 5; row < n; row += kTailThreads / 32) {
      const float *q = a.inv + (int64_t)row * n;
      float s = 0.f;
#pragma unroll 4
      for (int j = lane; j < n; j += 32) s = fmaf(q[j], ldv(xs + j), s);
#pragma unroll
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) stv(L.x + row, s);
    }
    __syncthreads();
  }
  for (int l = a.n - 2; l >= first; l--) {
    const TailLevel<V> &L = a.lv[l];
    for (int c = tid; c < L.nCell; c += kTailThreads) xs[c] = L.x[c];
    __syncthreads();
    prolong<V, true>(L, a.lv[l + 1], x, tid, kTailThreads);
    __syncthreads();
    smooth<V, true>(L, x, a.npost, true, false, tid, kTailThreads, sync);
    for (int c = tid; c < L.nCell; c += kTailThreads) L.x[c] = xs[c];
    __syncthreads();
  }
}

template <typename V>
__global__ void __launch_bounds__(kTailThreads, 1) kCoarseTail(const __grid_constant__ TailArgs<V> a) {
  __shared__ V xs[kTailSmall];
  const int t0 = blockIdx.x * kTailThreads + threadIdx.x, stride = gridDim.x * kTailThreads;
  unsigned target = 0;
  bool ok = true;
  auto sync = [&] {
    target += gridDim.x;
    ok = gridBarrier(a.bar, target);
    return ok;
  };
  for (int l = 0; l < a.firstSmall && ok; l++) {
    const XRef<V, false> x{a.lv[l].x};
    if (!smooth<V, false>(a.lv[l], x, a.npre, false, true, t0, stride, sync)) break;
    restrictResidual<V, false>(a.lv[l], a.lv[l + 1], x, t0, stride);
    sync();
  }
  if (ok && blockIdx.x == 0) smallLevels<V>(a, xs, a.firstSmall);
  if (ok && a.firstSmall > 0) sync();
  for (int l = a.firstSmall - 1; l >= 0 && ok; l--) {
    const XRef<V, false> x{a.lv[l].x};
    prolong<V, false>(a.lv[l], a.lv[l + 1], x, t0, stride);
    if (!sync()) break;
    smooth<V, false>(a.lv[l], x, a.npost, true, false, t0, stride, sync);
  }
  if (!ok && threadIdx.x == 0) atomicOr(a.status, 32);
}

// parent of every cell of the finer level (blocks of one cell), children of every coarse one
__global__ void kParentChild(const int32_t *__restrict__ activeF, int64_t n, int nbxF, int nbyF,
                             const int32_t *__restrict__ slotC, int nbxC, int nbyC, int32_t *__restrict__ parent,
                             int32_t *__restrict__ child) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int bid = activeF[i];
  const int bx = bid % nbxF, by = (bid / nbxF) % nbyF, bz = bid / (nbxF * nbyF);
  const int p = slotC[((int64_t)(bz >> 1) * nbyC + (by >> 1)) * nbxC + (bx >> 1)];
  parent[i] = p;
  child[8 * (int64_t)p + (bx & 1) + 2 * (by & 1) + 4 * (bz & 1)] = (int32_t)i;
}

}  // namespace

int tailBuildTables(msbg_gpu_ctx *ctx, PoissonState *ps) {
  MSBG_CUDA(ctx, cudaMalloc(&ps->dTailBar, sizeof(unsigned)));
  for (size_t l = 1; l < ps->levels.size(); l++) {
    MgLevel &F = ps->levels[l - 1], &C = ps->levels[l];
    if (C.sameSet) continue;
    const size_t n = (size_t)(C.nAct > 0 ? C.nAct : 1), nf = (size_t)(F.nAct > 0 ? F.nAct : 1);
    MSBG_CUDA(ctx, cudaMalloc(&C.nbr, n * 6 * 4));
    MSBG_CUDA(ctx, cudaMalloc(&C.bpar, n));
    MSBG_CUDA(ctx, cudaMalloc(&C.child, n * 8 * 4));
    MSBG_CUDA(ctx, cudaMalloc(&F.parent, nf * 4));
    MSBG_CUDA(ctx, cudaMemsetAsync(C.child, 0xff, n * 8 * 4, ctx->stream));
    if (C.nAct <= 0 || F.nAct <= 0) continue;
    int rc;
    if ((rc = blkNbrTable(ctx, C, C.nbr, C.bpar))) return rc;
    MSBG_LAUNCH(ctx, kParentChild, gridFor(F.nAct, 256), 256, 0, F.active, F.nAct, F.nbx, F.nby, C.slot, C.nbx, C.nby,
                F.parent, C.child);
  }
  return MSBG_GPU_OK;
}

// The V-cycle of the levels from l in one launch.  *done: whether this form takes them: every
// one is relaxed pointwise, the coarsest is solved by its inverse, and level l has at most
// kTailMaxCells cells.
template <typename V>
int coarseTail(msbg_gpu_ctx *ctx, PoissonState *ps, const PrecSet &P, size_t l, bool *done) {
  *done = false;
  const size_t nL = ps->levels.size();
  if (ps->coarsestIter > 0 || !ps->coarseInvValid || l + 1 >= nL || nL - l > kTailLevels) return MSBG_GPU_OK;
  if (ps->levels[l].tile || ps->levels[l].nCell > kTailMaxCells || ps->levels[nL - 1].nCell > kTailSmall)
    return MSBG_GPU_OK;
  TailArgs<V> a;
  a.n = (int)(nL - l);
  a.firstSmall = a.n - 1;
  for (int k = 0; k < a.n; k++) {
    const MgLevel &L = ps->levels[l + k];
    if (L.tile || L.nCell <= 0) return MSBG_GPU_OK;
    TailLevel<V> &t = a.lv[k];
    t.log2bs = L.log2bs;
    t.nCell = (int)L.nCell;
    t.nbr = L.sameSet ? ps->dNbr : L.nbr;
    t.bpar = L.sameSet ? ps->dBpar : L.bpar;
    t.x = (V *)P.x[l + k]; t.b = (V *)P.b[l + k];
    t.cx = (const V *)P.cx[l + k]; t.cy = (const V *)P.cy[l + k]; t.cz = (const V *)P.cz[l + k];
    t.d = (const V *)P.d[l + k];
    t.parent = L.parent;
    t.child = L.child;
    if (L.nCell <= kTailSmall && k < a.firstSmall) a.firstSmall = k;
  }
  a.npre = ps->preSweeps * ps->tileIters;
  a.npost = ps->postSweeps * ps->tileIters;
  a.inv = ps->dCoarseInv;
  a.bar = ps->dTailBar;
  a.status = ctx->dStatus;
  int dev = 0, nSm = 0;
  MSBG_CUDA(ctx, cudaGetDevice(&dev));
  MSBG_CUDA(ctx, cudaDeviceGetAttribute(&nSm, cudaDevAttrMultiProcessorCount, dev));
  // one CTA per SM at most (co-resident), and no more than the largest half sweep has threads for
  int64_t grid = (a.lv[0].nCell / 2 + kTailThreads - 1) / kTailThreads;
  if (grid > nSm) grid = nSm;
  if (grid < 1 || a.firstSmall == 0) grid = 1;
  // The counter starts at zero for every launch: one that a kernel's last CTA had reset stayed
  // as it was when a wait gave up, and the next launch's phases would not have been separated.
  MSBG_CUDA(ctx, cudaMemsetAsync(ps->dTailBar, 0, sizeof(unsigned), ctx->stream));
  void *args[] = {&a};
  MSBG_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)kCoarseTail<V>, dim3((unsigned)grid), dim3(kTailThreads), args, 0,
                                             ctx->stream));
  ctx->launches++;
  *done = true;
  return MSBG_GPU_OK;
}

int tailCounterGaveUp(msbg_gpu_ctx *ctx) {
  if (ctx->poisson && ctx->poisson->dTailBar)
    MSBG_CUDA(ctx, cudaMemsetAsync(ctx->poisson->dTailBar, 0x01, sizeof(unsigned), ctx->stream));
  return MSBG_GPU_OK;
}

template int coarseTail<float>(msbg_gpu_ctx *, PoissonState *, const PrecSet &, size_t, bool *);
template int coarseTail<__half>(msbg_gpu_ctx *, PoissonState *, const PrecSet &, size_t, bool *);

}  // namespace msbg
