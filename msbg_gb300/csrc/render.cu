// Ray-march render of the iso-0.5 surface of a value-block channel into an RGB buffer.
//
// Reference: RDR::RaymarchRenderer (src/render.h:52-160, src/render.cpp:20-101), the demo's
// visual check of the splatted and smoothed density (src/msbg_demo.cpp:129-175).  There it
// renders a BMP bitmap on the CPU, one thread per image row; here one thread per pixel
// writes 3 bytes of a device buffer (row-major, top row first), with no graphics API.
//
// Per pixel, in FP64 as the reference (RealType = double):
//  - camera basis forward = normalize(lookAt - pos), right = normalize(cross(forward, +y)),
//    up = cross(right, forward); ndc = ((x + .5)/W - .5) * 2 * aspect, (.5 - (y + .5)/H) * 2;
//    dir = normalize(forward * zoom + right * ndcX + up * ndcY);
//  - the ray starts at the camera and moves by dir / res per step (res = max(sx, sy, sz)),
//    at most 2 units;
//  - density(p) (sampleDensity, src/render.h:89-117): 0 outside the domain or in a block
//    without payload, else the trilinear interpolant at res * p (FP32; uint16 times
//    1/65535);
//  - the first step whose density crosses 0.5 upwards is the hit, placed by linear
//    interpolation; normal = -grad of the cubic B-spline interpolant there
//    (interpolateWithDerivs0<IP_BSPLINE_CUBIC>, src/sbg.h:3903-4133; window voxels outside
//    the domain clamped to it), Lambert shading with the sun, channels rounded to 8 bits.
// Where the reference's -ffast-math build fuses a multiply into an add, the code here uses
// the same fused forms (dot products, cross products, ndc, hit placement); every operation
// is an explicitly rounded intrinsic, so nothing else is contracted.  The CPU restatement
// (orc_render) uses the same forms; both agree with the reference's image except for a
// few pixels one step apart in a colour channel.
//
// A ray that has left the domain on an axis while moving outward on it can never read a
// nonzero density again (positions are monotonic per axis under rounded addition), so it
// stops there; the result is the same as marching to the end.
//
// Marching without the FP64 pipe.  GB300 retires 2 FP64 lanes per clock and SM, and 6 of a
// step's operations were FP64 (88% of that pipe's time).  Inside one binade a repeated
// p <- RN(p + inc) moves p by the same whole number j of its units in the last place each
// time (inc rounded to them), so a step is an integer addition on p's bit pattern, and n
// steps through space that is known to read 0 are one addition of n j.  Space known to be
// empty: the ray's block, or the aligned 4^3 or 16^3 group of blocks around it, from two
// occupancy maps built per call (one pass over the slot table).  A jump ends inside its
// cell and its positions' binades; its last position is converted as a step's is and must
// lie in the cell, and as positions are monotonic per axis, all between do.  The conversion
// to FP32 rounds the pattern in integer arithmetic.  Every position, density and hit is the
// one that stepping gives, bit for bit.  1280x720 of a 48-cluster crop of the 4096^3 FP16
// layout: 60.3 ms stepping, 1.81 ms so.  Bound now: issue and instruction fetch (34% of
// issue slots, 24 of 32 lanes active), the rays of a warp parting at cell faces.
#include <type_traits>

#include "interp_common.cuh"

namespace msbg {

namespace {

struct RV {
  double x, y, z;
};

__device__ __forceinline__ RV rsub(RV a, RV b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
// a.x*b.x + a.y*b.y + a.z*b.z, fused left to right
__device__ __forceinline__ double rdot(RV a, RV b) {
  return __fma_rn(a.z, b.z, __fma_rn(a.y, b.y, __dmul_rn(a.x, b.x)));
}
__device__ __forceinline__ RV rnormalize(RV v) {
  const double len = __dsqrt_rn(rdot(v, v));
  if (!(len > (double)1e-20f)) return {0.0, 1.0, 0.0};
  return {__ddiv_rn(v.x, len), __ddiv_rn(v.y, len), __ddiv_rn(v.z, len)};
}
// a.y*b.z - a.z*b.y, ... fused as fma(a.y, b.z, -(a.z*b.y))
__device__ __forceinline__ RV rcross(RV a, RV b) {
  return {__fma_rn(a.y, b.z, -__dmul_rn(a.z, b.y)), __fma_rn(a.z, b.x, -__dmul_rn(a.x, b.z)),
          __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x))};
}

// Empty space: byte maps of the aligned 4^3 and 16^3 groups of blocks that hold a value block.
struct Occupancy {
  const uint8_t *g4, *g16;
  int n4x, n4y, n16x, n16y;
};

__global__ void kOccupancy(const int32_t *__restrict__ slot, int nbx, int nby, int nbz, int n4x, int n4y, int n4z,
                           int n16x, int n16y, uint8_t *__restrict__ g4, uint8_t *__restrict__ g16) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4x * n4y * n4z) return;
  const int x = i % n4x, y = (i / n4x) % n4y, z = i / (n4x * n4y);
  bool any = false;
  for (int bz = 4 * z; bz < min(4 * z + 4, nbz); bz++)
    for (int by = 4 * y; by < min(4 * y + 4, nby); by++)
      for (int bx = 4 * x; bx < min(4 * x + 4, nbx); bx++)
        any |= __ldg(slot + ((int64_t)bz * nby + by) * nbx + bx) >= 0;
  g4[i] = any;
  if (any) g16[((z >> 2) * n16y + (y >> 2)) * n16x + (x >> 2)] = 1;  // zeroed before; every writer writes 1
}

// One axis of a ray: the position's bit pattern, and the pattern's change per step while
// the position stays in its binade.
struct Axis {
  long long b;  // bits of the FP64 position
  long long j;  // change per step, when fast
  bool fast;
};
constexpr long long kMant = (1ll << 52) - 1;

// j = inc / ulp(p) rounded to nearest; not fast for p <= 0, subnormal or not finite, and for
// an increment not below the binade.  A tie (one ray in 2^shift: shift is 8 to 12 for most
// of a ray) rounds to the even sum, so from an even pattern j is the even neighbour, and
// the pattern stays even; an odd pattern takes one general step, which makes it even.
__device__ __forceinline__ void axisDerive(Axis &a, double inc) {
  const long long ib = __double_as_longlong(inc);
  const int e = (int)(a.b >> 52), ei = (int)((ib >> 52) & 0x7ff);
  a.fast = false;
  a.j = 0;
  if (a.b <= 0 || e == 0 || e >= 0x7ff) return;
  if ((ib & 0x7fffffffffffffffll) == 0) { a.fast = true; return; }
  const int shift = e - ei;
  if (ei == 0 || shift < 1) return;
  if (shift > 54) { a.fast = true; return; }  // less than half a unit
  const unsigned long long m = (unsigned long long)((ib & kMant) | (1ll << 52)), half = 1ull << (shift - 1);
  const unsigned long long rem = m & (2 * half - 1);
  long long q = (long long)(m >> shift) + (rem > half);
  if (rem == half) {
    if (a.b & 1) return;
    q += q & 1;
  }
  a.j = ib < 0 ? -q : q;
  a.fast = true;
}
// The pattern after n steps (n j does not overflow: a valid result differs by less than
// 2^52); false when the position leaves the binade.  Moving down, the binade's lowest value
// is left to the general way: the exact sum may lie below it, where the units are finer.
__device__ __forceinline__ bool axisAhead(const Axis &a, bool down, long long n, long long &nb) {
  nb = a.b + n * a.j;
  return a.fast && ((nb ^ a.b) >> 52) == 0 && !(down && (nb & kMant) == 0);
}
// FEW: the rounded sum itself; j is then derived before a jump.
template <bool FEW>
__device__ __forceinline__ void axisStep(Axis &a, bool down, double inc) {
  long long nb;
  if (FEW) {
    a.b = __double_as_longlong(__dadd_rn(__longlong_as_double(a.b), inc));
  } else if (axisAhead(a, down, 1, nb)) {
    a.b = nb;
  } else {
    a.b = __double_as_longlong(__dadd_rn(__longlong_as_double(a.b), inc));
    axisDerive(a, inc);
  }
}
// __double2float_rn of a position's pattern
template <bool FEW>
__device__ __forceinline__ float patternToFloat(long long b) {
  const int e = (int)((b >> 52) & 0x7ff);
  if (FEW || b < 0 || e <= 1023 - 126 || e >= 1023 + 126) return __double2float_rn(__longlong_as_double(b));
  const unsigned long long f = (unsigned long long)(b - ((1023ll - 127) << 52));
  return __uint_as_float((uint32_t)((f + 0x0fffffffull + ((f >> 29) & 1)) >> 29));
}

struct RenderArgs {
  IpGeom g;
  Occupancy occ;
  const int32_t *slot;
  const void *payload;
  int width, height, maxSteps;
  float res;
  double hstep, invW, invH, aspect, zoom;
  RV camPos, lookAt, sun, color;
  float domMin[3], domMax[3];
  uint8_t *out;
};

// MtCubicBSplineWeights1D (src/mtool.h:344-362), each operation rounded in source order
__device__ __forceinline__ void bspline3(float t, float w[4], float d[4]) {
  const float s = __fsub_rn(1.0f, t), c6 = 1.0f / 6.0f, c23 = 2.0f / 3.0f;
  w[0] = __fmul_rn(__fmul_rn(__fmul_rn(c6, s), s), s);
  w[1] = __fsub_rn(c23, __fmul_rn(__fmul_rn(__fmul_rn(0.5f, t), t), __fsub_rn(2.0f, t)));
  w[2] = __fsub_rn(c23, __fmul_rn(__fmul_rn(__fmul_rn(0.5f, s), s), __fadd_rn(1.0f, t)));
  w[3] = __fmul_rn(__fmul_rn(__fmul_rn(c6, t), t), t);
  d[0] = __fdiv_rn(__fmul_rn(-s, s), 2.0f);
  d[1] = __fsub_rn(__fmul_rn(__fmul_rn(0.5f, t), t), __fmul_rn(__fmul_rn(1.0f, __fsub_rn(2.0f, t)), t));
  d[2] = __fsub_rn(__fmul_rn(__fmul_rn(1.0f, s), __fadd_rn(t, 1.0f)), __fmul_rn(__fmul_rn(0.5f, s), s));
  d[3] = __fdiv_rn(__fmul_rn(t, t), 2.0f);
}

enum { kOutside, kEmpty, kValue };  // what a position lies in
template <typename T>
__device__ __forceinline__ float density(const RenderArgs &a, const float q[3], int ip[3], int &where) {
  const int s[3] = {a.g.sx, a.g.sy, a.g.sz};
  where = kOutside;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    ip[k] = (int)floorf(q[k]);
    if (ip[k] < 0 || ip[k] > s[k] - 1) return 0.0f;
  }
  const int L = a.g.log2bs;
  const int64_t bid = (int64_t)(ip[0] >> L) + (int64_t)(ip[1] >> L) * a.g.nbx + (int64_t)(ip[2] >> L) * a.g.nxy;
  where = kEmpty;
  if (__ldg(a.slot + bid) < 0) return 0.0f;  // skip fast over empty blocks
  where = kValue;
  return ipValue<T>(a.g, a.slot, (const T *)a.payload, q[0], q[1], q[2]);
}

template <typename T>
__device__ RV gradient(const RenderArgs &a, RV p) {
  const float q[3] = {__fmul_rn(a.res, __double2float_rn(p.x)), __fmul_rn(a.res, __double2float_rn(p.y)),
                      __fmul_rn(a.res, __double2float_rn(p.z))};
#pragma unroll
  for (int k = 0; k < 3; k++)
    if (q[k] < a.domMin[k] || q[k] > a.domMax[k]) return {-0.0, -0.0, -0.0};
  const int s[3] = {a.g.sx, a.g.sy, a.g.sz};
  float w[3][4], d[3][4];
  int i0[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float pos = __fsub_rn(q[k], 0.5f), pf = floorf(pos);
    i0[k] = (int)pf - 1;
    bspline3(__fsub_rn(pos, pf), w[k], d[k]);
  }
  const T *pay = (const T *)a.payload;
  float gx = 0.0f, gy = 0.0f, gz = 0.0f;
  for (int dz = 0; dz < 4; dz++) {
    const int z = min(max(i0[2] + dz, 0), s[2] - 1);
    for (int dy = 0; dy < 4; dy++) {
      const int y = min(max(i0[1] + dy, 0), s[1] - 1);
      const float wyz = __fmul_rn(w[2][dz], w[1][dy]);
      const float wgy = __fmul_rn(w[2][dz], d[1][dy]);
      const float wgz = __fmul_rn(d[2][dz], w[1][dy]);
#pragma unroll
      for (int dx = 0; dx < 4; dx++) {
        const int x = min(max(i0[0] + dx, 0), s[0] - 1);
        const float f = voxel(a.g, a.slot, pay, x, y, z);
        gx = __fmaf_rn(__fmul_rn(wyz, d[0][dx]), f, gx);
        gy = __fmaf_rn(__fmul_rn(wgy, w[0][dx]), f, gy);
        gz = __fmaf_rn(__fmul_rn(wgz, w[0][dx]), f, gz);
      }
    }
  }
  if (a.g.renderDens) {
    gx = __fmul_rn(gx, kU16ToF);
    gy = __fmul_rn(gy, kU16ToF);
    gz = __fmul_rn(gz, kU16ToF);
  }
  return {-(double)gx, -(double)gy, -(double)gz};
}

// FEW: pictures whose CTAs all fit the chip at four an SM.  Their rays are as long as the steps'
// latency, not as the FP64 pipe or issue take, and an FP64 sum is shorter than the integer step
// (and its spills at 80 registers): full layouts of 16^3 blocks that no ray hits, 48x27 563 us
// with integer steps, 469 so, 434 before the integer steps; 320x180 511 / 442 / 479; 480x270
// (1020 CTAs) 679 / 678 / 750; 1280x720 2782 / 3207 / 4197.
constexpr unsigned kFewCtas = 152 * 4;
template <typename T, bool FEW>
__global__ void __launch_bounds__(128, FEW ? 4 : 6) kRender(RenderArgs a) {
  // a warp takes 8x4 pixels, whose rays stay together longer than a 16x2 row pair's
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7), y = blockIdx.y * 8 + (warp >> 1) * 4 + (lane >> 3);
  if (x >= a.width || y >= a.height) return;
  const RV fwd = rnormalize(rsub(a.lookAt, a.camPos));
  const RV right = rnormalize(rcross(fwd, RV{0.0, 1.0, 0.0}));
  const RV up = rcross(right, fwd);
  const double ndcX = __dmul_rn(__dmul_rn(__fma_rn((double)__fadd_rn((float)x, 0.5f), a.invW, -0.5), 2.0), a.aspect);
  const double ndcY = __dmul_rn(__fma_rn(-(double)__fadd_rn((float)y, 0.5f), a.invH, 0.5), 2.0);
  const RV dir = rnormalize({__fma_rn(up.x, ndcY, __fma_rn(right.x, ndcX, __dmul_rn(fwd.x, a.zoom))),
                             __fma_rn(up.y, ndcY, __fma_rn(right.y, ndcX, __dmul_rn(fwd.y, a.zoom))),
                             __fma_rn(up.z, ndcY, __fma_rn(right.z, ndcX, __dmul_rn(fwd.z, a.zoom)))});
  const RV inc = {__dmul_rn(dir.x, a.hstep), __dmul_rn(dir.y, a.hstep), __dmul_rn(dir.z, a.hstep)};
  const int s[3] = {a.g.sx, a.g.sy, a.g.sz};
  const double incv[3] = {inc.x, inc.y, inc.z};
  Axis ax[3];
  const double start[3] = {a.camPos.x, a.camPos.y, a.camPos.z};
  float q[3], dirV[3], invDir[3];  // voxels; voxels per step and its reciprocal (estimates only)
  bool down[3], zero[3];  // the increment's sign, from its bits, so that no step compares FP64 values
#pragma unroll
  for (int k = 0; k < 3; k++) {
    ax[k].b = __double_as_longlong(start[k]);
    zero[k] = (__double_as_longlong(incv[k]) << 1) == 0;
    down[k] = __double2hiint(incv[k]) < 0 && !zero[k];
    if (!FEW) axisDerive(ax[k], incv[k]);
    q[k] = __fmul_rn(a.res, __double2float_rn(start[k]));
    dirV[k] = a.res * (float)incv[k];
    invDir[k] = dirV[k] != 0.0f ? 1.0f / dirV[k] : 0.0f;
  }
  auto at = [&]() -> RV {
    return {__longlong_as_double(ax[0].b), __longlong_as_double(ax[1].b), __longlong_as_double(ax[2].b)};
  };
  RV prevPos = a.camPos, hitPos = a.camPos;
  int ip[3], where;
  float prev = density<T>(a, q, ip, where);
  bool hit = false;
  for (int step = 0; step < a.maxSteps; step++) {
    if (where == kEmpty) {
      // jump within the largest empty cell around the position
      const int L = a.g.log2bs;
      const int b4x = ip[0] >> (L + 2), b4y = ip[1] >> (L + 2), b4z = ip[2] >> (L + 2);
      int lc = L;
      if (!a.occ.g4[(b4z * a.occ.n4y + b4y) * a.occ.n4x + b4x])
        lc = a.occ.g16[((b4z >> 2) * a.occ.n16y + (b4y >> 2)) * a.occ.n16x + (b4x >> 2)] ? L + 2 : L + 4;
      float n = (float)(a.maxSteps - step);
      int lo[3], hi[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        lo[k] = (ip[k] >> lc) << lc;
        hi[k] = min(lo[k] + (1 << lc), s[k]);
        // to the cell's face, or to the end of the position's binade
        const int e = (int)((ax[k].b >> 52) & 0x7ff) - (1023 - 127);
        const float bin = e > 0 && e < 254 ? a.res * __uint_as_float((uint32_t)e << 23) : 0.0f;
        const float face = dirV[k] > 0.0f ? fminf((float)hi[k], 2.0f * bin) : fmaxf((float)lo[k], bin);
        if (dirV[k] != 0.0f) n = fminf(n, (face - q[k]) * invDir[k]);
      }
      const int steps = (int)fmaxf(n, 0.0f) - 1;
      if (steps >= 3) {
        long long nb[3];
        bool in = true;
        float q2[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
          if (FEW) axisDerive(ax[k], incv[k]);
          in = axisAhead(ax[k], down[k], steps, nb[k]) && in;
          q2[k] = __fmul_rn(a.res, patternToFloat<FEW>(nb[k]));
          const float f = floorf(q2[k]);
          in = in && f >= (float)lo[k] && f < (float)hi[k];
        }
        if (in) {
#pragma unroll
          for (int k = 0; k < 3; k++) { ax[k].b = nb[k]; q[k] = q2[k]; }
          step += steps;
          prev = 0.0f;
          prevPos = at();
          if (step >= a.maxSteps) break;
        }
      }
    }
    // Inside a value block the next kAhead steps are evaluated together, so that their
    // gathers overlap; they are then looked at in order, as single steps are.  Two: one
    // takes 2.00 ms, four 2.58 (instruction fetch), on the view named at the top.  FEW: one, as
    // two lengthen the step (48x27 as above 1.30x against 1.16x with integer steps).
    constexpr int kAhead = FEW ? 1 : 2;
    const int nAhead = where == kValue ? kAhead : 1;
    Axis at1[3] = {ax[0], ax[1], ax[2]};
    long long pb[kAhead][3];
    float dens[kAhead];
    bool gone[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; i++) {
      dens[i] = 0.0f;
      gone[i] = false;
      if (i >= nAhead) continue;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        axisStep<FEW>(at1[k], down[k], incv[k]);
        pb[i][k] = at1[k].b;
        q[k] = __fmul_rn(a.res, patternToFloat<FEW>(at1[k].b));
        const float f = floorf(q[k]);
        gone[i] |= (f < 0.0f && (down[k] || zero[k])) || (f > (float)(s[k] - 1) && !down[k]);
      }
      dens[i] = density<T>(a, q, ip, where);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) ax[k] = at1[k];
    bool stop = false;
#pragma unroll
    for (int i = 0; i < kAhead; i++) {
      if (i >= nAhead || stop) continue;
      if (i > 0 && ++step >= a.maxSteps) { stop = true; continue; }
      if (gone[i]) { stop = true; continue; }  // outside and moving away: the density stays 0
      const RV pos = {__longlong_as_double(pb[i][0]), __longlong_as_double(pb[i][1]), __longlong_as_double(pb[i][2])};
      if (prev < 0.5f && dens[i] >= 0.5f) {
        const double t = __ddiv_rn(__dsub_rn(0.5, (double)prev), __dsub_rn((double)dens[i], (double)prev));
        hitPos = {__fma_rn(__dsub_rn(pos.x, prevPos.x), t, prevPos.x),
                  __fma_rn(__dsub_rn(pos.y, prevPos.y), t, prevPos.y),
                  __fma_rn(__dsub_rn(pos.z, prevPos.z), t, prevPos.z)};
        hit = stop = true;
        continue;
      }
      prev = dens[i];
      prevPos = pos;
    }
    if (stop) break;
  }
  uint8_t rgb[3] = {0, 0, 0};
  if (hit) {
    const RV nrm = rnormalize(gradient<T>(a, hitPos));
    const RV ld = rnormalize(rsub(a.sun, hitPos));
    double diff = rdot(nrm, ld);
    diff = diff > 0.0 ? diff : 0.0;
    const double col[3] = {a.color.x, a.color.y, a.color.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double v = __dmul_rn(col[k], diff);
      v = v < 0.0 ? 0.0 : v > 1.0 ? 1.0 : v;
      rgb[k] = (uint8_t)(int)__fma_rn(v, 255.0, 0.5);
    }
  }
  uint8_t *o = a.out + ((int64_t)y * a.width + x) * 3;
  o[0] = rgb[0];
  o[1] = rgb[1];
  o[2] = rgb[2];
}

}  // namespace

}  // namespace msbg

using namespace msbg;

extern "C" int msbg_gpu_render(msbg_gpu_ctx *ctx, int chan, int width, int height, const msbg_gpu_camera *cam,
                               uint8_t *dRGB) {
  if (!ctx) return MSBG_GPU_ERR_ARG;
  if (width <= 0 || height <= 0 || height > 65535 * 8 || (int64_t)width * height > ((int64_t)1 << 31) || !cam ||
      !dRGB)
    return fail(ctx, MSBG_GPU_ERR_ARG, "render: bad image size or null argument");
  if (chan < 0 || chan >= kMaxChannels || !ctx->ch[chan].exists)
    return fail(ctx, MSBG_GPU_ERR_ARG, "channel %d does not exist", chan);
  if (!ctx->layoutValid) return fail(ctx, MSBG_GPU_ERR_STATE, "no block layout: call set_refinement_map");
  const Channel &c = ctx->ch[chan];
  RenderArgs a;
  a.g.sx = ctx->sx; a.g.sy = ctx->sy; a.g.sz = ctx->sz;
  a.g.log2bs = ctx->log2bs;
  a.g.nbx = ctx->nbx;
  a.g.nxy = (int64_t)ctx->nbx * ctx->nby;
  a.g.vpb = ctx->voxPerBlock;
  a.g.po = 0.5f;
  a.g.dirichlet = a.g.dirichletOld = 0;
  a.g.renderDens = c.storage == MSBG_GPU_U16;
  a.slot = ctx->dSlot;
  a.payload = c.d;
  a.width = width;
  a.height = height;
  const int res = ctx->sx > ctx->sy ? (ctx->sx > ctx->sz ? ctx->sx : ctx->sz) : (ctx->sy > ctx->sz ? ctx->sy : ctx->sz);
  a.res = (float)res;
  a.hstep = 1.0 / (double)res;
  a.maxSteps = (int)(2.0 / a.hstep);
  a.invW = 1.0 / (double)width;
  a.invH = 1.0 / (double)height;
  a.aspect = (double)width / (double)height;
  a.zoom = cam->zoom;
  a.camPos = {cam->pos[0], cam->pos[1], cam->pos[2]};
  a.lookAt = {cam->lookAt[0], cam->lookAt[1], cam->lookAt[2]};
  a.sun = {cam->sun[0], cam->sun[1], cam->sun[2]};
  a.color = {cam->color[0], cam->color[1], cam->color[2]};
  for (int k = 0; k < 3; k++) {
    a.domMin[k] = ctx->domMin[k];
    a.domMax[k] = ctx->domMax[k];
  }
  a.out = dRGB;
  // occupancy maps: n4 bytes of 4^3 groups, then the 16^3 groups
  const int n4x = (ctx->nbx + 3) / 4, n4y = (ctx->nby + 3) / 4, n4z = (ctx->nbz + 3) / 4;
  const int n16x = (n4x + 3) / 4, n16y = (n4y + 3) / 4, n16z = (n4z + 3) / 4;
  const int64_t n4 = (int64_t)n4x * n4y * n4z;
  uint8_t *g16 = ctx->dOccupancy + n4;
  MSBG_CUDA(ctx, cudaMemsetAsync(g16, 0, (size_t)n16x * n16y * n16z, ctx->stream));
  MSBG_LAUNCH(ctx, kOccupancy, gridFor(n4, 256), 256, 0, ctx->dSlot, ctx->nbx, ctx->nby, ctx->nbz, n4x, n4y, n4z, n16x,
              n16y, ctx->dOccupancy, g16);
  a.occ = {ctx->dOccupancy, g16, n4x, n4y, n16x, n16y};
  const dim3 grid((unsigned)((width + 15) / 16), (unsigned)((height + 7) / 8));
  auto launch = [&](auto few) -> int {
    constexpr bool FEW = decltype(few)::value;
    switch (c.storage) {
      case MSBG_GPU_F32: MSBG_LAUNCH(ctx, (kRender<float, FEW>), grid, 128, 0, a); break;
      case MSBG_GPU_F16: MSBG_LAUNCH(ctx, (kRender<__half, FEW>), grid, 128, 0, a); break;
      case MSBG_GPU_U16: MSBG_LAUNCH(ctx, (kRender<uint16_t, FEW>), grid, 128, 0, a); break;
      default: return fail(ctx, MSBG_GPU_ERR_UNSUPPORTED, "render: FP64 channels are not supported");
    }
    return MSBG_GPU_OK;
  };
  return (int64_t)grid.x * grid.y <= kFewCtas ? launch(std::true_type{}) : launch(std::false_type{});
}
