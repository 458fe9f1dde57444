// GPU fill pipeline: pixie's commandsToShapes (cubic/quadratic flattening),
// shapesToSegments, computeBounds/snapToPixels, partitionSegments and the
// fillShapes row loop (src/pixie/paths.nim:654-1912), restated for sm_103a.
//
// k_setup       a cluster of 1 to 8 CTAs per fill job (setup.cuh): flatten the
//               primitives, emit pixie's segments (quantised, oriented,
//               horizontals dropped) in the reference's order, reduce the bounds,
//               derive the partition geometry, each band's count, flag and list of
//               segments.
// k_rows_fast   the row engine (rowfast.cuh): a warp takes chunks of rows from a
//               queue; a row's band entries are clipped as partitionSegments does,
//               then the reference's per-row decision (the non-AA two-edge fill, the
//               trapezoid fast path, or 5-sample coverage with the nonzero/even-odd
//               walk) and the fused coverage -> paint -> blend write.
// k_rows_lines  the same with a CTA per row and a warp per sample line, for few
//               rows of many crossings; k_rows_huge for rows of more than 256.
// k_rows        the general row code (process_row), one row a warp: MaskBlend and
//               images too wide for the row engine's keys; k_rows_wide takes the
//               rows that the other kernels hand on.
// k_scene_rec, k_scene_big, k_scene_huge, k_scene_rest, k_scene  many paths on one
//               canvas: rows recorded by the same code, then drawn in path order.
// Float math is compiled with -fmad=false: every expression keeps the
// reference's float32 operation order.
#include <algorithm>
#include <cfloat>
#include <climits>

#include "pxg_device.cuh"
#include "raster.cuh"

namespace pxg {

static __device__ constexpr float kEps = (float)(0.0001 * 3.141592653589793);  // paths.nim:44
static constexpr long long kIterCap = 1LL << 24;
static constexpr int kBandWindow = 1024;  // bands the setup kernel counts and lists at a time

struct V2 {
  float x, y;
};
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return V2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return V2{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ V2 operator*(V2 a, float s) { return V2{a.x * s, a.y * s}; }
__device__ __forceinline__ V2 operator/(V2 a, float s) { return V2{a.x / s, a.y / s}; }
__device__ __forceinline__ float lengthSq(V2 v) { return v.x * v.x + v.y * v.y; }
__device__ __forceinline__ float length(V2 v) { return sqrtf(lengthSq(v)); }

// ---------------------------------------------------------------------------
// Flattening  paths.nim:677-762
// ---------------------------------------------------------------------------
__device__ __forceinline__ V2 cubicAt(V2 a, V2 c1, V2 c2, V2 to, float t) {
  float t2 = t * t, t3 = t2 * t;
  return a * (((-t3 + 3 * t2) - 3 * t) + 1) + c1 * ((3 * t3 - 6 * t2) + 3 * t) +
         c2 * (-3 * t3 + 3 * t2) + to * (t3);
}
__device__ __forceinline__ V2 cubicDeriv(V2 a, V2 c1, V2 c2, V2 to, float t) {
  float t2 = t * t;
  return a * ((-3 * t2 + 6 * t) - 3) + c1 * ((9 * t2 - 12 * t) + 3) + c2 * (-9 * t2 + 6 * t) +
         to * (3 * t2);
}
__device__ __forceinline__ V2 quadAt(V2 a, V2 c, V2 to, float t) {
  float t2 = t * t;
  return a * ((t2 - 2 * t) + 1) + c * (-2 * t2 + 2 * t) + to * t2;
}

__device__ __forceinline__ float pow2neg(int k) {  // 2^-k for 0 <= k < 126
  return __int_as_float((127 - k) << 23);
}

// transform + shapesToSegments for one emitted pair (paths.nim:1059-1096).
// vmath quantize(v, 1/256) = sign(v) * floor(|v| / n) * n.
__device__ __forceinline__ float quantize256(float v) {
  const float n = 1.0f / 256;
  float sgn = v >= 0 ? 1.0f : -1.0f;
  return sgn * (floorf(fabsf(v) / n) * n);
}
struct SegMat {  // the job's transform: (x, y) -> (mx . (x, y, 1), my . (x, y, 1))
  float mx[3], my[3];
  int identity;
};
__device__ __forceinline__ bool make_seg(const SegMat& M, V2 a, V2 b, float4& s, int& w) {
  if (!M.identity) {
    a = V2{M.mx[0] * a.x + M.mx[1] * a.y + M.mx[2], M.my[0] * a.x + M.my[1] * a.y + M.my[2]};
    b = V2{M.mx[0] * b.x + M.mx[1] * b.y + M.mx[2], M.my[0] * b.x + M.my[1] * b.y + M.my[2]};
  }
  a.y = quantize256(a.y);
  b.y = quantize256(b.y);
  if (a.y == b.y) return false;
  w = 1;
  if (a.y > b.y) {
    V2 t = a;
    a = b;
    b = t;
    w = -1;
  }
  s = make_float4(a.x, a.y, b.x, b.y);
  return true;
}

// ---------------------------------------------------------------------------
// Partitions  paths.nim:1127-1262
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool hasFractional(float v) { return v - truncf(v) != 0; }
__device__ __forceinline__ bool segRequiresAA(float4 s) {  // :1149-1160
  return s.x != s.z || hasFractional(s.x) || hasFractional(s.y) || hasFractional(s.w);
}
// bumpy intersects(Segment, Line): the parametric form of internal.nim:36-48
// without the range check on the line parameter; the point is on the segment.
__device__ __forceinline__ bool intersectSegLine(V2 sa, V2 sb, V2 l0, V2 l1, V2& at) {
  V2 s1 = sb - sa, s2 = l1 - l0;
  float den = (-s2.x * s1.y + s1.x * s2.y);
  float t = (s2.x * (sa.y - l0.y) - s2.y * (sa.x - l0.x)) / den;
  if (t >= 0 && t <= 1) {
    at = sa + s1 * t;
    return true;
  }
  return false;
}
__device__ __forceinline__ bool intersectsInside(V2 aa, V2 ab, V2 ba, V2 bb) {  // internal.nim:36-48
  V2 s1 = ab - aa, s2 = bb - ba;
  float den = (-s2.x * s1.y + s1.x * s2.y);
  float s = (-s1.y * (aa.x - ba.x) + s1.x * (aa.y - ba.y)) / den;
  float t = (s2.x * (aa.y - ba.y) - s2.y * (aa.x - ba.x)) / den;
  return s > 0 && s < 1 && t > 0 && t < 1;
}
__device__ __forceinline__ Entry make_entry(float4 s, int w, float top, float bottom) {
  Entry e;
  e.w = w;
  e.pad = 0;
  e.m = 0;
  e.b = 0;
  float d = s.x - s.z;  // initPartitionEntry :1127-1135
  if (d == 0) {
    e.b = s.x;
  } else {
    e.m = (s.y - s.w) / d;
    e.b = s.y - e.m * s.x;
  }
  V2 a{s.x, s.y}, b{s.z, s.w};
  if (a.y <= top && b.y >= bottom) {  // clip :1236-1248
    V2 at{0, 0};
    intersectSegLine(a, b, V2{0, top}, V2{1000, top}, at);
    a = at;
    intersectSegLine(a, b, V2{0, bottom}, V2{1000, bottom}, at);
    b = at;
  }
  e.ax = a.x;
  e.ay = a.y;
  e.bx = b.x;
  e.by = b.y;
  return e;
}

// ---------------------------------------------------------------------------
// k_rows: the per-row loop of fillShapes (:1631-1908), one warp per row
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool shouldFill(int rule, long long count) {  // :1288-1296
  return rule == 0 ? count != 0 : (count % 2 != 0);
}
// The generic blender, kept out of line: the row code calls it from several
// places, and one copy keeps the kernels small enough for the instruction
// cache.  NormalBlend stays inline at every call site.
static __device__ __noinline__ uint32_t blend_any(int mode, const uint8_t* tbl, uint32_t b, uint32_t s) {
  return blend_px(mode, tbl, b, s);
}
__device__ __forceinline__ uint32_t blend_row(int mode, const uint8_t* tbl, uint32_t b, uint32_t s) {
  return mode == kNormal ? blendNormal(b, s) : blend_any(mode, tbl, b, s);
}
// FILL: a fillHits span (:1540-1591)
__device__ __forceinline__ uint32_t op_fill(int mode, const uint8_t* tbl, uint32_t b, uint32_t c) {
  switch (mode) {
    case kOverwrite: return c;
    case kNormal: return (c >> 24) == 255 ? c : blendNormal(b, c);
    case kMask: return (c >> 24) != 255 ? blendMaskPx(b, c) : b;
    default: return blend_any(mode, tbl, b, c);
  }
}
// COV: fillCoverage with coverage k (:1442-1526)
__device__ __forceinline__ uint32_t op_cov(int mode, const uint8_t* tbl, uint32_t b, uint32_t c, uint32_t k) {
  if (mode == kMask) return k != 255 ? blendMaskPx(b, mul_c(c, k)) : b;
  if (k == 0) return b;
  if (mode == kOverwrite) return mul_c(c, k);
  if (mode == kNormal) return blendNormal(b, mul_c(c, k));
  return blend_any(mode, tbl, b, mul_c(c, k));
}

template <int MAXH, int XT>
struct RowScratch {
  static constexpr int SPCAP = 5 * (MAXH / 2 + 2);
  Entry ent[MAXH];  // the band's entries overlapping the row, in segment order
  int idx[MAXH];
  int a0[MAXH], a1[MAXH], a2[MAXH], a3[MAXH], a4[MAXH], a5[MAXH];
  int2 sp[SPCAP];
  int acc[XT + 1];
  int nsp, flag;
};

// Stable rank of element i among n keys (ties keep the original order).
__device__ __forceinline__ int stable_rank_i(const int* keys, int n, int i) {
  int ki = keys[i], r = 0;
  for (int j = 0; j < n; j++) {
    int kj = keys[j];
    r += (kj < ki) || (kj == ki && j < i);
  }
  return r;
}
__device__ __forceinline__ int stable_rank_f(const float* keys, int n, int i) {
  float ki = keys[i];
  int r = 0;
#pragma unroll 2
  for (int j = 0; j < n; j++) {
    float kj = keys[j];
    r += (kj < ki) || (kj == ki && j < i);
  }
  return r;
}

// One row of the destination: premultiplied RGBX (4 bytes per pixel), or an
// 8-bit alpha mask (A8) read as (a, a, a, a) and written as the alpha byte.
// A mask render paints a white opaque colour with NormalBlend onto a
// transparent mask, so every pixel keeps four equal channels and the alpha
// byte holds the whole RGBX value.
template <bool A8>
struct PxRef {
  unsigned char* p;
  __device__ __forceinline__ operator uint32_t() const {
    if (A8) return (uint32_t)*p * 0x01010101u;
    return *reinterpret_cast<const uint32_t*>(p);
  }
  __device__ __forceinline__ const PxRef& operator=(uint32_t v) const {
    if (A8) *p = (unsigned char)(v >> 24);
    else *reinterpret_cast<uint32_t*>(p) = v;
    return *this;
  }
};
// base holds pixel x0 (0 for a whole image row; a row slice staged in shared
// memory starts at its first pixel).
template <bool A8>
struct RowPx {
  unsigned char* base;
  long long x0;
  __device__ __forceinline__ PxRef<A8> operator[](long long x) const {
    return PxRef<A8>{base + (x - x0) * (A8 ? 1 : 4)};
  }
};
template <bool A8>
__device__ __forceinline__ RowPx<A8> row_of(const PathJob& J, long long y) {
  return RowPx<A8>{J.img + y * J.W * (A8 ? 1 : 4), 0};
}

// Linear-index clear of [y*W + a, y*W + b) (clearUnsafe :1433-1440 with
// startY == toY).  Pixels before row y are recorded for the cross-row pass.
template <bool A8>
__device__ void clear_span_linear(const PathJob& J, const Arena& A, int job, RowPx<A8> row,
                                  long long y, long long a, long long b, int lane, long long xa,
                                  long long xb) {
  if (a == J.W) return;
  if (b <= a) return;
  for (long long x = max(max(a, 0LL), xa) + lane; x < min(b, xb); x += 32) row[x] = 0u;
  if (a < 0 && lane == 0 && xa == 0) {
    long long lo = y * J.W + a, hi = y * J.W + min(b, 0LL);
    if (lo < 0) lo = 0;
    if (hi > lo) {
      unsigned long long slot = atomicAdd(&A.counters[kCtrXClears], 1ull);
      if ((long long)slot < A.xclear_cap) {
        A.xclears[3 * slot] = job;
        A.xclears[3 * slot + 1] = lo;
        A.xclears[3 * slot + 2] = hi;
      }
    }
  }
}

// The covered area of pixel x in the left sliver of a trapezoid pair: the edge
// (m, b) crosses the row's top and bottom at t0 and t1; xs is the sliver's
// first pixel (:1752-1788).
__device__ __forceinline__ float trap_left_area(float m, float b, float t0, float t1, long long x, long long xs,
                                                long long y) {
  const bool inv = t0 < t1;
  const float sliverStart = nmin(t0, t1), rectStart = nmax(t0, t1);
  float prevPen = x == xs ? sliverStart : (float)x;
  float pen = (float)(x + 1);
  float rightRectArea = 0;
  if (pen > rectStart) {
    rightRectArea = pen - rectStart;
    pen = rectStart;
  }
  float prevPenY = x == xs ? (inv ? (float)y : (float)(y + 1)) : m * (float)x + b;
  float penY = m * pen + b;
  float run = pen - prevPen;
  float tri = 0.5f * run * fabsf(penY - prevPenY);
  float rect = inv ? (prevPenY - (float)y) * run : ((float)(y + 1) - prevPenY) * run;
  return tri + rect + rightRectArea;
}
// ... and in the right sliver (:1790-1828)
__device__ __forceinline__ float trap_right_area(float m, float b, float t0, float t1, long long x, long long xs,
                                                 long long y) {
  const bool inv = t0 > t1;
  const float rectEnd = nmin(t0, t1), sliverEnd = nmax(t0, t1);
  float prevPen = x == xs ? rectEnd : (float)x;
  float pen = (float)(x + 1);
  float ap = fabsf(prevPen);
  float leftRectArea = ap - floorf(ap);  // vmath fractional: fractional part of |v|
  if (pen > sliverEnd) pen = sliverEnd;
  float prevPenY = x == xs ? (inv ? (float)(y + 1) : (float)y) : m * (float)x + b;
  float penY = m * pen + b;
  float run = pen - prevPen;
  float tri = 0.5f * run * fabsf(penY - prevPenY);
  float rect = inv ? (penY - (float)y) * run : ((float)(y + 1) - penY) * run;
  return leftRectArea + tri + rect;
}

// The pixels [x0, x1) of a row filled (op_fill), 16-byte quads between the
// ragged ends of an RGBX row.
template <bool A8>
__device__ __forceinline__ void fill_span(RowPx<A8> row, int mode, const uint8_t* tbl, uint32_t rgbx, long long x0,
                                          long long x1, int lane, unsigned* cnt = nullptr) {
  if (!A8 && x1 - x0 >= 64) {
    uint32_t* p = reinterpret_cast<uint32_t*>(row.base) + (x0 - row.x0);
    const long long n = x1 - x0;
    const int head = (int)((4 - ((reinterpret_cast<uintptr_t>(p) >> 2) & 3)) & 3);
    const long long nq = (n - head) >> 2;
    const int tail = (int)(n - head - 4 * nq);
    if (lane < head) p[lane] = op_fill(mode, tbl, p[lane], rgbx);
    if (lane < tail) p[n - tail + lane] = op_fill(mode, tbl, p[n - tail + lane], rgbx);
    uint4* q = reinterpret_cast<uint4*>(p + head);
    if (mode == kOverwrite || (mode == kNormal && (rgbx >> 24) == 255)) {
      for (long long i = lane; i < nq; i += 32) q[i] = make_uint4(rgbx, rgbx, rgbx, rgbx);
    } else {
      for (long long i = lane; i < nq; i += 32) {
        uint4 v = q[i];
        v.x = op_fill(mode, tbl, v.x, rgbx);
        v.y = op_fill(mode, tbl, v.y, rgbx);
        v.z = op_fill(mode, tbl, v.z, rgbx);
        v.w = op_fill(mode, tbl, v.w, rgbx);
        q[i] = v;
      }
    }
    if (cnt) *cnt += (unsigned)((lane < head) + (lane < tail) + 4 * ((nq - lane + 31) / 32));
    return;
  }
  for (long long x = x0 + lane; x < x1; x += 32) {
    row[x] = op_fill(mode, tbl, row[x], rgbx);
    if (cnt) ++*cnt;
  }
}

// The trapezoid path's pixels for one pair of entries, left (Lm, Lb) and
// right (Rm, Rb), crossing the row at tl0/tl1 and tr0/tr1 (:1752-1835), drawn
// within [xa, xb).
template <bool A8>
__device__ __forceinline__ void apply_trap_pair(RowPx<A8> row, int mode, const uint8_t* tbl, uint32_t rgbx,
                                                long long y, long long W, float Lm, float Lb, float Rm,
                                                float Rb, float tl0, float tl1, float tr0, float tr1,
                                                long long xa, long long xb, int lane, unsigned* cnt = nullptr) {
  const float leftMaxX = nmax(tl0, tl1), rightMinX = nmin(tr0, tr1);
  const long long leftCoverEnd = nim_int(ceilf(leftMaxX));
  const long long rightCoverBegin = nim_int(truncf(rightMinX));
  {  // left sliver (:1752-1788)
    const long long xs = nim_int(nmin(tl0, tl1));
    for (long long x = max(max(xs, 0LL), xa) + lane; x < min(min(leftCoverEnd, W), xb); x += 32) {
      row[x] = blend_row(mode, tbl, row[x], mul_f(rgbx, trap_left_area(Lm, Lb, tl0, tl1, x, xs, y)));
      if (cnt) ++*cnt;
    }
  }
  {  // right sliver (:1790-1828)
    const long long xs = nim_int(rightMinX), xe = nim_int(ceilf(nmax(tr0, tr1)));
    for (long long x = max(max(xs, 0LL), xa) + lane; x < min(min(xe, W), xb); x += 32) {
      row[x] = blend_row(mode, tbl, row[x], mul_f(rgbx, trap_right_area(Rm, Rb, tr0, tr1, x, xs, y)));
      if (cnt) ++*cnt;
    }
  }
  // the fully covered middle (:1830-1835)
  const long long fb = max(min(max(leftCoverEnd, 0LL), W), xa), fe = min(min(max(rightCoverBegin, 0LL), W), xb);
  if (fe > fb) fill_span<A8>(row, mode, tbl, rgbx, fb, fe, lane, cnt);
}

// computeCoverage's accumulation of the sample spans (prevAt, at) in 24.8
// fixed point (:1398-1431) and fillCoverage (:1442-1526) over [cx0, cx1), in
// tiles of XT pixels through the difference array acc (XT + 1 ints).
// computeCoverage's accumulation of the sample spans (prevAt, at) in 24.8
// fixed point (:1398-1431) over the pixels [tx0, tx1) (at most XT): leaves
// acc[i] = coverage of pixel tx0 + i, modulo 256.
template <int XT>
__device__ void cov_tile(const int2* sp, int nsp, int sc, long long tx0, long long tx1, int* acc, int lane) {
  const int L = (int)(tx1 - tx0);
  for (int i = lane; i <= L; i += 32) acc[i] = 0;
  __syncwarp();
  for (int j = lane; j < nsp; j += 32) {
    const int2 spj = sp[j];
    int prevAt = spj.x, at = spj.y;
    long long pi = prevAt / 256, ai = at / 256;
    long long fillStart = pi;
    bool crossed = ai != pi;
    int leftCover = crossed ? (prevAt / 256) * 256 + 256 - prevAt : at - prevAt;
    if (leftCover != 0) {
      fillStart++;
      int v = ((leftCover * sc) / 256) & 255;
      if (pi >= tx0 && pi < tx1) {
        atomicAdd(&acc[pi - tx0], v);
        atomicAdd(&acc[pi - tx0 + 1], -v);
      }
    }
    if (crossed) {
      int rightCover = at - (at / 256) * 256;
      if (rightCover > 0) {
        int v = ((rightCover * sc) / 256) & 255;
        if (ai >= tx0 && ai < tx1) {
          atomicAdd(&acc[ai - tx0], v);
          atomicAdd(&acc[ai - tx0 + 1], -v);
        }
      }
    }
    long long fe = ai;
    long long lo = max(fillStart, tx0), hi = min(fe, tx1);
    if (hi > lo) {
      atomicAdd(&acc[lo - tx0], sc);
      atomicAdd(&acc[hi - tx0], -sc);
    }
  }
  __syncwarp();
  // prefix sum of the difference array, 32 entries per step (lane i holds
  // entry c0 + i: no bank conflicts)
  int carry = 0;
  for (int c0 = 0; c0 < L; c0 += 32) {
    const int i = c0 + lane;
    int v = i < L ? acc[i] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    v += carry;
    if (i < L) acc[i] = v;
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
  __syncwarp();
}

// fillCoverage (:1442-1526) of the sample spans over [cx0, cx1), in tiles of
// XT pixels through the difference array acc (XT + 1 ints).
template <bool A8, int XT>
__device__ void apply_cov(RowPx<A8> row, int mode, const uint8_t* tbl, uint32_t rgbx, const int2* sp, int nsp,
                          int sc, long long cx0, long long cx1, int* acc, int lane, unsigned* cnt = nullptr) {
  const bool maskMode = mode == kMask;
  for (long long tx0 = cx0; tx0 < cx1; tx0 += XT) {
    const long long tx1 = min(tx0 + (long long)XT, cx1);
    const int L = (int)(tx1 - tx0);
    cov_tile<XT>(sp, nsp, sc, tx0, tx1, acc, lane);
    // pixels op_cov leaves unchanged are neither read nor written; the next
    // pixel's backdrop is loaded while the current one is blended
    {
      const uint32_t keep = maskMode ? 255u : 0u;
      uint32_t cvN = lane < L ? ((uint32_t)acc[lane] & 255u) : keep;
      uint32_t bdN = cvN != keep ? (uint32_t)row[tx0 + lane] : 0u;
#pragma unroll 1
      for (int i = lane; i < L; i += 32) {
        const uint32_t cv = cvN, bd = bdN;
        const int in = i + 32;
        cvN = in < L ? ((uint32_t)acc[in] & 255u) : keep;
        bdN = cvN != keep ? (uint32_t)row[tx0 + in] : 0u;
        if (cv != keep) {
          row[tx0 + i] = op_cov(mode, tbl, bd, rgbx, cv);
          if (cnt) ++*cnt;
        }
      }
    }
    __syncwarp();
  }
}

// fillHits (:1540-1591) for a non-mask mode: the single sample's spans are
// sorted and disjoint, so a pixel is inside at most one.
template <bool A8>
__device__ void apply_hits(RowPx<A8> row, int mode, const uint8_t* tbl, uint32_t rgbx, const int2* sp, int nsp,
                           long long xa, long long xb, int lane, unsigned* cnt = nullptr) {
  for (long long x = xa + lane; x < xb; x += 32) {
    bool inside = false;
    for (int j = 0; j < nsp && !inside; j++) {
      long long fs = sp[j].x / 256, fe = sp[j].y / 256;
      if (fe - fs > 0 && x >= fs && x < fe) inside = true;
    }
    if (inside) {
      row[x] = op_fill(mode, tbl, row[x], rgbx);
      if (cnt) ++*cnt;
    }
  }
}

// Row programs: what a row of a path draws, recorded by the scene's first
// pass and replayed by its second.  A program is a header unit then data:
//   kRecCov   n sample spans, coverage step  (computeCoverage + fillCoverage)
//   kRecHits  n spans                        (fillHits, non-AA)
//   kRecTrap  n pairs: {Lm, Lb, Rm, Rb}, {tl0, tl1, tr0, tr1} per pair
// Each row of each path has a header {kind, place, lo, hi} in Arena::rowhdr;
// zero: the row draws nothing.
//   kRecFill  pixels [lo, hi) filled, nothing else stored
//   kRecCov8  coverage bytes of pixels [lo, hi) -- lo a multiple of 16 -- from
//             unit `place` (16 bytes) of Arena::cov8 (the accumulation done
//             once, at record time); zero: the pixel is left alone
//   kRecCov8Z a list at unit `place` of Arena::prog: {cov8 unit, n, first, last}
//             and n pixels besides (at most kZeroCap, between first and last), each
//             {x, area}: blended with an empty source or a multiplier above 255
//   kRecProg  a program at unit `place` of Arena::prog
enum RecKind { kRecFill = 1, kRecCov = 2, kRecHits = 3, kRecTrap = 4, kRecCov8 = 5, kRecCov8Z = 6, kRecProg = 7 };

// Allocates `units` 16-byte units for row y of job J's program, stores its
// place for the row (drawn within [lo, hi)), and returns it (lane-uniform);
// -1 if the arena is full.
__device__ __forceinline__ long long rec_alloc(const PathJob& J, const Arena& A, long long y, int kind, int units,
                                               long long lo, long long hi, int lane) {
  unsigned long long base = 0;
  if (lane == 0) {
    base = atomicAdd(&A.counters[kCtrProg], (unsigned long long)units);
    if ((long long)(base + units) > A.prog_cap || base + units > (unsigned long long)INT_MAX) {
      atomicOr(&A.counters[kCtrProgFull], 1ull);
      base = ~0ull;
    } else {
      A.rowhdr[J.ri_off + y * J.ri_stride] = make_int4(kind, (int)base, (int)lo, (int)hi);
    }
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  return base == ~0ull ? -1 : (long long)base;
}

// Draws the pixels [xa, xb) of row y of job J (the whole row: 0, W).
// Returns false, having drawn nothing, when the row's crossings exceed MAXH
// (the caller retries it with a larger scratch).
// With REC the row is not drawn: its program is recorded instead (non-mask
// modes only).
template <int MAXH, int XT, bool A8, bool REC = false>
__device__ bool process_row(const PathJob& J, const Arena& A, const uint8_t* tbl, int job,
                            long long y, RowScratch<MAXH, XT>& S, int lane, long long xa,
                            long long xb) {
  const long long W = J.W;
  const RowPx<A8> row = row_of<A8>(J, y);
  const int mode = J.mode;
  const uint32_t rgbx = J.rgbx;
  const bool maskMode = mode == kMask;
  const unsigned lt = (1u << lane) - 1;

  long long k = (y - J.startY) / (long long)J.ph;
  if (k >= J.nb) k = J.nb - 1;
  const Band bd = A.bands[J.band_off + k];
  const float scanTop = (float)y, scanBottom = (float)(y + 1);
  // the band's top and bottom (:1178-1190)
  const float top = (float)(J.startY + k * (long long)J.ph);
  const float bottom = (float)(k == J.nb - 1 ? J.pathHeight : J.startY + (k + 1) * (long long)J.ph);
  const float4* SG = A.segs + J.seg_off;
  const int* SW = A.segw + J.seg_off;
  const int* BL = A.bandseg + bd.off;  // the band's segments, ascending
  const int nb = bd.count;
  Entry* E = S.ent;

  // a band of exactly two entries: are they two non-intersecting segments
  // spanning the band (:1250-1262)?
  bool two = false;
  if (nb == 2) {
    if (lane < 2) {
      const int i = BL[lane];
      E[lane] = make_entry(SG[i], SW[i], top, bottom);
    }
    __syncwarp();
    Entry e0 = E[0], e1 = E[1];
    if (!intersectsInside(V2{e0.ax, e0.ay}, V2{e0.bx, e0.by}, V2{e1.ax, e1.ay}, V2{e1.bx, e1.by}) &&
        e0.ay <= top && e0.by >= bottom && e1.ay <= top && e1.by >= bottom) {
      two = true;
      if ((e0.ax + e0.bx) * 0.5f > (e1.ax + e1.bx) * 0.5f) {
        __syncwarp();
        if (lane == 0) {
          E[0] = e1;
          E[1] = e0;
        }
      }
    }
    __syncwarp();
  }

  // (i) non-AA band with two spanning vertical edges (:1644-1668)
  if (two && !(bd.flags & kBandAA)) {
    long long minX = min(max(nim_int(E[0].ax), 0LL), W);
    long long maxX = min(max(nim_int(E[1].ax), 0LL), W);
    if (REC) {
      if (lane == 0 && maxX > minX)
        A.rowhdr[J.ri_off + y * J.ri_stride] = make_int4(kRecFill, 0, (int)minX, (int)maxX);
      return true;
    }
    for (long long x = xa + lane; x < xb; x += 32) {
      if (x >= minX && x < maxX) row[x] = op_fill(mode, tbl, row[x], rgbx);
      else if (maskMode) row[x] = 0u;
    }
    return true;
  }

  // entries overlapping the scanline [y, y+1) in band order (:1677-1693)
  int n = 0;
  bool allSpan = true;
  if (two) {
    n = 2;
  } else {
    for (int c0 = 0; c0 < nb; c0 += 32) {
      const int j = c0 + lane;
      bool pred = false, ns = false;
      Entry e;
      if (j < nb) {
        const int i = BL[j];
        e = make_entry(SG[i], SW[i], top, bottom);
        pred = !(e.by <= scanTop || e.ay >= scanBottom);
        ns = e.ay > scanTop || e.by < scanBottom;
      }
      unsigned m = __ballot_sync(0xffffffffu, pred);
      if (__any_sync(0xffffffffu, pred && ns)) allSpan = false;
      int pos = n + __popc(m & lt);
      if (pred && pos < MAXH) E[pos] = e;
      n += __popc(m);
    }
  }
  for (int i = lane; i < min(n, MAXH); i += 32) S.idx[i] = i;
  if (n > MAXH) return false;  // too many crossings for this scratch
  __syncwarp();

  // (ii) trapezoid fast path (:1695-1872)
  if (allSpan && (n % 2) == 0) {
    float* t0 = reinterpret_cast<float*>(S.a0);
    float* t1 = reinterpret_cast<float*>(S.a1);
    float* key = reinterpret_cast<float*>(S.a2);
    bool anyNaN = false;
    for (int i = lane; i < n; i += 32) {
      Entry e = E[S.idx[i]];
      float xt = e.m == 0 ? e.b : (scanTop - e.b) / e.m;   // solveX :1137-1141
      float xbt = e.m == 0 ? e.b : (scanBottom - e.b) / e.m;
      t0[i] = xt;
      t1[i] = xbt;
      key[i] = (xt + xbt) * 0.5f;
      anyNaN |= isnan(key[i]);
    }
    anyNaN = __any_sync(0xffffffffu, anyNaN);
    __syncwarp();
    // stable insertion sort by midpoint (:1710-1719)
    if (anyNaN) {
      if (lane == 0) {
        for (int i = 1; i < n; i++) {
          int j = i - 1, kk = i;
          while (j >= 0 && key[j] > key[kk]) {
            float tk = key[j]; key[j] = key[j + 1]; key[j + 1] = tk;
            float ta = t0[j]; t0[j] = t0[j + 1]; t0[j + 1] = ta;
            float tb = t1[j]; t1[j] = t1[j + 1]; t1[j + 1] = tb;
            int ti = S.idx[j]; S.idx[j] = S.idx[j + 1]; S.idx[j + 1] = ti;
            j--;
            kk--;
          }
        }
      }
    } else {
      float* t0s = reinterpret_cast<float*>(S.a3);
      float* t1s = reinterpret_cast<float*>(S.a4);
      for (int i = lane; i < n; i += 32) {
        int r = stable_rank_f(key, n, i);
        S.a5[r] = S.idx[i];
        t0s[r] = t0[i];
        t1s[r] = t1[i];
      }
      __syncwarp();
      for (int i = lane; i < n; i += 32) {
        S.idx[i] = S.a5[i];
        t0[i] = t0s[i];
        t1[i] = t1s[i];
      }
    }
    __syncwarp();
    // partial coverage of neighbours must not overlap (:1721-1731)
    bool overlap = false;
    for (int i = lane; i < n - 1; i += 32) {
      float leftMaxX = nmax(t0[i], t1[i]);
      float rightMinX = nmin(t0[i + 1], t1[i + 1]);
      if (nim_int(ceilf(leftMaxX)) > nim_int(rightMinX)) overlap = true;
    }
    overlap = __any_sync(0xffffffffu, overlap);
    bool simple = false;
    if (!overlap) {  // pairs must be simple fills (:1733-1750)
      int ok = 1;
      if (lane == 0) {
        long long wc = 0;
        for (int i = 0; i < n; i += 2) {
          wc += E[S.idx[i]].w;
          if (!shouldFill(J.winding, wc)) { ok = 0; break; }
          wc += E[S.idx[i + 1]].w;
          if (shouldFill(J.winding, wc)) { ok = 0; break; }
        }
      }
      simple = __shfl_sync(0xffffffffu, ok, 0) != 0;
    }
    if (simple && REC) {
      const int np = n / 2;
      const long long at = rec_alloc(J, A, y, kRecProg, 1 + 2 * np, 0, W, lane);
      if (at >= 0) {
        if (lane == 0) A.prog[at] = make_int4(kRecTrap, np, 0, 0);
        for (int p = lane; p < np; p += 32) {
          const Entry L = E[S.idx[2 * p]], R = E[S.idx[2 * p + 1]];
          A.prog[at + 1 + 2 * p] = make_int4(__float_as_int(L.m), __float_as_int(L.b), __float_as_int(R.m),
                                             __float_as_int(R.b));
          A.prog[at + 2 + 2 * p] = make_int4(__float_as_int(t0[2 * p]), __float_as_int(t1[2 * p]),
                                             __float_as_int(t0[2 * p + 1]), __float_as_int(t1[2 * p + 1]));
        }
      }
      return true;
    }
    if (simple) {
      long long filledTo = 0;
      for (int i = 0; i < n; i += 2) {
        const Entry L = E[S.idx[i]], R = E[S.idx[i + 1]];
        const float tl0 = t0[i], tl1 = t1[i], tr0 = t0[i + 1], tr1 = t1[i + 1];
        apply_trap_pair<A8>(row, mode, tbl, rgbx, y, W, L.m, L.b, R.m, R.b, tl0, tl1, tr0, tr1, xa, xb, lane);
        if (maskMode) {  // :1837-1845
          long long clearTo = nim_int(nmin(tl0, tl1));
          clear_span_linear(J, A, job, row, y, min(filledTo, W), min(clearTo, W), lane, xa, xb);
        }
        filledTo = nim_int(ceilf(nmax(tr0, tr1)));
      }
      if (maskMode) clear_span_linear(J, A, job, row, y, min(filledTo, W), W, lane, xa, xb);
      return true;
    }
  }

  // (iii) computeCoverage (:1350-1431) + fillCoverage / fillHits
  const bool aa = (bd.flags & kBandAA) != 0;
  const int quality = aa ? 5 : 1;
  const int sc = 255 / quality;
  const float offset = 1.0f / (float)quality;
  const float initialOffset = offset / 2 + kEps;
  float yLine = (float)y + initialOffset - offset;
  if (lane == 0) S.nsp = 0;
  __syncwarp();
  for (int m = 0; m < quality; m++) {
    yLine += offset;
    int nh = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
      int i = c0 + lane;
      bool hit = false;
      int fx = 0, w = 0;
      if (i < n) {
        Entry e = E[S.idx[i]];
        if (e.ay <= yLine && e.by >= yLine) {
          hit = true;
          float x = e.m == 0 ? e.b : (yLine - e.b) / e.m;
          fx = nim_i32(nmin(x, (float)W) * 256.0f);
          w = e.w;
        }
      }
      unsigned msk = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        int pos = nh + __popc(msk & lt);
        S.a0[pos] = fx;
        S.a1[pos] = w;
      }
      nh += __popc(msk);
    }
    __syncwarp();
    for (int i = lane; i < nh; i += 32) {  // stable sort (:1277-1286)
      int r = stable_rank_i(S.a0, nh, i);
      S.a2[r] = S.a0[i];
      S.a3[r] = S.a1[i];
    }
    __syncwarp();
    // walk (:1298-1334).  Without two adjacent hits at the same position the
    // look-ahead that skips a cancelling pair never fires, and every hit's
    // part in the walk follows from the winding count before it (a prefix
    // sum): the warp walks 32 hits at a time.  Otherwise lane 0 walks.
    bool adjEq = false;
    for (int i = lane; i + 1 < nh; i += 32) adjEq |= S.a2[i] == S.a2[i + 1];
    if (!__any_sync(0xffffffffu, adjEq)) {
      int ns = S.nsp, carry = 0, prevCarry = 0;
      for (int c0 = 0; c0 < nh; c0 += 32) {
        const int i = c0 + lane;
        const bool valid = i < nh;
        const int at = valid ? S.a2[i] : 0, w = valid ? S.a3[i] : 0;
        int incl = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const int count = carry + incl - w;
        const bool pos = valid && at > 0;
        const bool fill = shouldFill(J.winding, count);
        const bool shortcut = fill && i < nh - 1 && J.winding == 0 && count + w != 0;
        const bool emit = pos && fill && !shortcut;
        const bool upd = pos && (!fill || emit);  // hits that set prevAt
        const unsigned um = __ballot_sync(0xffffffffu, upd);
        const unsigned below = um & lt;
        const int src = below ? 31 - __clz(below) : lane;
        const int pa = __shfl_sync(0xffffffffu, at, src);
        const int prevAt = below ? pa : prevCarry;
        const unsigned em = __ballot_sync(0xffffffffu, emit);
        const int slot = ns + __popc(em & lt);
        if (emit && slot < RowScratch<MAXH, XT>::SPCAP) S.sp[slot] = make_int2(prevAt, at);
        ns += __popc(em);
        carry += __shfl_sync(0xffffffffu, incl, 31);
        if (um) prevCarry = __shfl_sync(0xffffffffu, at, 31 - __clz(um));
      }
      __syncwarp();
      if (lane == 0) S.nsp = ns;
    } else if (lane == 0) {
      int i = 0, ns = S.nsp;
      long long count = 0;
      int prevAt = 0;
      while (i < nh) {
        int at = S.a2[i], winding = S.a3[i];
        if (at > 0) {
          if (shouldFill(J.winding, count)) {
            if (i < nh - 1) {
              int nextAt = S.a2[i + 1], nextW = S.a3[i + 1];
              if (nextAt == at && winding + nextW == 0) {
                i += 2;
                continue;
              }
              if (J.winding == 0 && count + winding != 0) {
                count += winding;
                i++;
                continue;
              }
            }
            if (ns < RowScratch<MAXH, XT>::SPCAP) S.sp[ns] = make_int2(prevAt, at);
            ns++;
          }
          prevAt = at;
        }
        count += winding;
        i++;
      }
      S.nsp = ns;
    }
    __syncwarp();
  }
  const int nsp = min(S.nsp, RowScratch<MAXH, XT>::SPCAP);

  if (REC) {
    if (nsp > 0 && aa) {
      // the pixels the spans can touch, within the path's bounds
      long long lo = LLONG_MAX, hi = LLONG_MIN;
      for (int j = lane; j < nsp; j += 32) {
        lo = min(lo, (long long)(S.sp[j].x / 256));
        hi = max(hi, (long long)(S.sp[j].y / 256) + 1);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      lo = max(lo, J.startX);
      hi = min(hi, J.startX + J.pathWidth);
      if (hi <= lo) return true;
      // coverage bytes when the arena has room (else the spans are recorded)
      const long long lo16 = lo & ~15LL;
      const unsigned long long nbytes = (unsigned long long)((hi - lo16 + 15) & ~15LL);
      unsigned long long cb = 0;
      if (lane == 0) {
        cb = atomicAdd(&A.counters[kCtrCov8], nbytes);
        if ((long long)(cb + nbytes) > A.cov8_cap) cb = ~0ull;
      }
      cb = __shfl_sync(0xffffffffu, cb, 0);
      if (cb != ~0ull) {
        if (lane == 0)
          A.rowhdr[J.ri_off + y * J.ri_stride] = make_int4(kRecCov8, (int)(cb >> 4), (int)lo16, (int)hi);
        uint8_t* dst = A.cov8 + cb;
        for (int i = lane; i < (int)(lo - lo16); i += 32) dst[i] = 0;
        for (long long i = hi - lo16 + lane; i < (long long)nbytes; i += 32) dst[i] = 0;
        for (long long tx0 = lo; tx0 < hi; tx0 += XT) {
          const long long tx1 = min(tx0 + (long long)XT, hi);
          cov_tile<XT>(S.sp, nsp, sc, tx0, tx1, S.acc, lane);
          for (int i = lane; i < (int)(tx1 - tx0); i += 32) dst[tx0 - lo16 + i] = (uint8_t)(S.acc[i] & 255);
          __syncwarp();
        }
        return true;
      }
    }
    const long long at =
        nsp > 0 ? rec_alloc(J, A, y, kRecProg, 1 + (nsp + 1) / 2, aa ? J.startX : 0, aa ? J.startX + J.pathWidth : W, lane) : -1;
    if (at >= 0) {
      if (lane == 0) A.prog[at] = make_int4(aa ? kRecCov : kRecHits, nsp, sc, 0);
      int2* d = reinterpret_cast<int2*>(A.prog + at + 1);
      for (int j = lane; j < nsp; j += 32) d[j] = S.sp[j];
    }
    return true;
  }
  if (aa) {
    // coverage row over [startX, startX + pathWidth) in tiles of XT pixels
    const long long px0 = J.startX, px1 = J.startX + J.pathWidth;
    if (maskMode) {
      for (long long x = xa + lane; x < xb; x += 32)
        if (x < px0 || x >= px1) row[x] = 0u;
    }
    apply_cov<A8, XT>(row, mode, tbl, rgbx, S.sp, nsp, sc, max(px0, xa), min(px1, xb), S.acc, lane);
  } else if (maskMode) {
    // fillHits with the single sample's spans (:1540-1591); spans are sorted
    // and disjoint, so a pixel is inside at most one.
    const long long startX = J.startX;
    for (long long x = xa + lane; x < xb; x += 32) {
      bool inside = false;
      for (int j = 0; j < nsp && !inside; j++) {
        long long fs = S.sp[j].x / 256, fe = S.sp[j].y / 256;
        if (fe - fs > 0 && x >= fs && x < fe) inside = true;
      }
      row[x] = (x >= startX && inside) ? op_fill(mode, tbl, row[x], rgbx) : 0u;
    }
  } else {
    apply_hits<A8>(row, mode, tbl, rgbx, S.sp, nsp, xa, xb, lane);
  }
  return true;
}

}  // namespace pxg
#include "rowfast.cuh"
#include "setup.cuh"
namespace pxg {

constexpr int kFastMaxH = 256, kFastXT = 1024, kFastWarps = 4;
constexpr int kWideMaxH = 2048, kWideXT = 1024;

// The persistent row kernel: every warp takes work items -- rpi consecutive
// rows of one job's path -- from a device queue (one atomic per item, issued
// while the item before is drawn) until the queue is empty, so jobs of uneven
// height share the GPU evenly.  Rows the engine hands on go to the wide
// kernel.  NB = 64 with a 256-pixel tile is for small paths such as glyphs:
// a quarter of the shared memory per warp.
template <int OUT, int NB, int XT, int WARPS, int TILES>
__global__ void __launch_bounds__(WARPS * 32) k_rows_fast(PathJob* jobs, const long long* offs, int njobs, Arena A,
                                                          const uint8_t* tbl, long long totalItems, int rpi) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  FastRow<NB, XT>& S = reinterpret_cast<FastRow<NB, XT>*>(rsm)[warp];
  init_fast_row(S, lane);
  pdl_trigger();
  pdl_wait();  // the setup's segments, bands and queue counters
  unsigned long long q = 0;
  if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue], 1ull);
  while (true) {
    const long long item = (long long)__shfl_sync(0xffffffffu, q, 0);
    if (item >= totalItems) break;
    if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue], 1ull);
    int lo = 0, hi = njobs - 1;  // job with row_off <= item (offs: the jobs' row_off, packed)
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (offs[mid] <= item) lo = mid;
      else hi = mid - 1;
    }
    const PathJob& J = jobs[lo];
    if (J.status != kOk) continue;
    int r = rpi;
    if (OUT == kOutRgbx && rpi > 1) {
      // the host chose by the image's rows; a path that has few of them is spread
      // over all of the job's items (64 rows of a 64 x 20000 image are 16 chains of
      // four by the image's, 69 us; 56 us so)
      const int chunks = (int)((J.H + rpi - 1) / rpi);
      r = (int)((J.pathHeight - J.startY + chunks - 1) / chunks);
    }
    const long long yA = J.startY + (item - J.row_off) * r, yB = min(yA + r, J.pathHeight);
    if (yA < yB) fast_rows<OUT, NB, XT, TILES>(J, A, tbl, lo, (int)yA, (int)yB, S, lane);
  }
}
constexpr int kRowsNB = 256, kRowsXT = 1024, kRowsWarps = 4;

// The same for launches whose rows all fit the GPU at once, a CTA each: the
// launch lasts as long as the busiest row, and a warp per sample line shortens
// it (64 cubics on 512 x 512: 29 -> 21 us).
constexpr int kRowsLineThreads = kLineWarps * 32;
template <int TILES>
__global__ void __launch_bounds__(kRowsLineThreads) k_rows_lines(PathJob* jobs, const long long* offs, int njobs,
                                                                 Arena A, const uint8_t* tbl, long long totalItems) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LineRow<kRowsNB, kRowsXT>& S = *reinterpret_cast<LineRow<kRowsNB, kRowsXT>*>(rsm);
  pdl_trigger();
  pdl_wait();
  if (warp > 0) {
    line_warps<true>(S, warp, lane);
    return;
  }
  init_fast_row(S.row, lane);
#pragma unroll 1
  for (long long item = blockIdx.x; item < totalItems; item += gridDim.x) {
    int lo = 0, hi = njobs - 1;
#pragma unroll 1
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (offs[mid] <= item) lo = mid;
      else hi = mid - 1;
    }
    const PathJob& J = jobs[lo];
    const int y = (int)(J.startY + (item - J.row_off));
    if (J.status != kOk || y >= (int)J.pathHeight) continue;
    fast_rows<kOutRgbx, kRowsNB, kRowsXT, TILES, 0, true>(J, A, tbl, lo, y, y + 1, S.row, lane, &S.work, S.line);
  }
  line_warps_end(S.work, lane);
}

__host__ __device__ bool rows_huge_fits(long long W) { return W < fast_max_w(kWideMaxH); }
// Rows of RGBX launches with more than kRowsNB crossings (list 0), up to
// kWideMaxH of them; the rest to list 1.  They are few and each takes long: a
// stroke of 300 points with round joins has five, 160 us by the general code
// on a warp each after a wait for the host, 56 so.
template <int TILES>
__global__ void __launch_bounds__(kRowsLineThreads) k_rows_huge(PathJob* jobs, Arena A, const uint8_t* tbl) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LineRow<kWideMaxH, kWideXT>& S = *reinterpret_cast<LineRow<kWideMaxH, kWideXT>*>(rsm);
  pdl_trigger();
  pdl_wait();
  if (warp > 0) {
    line_warps<true>(S, warp, lane);
    return;
  }
  init_fast_row(S.row, lane);
  const long long n = (long long)min((unsigned long long)A.ovf_cap, A.counters[kCtrOvfRows]);
#pragma unroll 1
  for (long long i = blockIdx.x; i < n; i += gridDim.x) {
    const long long v = A.ovf_rows[i];
    const int job = (int)(v >> 32), y = (int)(v & 0xffffffffLL);
    const PathJob& J = jobs[job];
    const int k = min((y - (int)J.startY) / (int)J.ph, J.nb - 1);
    // a band of more than kWideMaxH entries is an error, which the general kernel reports
    if (!rows_huge_fits(J.W) || A.bands[J.band_off + k].count > kWideMaxH) push_row(A, job, y, lane, 1);
    else fast_rows<kOutRgbx, kWideMaxH, kWideXT, TILES, 1, true>(J, A, tbl, job, y, y + 1, S.row, lane, &S.work, S.line);
  }
  line_warps_end(S.work, lane);
}
constexpr int kGlyphNB = 64, kGlyphXT = 256, kGlyphWarps = 8;

// The general row kernel (launches with MaskBlend paths, whose clears reach
// outside the path, or images too wide for the row engine's sort keys): the same queue,
// over all rows of the images.  Rows whose crossings exceed MAXH go to the
// wide kernel.
template <int MAXH, int XT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_rows(PathJob* jobs, const long long* offs, int njobs, Arena A,
                                                     const uint8_t* tbl, long long totalItems, int rpi) {
  extern __shared__ __align__(16) unsigned char rsm[];
  using Scratch = RowScratch<MAXH, XT>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Scratch& S = reinterpret_cast<Scratch*>(rsm)[warp];
  pdl_trigger();
  pdl_wait();  // the setup's segments, bands and queue counters
  while (true) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue], 1ull);
    const long long item = (long long)__shfl_sync(0xffffffffu, q, 0);
    if (item >= totalItems) break;
    int lo = 0, hi = njobs - 1;  // job with row_off <= item (offs: the jobs' row_off, packed)
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (offs[mid] <= item) lo = mid;
      else hi = mid - 1;
    }
    const PathJob& J = jobs[lo];
    if (J.status != kOk) continue;
    const long long y0 = (item - J.row_off) * rpi;
    for (long long y = y0; y < y0 + rpi && y < J.H; y++) {
      if (y < J.startY || y >= J.pathHeight) {
        if (J.mode == kMask) {  // :1910-1912 (never an A8 job)
          const RowPx<false> row = row_of<false>(J, y);
          for (long long x = lane; x < J.W; x += 32) row[x] = 0u;
        }
        continue;
      }
      const bool ok = J.a8 ? process_row<MAXH, XT, true>(J, A, tbl, lo, y, S, lane, 0, J.W)
                           : process_row<MAXH, XT, false>(J, A, tbl, lo, y, S, lane, 0, J.W);
      if (!ok && lane == 0) {
        // too many crossings for this kernel: hand the row to the wide kernel
        unsigned long long slot = atomicAdd(&A.counters[kCtrOvfRows], 1ull);
        if ((long long)slot < A.ovf_cap) A.ovf_rows[slot] = ((long long)lo << 32) | y;
      }
      __syncwarp();
    }
  }
}

// Rows the kernels before handed on (list 0 or 1), by the general row code: one
// warp per CTA with room for kWideMaxH crossings.  They come in the order in
// which they were handed on and differ in length, so the CTAs take them from a
// queue.
__global__ void __launch_bounds__(32) k_rows_wide(PathJob* jobs, Arena A, const uint8_t* tbl, int list) {
  extern __shared__ __align__(16) unsigned char rsm[];
  using Scratch = RowScratch<kWideMaxH, kWideXT>;
  Scratch& S = *reinterpret_cast<Scratch*>(rsm);
  const int lane = threadIdx.x & 31;
  const long long n = (long long)min((unsigned long long)A.ovf_cap, A.counters[list ? kCtrOvfRows2 : kCtrOvfRows]);
  while (true) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue2], 1ull);
    const long long i = (long long)__shfl_sync(0xffffffffu, q, 0);
    if (i >= n) break;
    long long v = A.ovf_rows[list * A.ovf_cap + i];
    int job = (int)(v >> 32);
    long long y = v & 0xffffffffLL;
    PathJob& J = jobs[job];
    // a row whose band exceeds the wide kernel too reports an error
    long long k = (y - J.startY) / (long long)J.ph;
    if (k >= J.nb) k = J.nb - 1;
    const Band bd = A.bands[J.band_off + k];
    if (bd.count > kWideMaxH) {
      if (lane == 0) J.status = kErrRowTooComplex;
      continue;
    }
    const bool ok = J.a8 ? process_row<kWideMaxH, kWideXT, true>(J, A, tbl, job, y, S, lane, 0, J.W)
                         : process_row<kWideMaxH, kWideXT, false>(J, A, tbl, job, y, S, lane, 0, J.W);
    if (!ok && lane == 0) J.status = kErrRowTooComplex;
  }
}

// Clears that the reference's linear-index clearUnsafe applies to earlier
// rows (a trapezoid fill extending left of the image in MaskBlend); they
// run after every row has been drawn, as they did in the row-ordered loop.
__global__ void k_xclears(PathJob* jobs, Arena A) {
  long long n = (long long)min((unsigned long long)A.xclear_cap, A.counters[kCtrXClears]);
  for (long long i = blockIdx.x; i < n; i += gridDim.x) {
    const PathJob& J = jobs[A.xclears[3 * i]];
    uint32_t* px = reinterpret_cast<uint32_t*>(J.img);
    for (long long p = A.xclears[3 * i + 1] + threadIdx.x; p < A.xclears[3 * i + 2]; p += blockDim.x)
      px[p] = 0u;
  }
}

// Dense scenes, in two passes.
// k_scene_rec: every row of every path of the launch, independent of the
// pixels, in chunks from a device queue (rowfast.cuh): the row's coverage
// bytes (or, rarely, its program: RecKind).  k_scene_big,
// k_scene_huge and k_scene_rest record the rows it hands on.
// k_scene: a warp owns a slice of one canvas row (sliceW pixels) and replays
// every path's program for that row in submission order, so each pixel sees
// the paths in the order the reference's sequence of fillPath/strokePath
// calls applies them.  A path that failed in setup stops its run there (the
// reference raises at that call).  If the program arena overflowed, k_scene
// draws nothing and the host reruns the launch with a larger arena.
constexpr int kRecNB = 128, kRecRowXT = 1024, kRecRowWarps = 4;
__global__ void __launch_bounds__(kRecRowWarps * 32, 7) k_scene_rec(PathJob* jobs, const RecOrder* order, int njobs,
                                                                 long long totalItems, int rpi, Arena A) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  FastRow<kRecNB, kRecRowXT>& S = reinterpret_cast<FastRow<kRecNB, kRecRowXT>*>(rsm)[warp];
  init_fast_row(S, lane);
  pdl_trigger();
  pdl_wait();
  unsigned long long q = 0;
  if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue], 1ull);
#pragma unroll 1
  while (true) {
    const long long item = (long long)__shfl_sync(0xffffffffu, q, 0);
    if (item >= totalItems) break;
    if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue], 1ull);
    // chunks of rpi rows, path by path in the launch's recording order
    int lo = 0, hi = njobs - 1;
#pragma unroll 1
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (order[mid].first <= item) lo = mid;
      else hi = mid - 1;
    }
    const int job = order[lo].job;
    const PathJob& J = jobs[job];
    if (J.status != kOk) continue;
    const int yA = (int)J.startY + (int)(item - order[lo].first) * rpi, yB = min(yA + rpi, (int)J.pathHeight);
    if (yA >= yB) continue;
    if (J.W >= fast_max_w(kRecNB)) {
#pragma unroll 1
      for (int y = yA; y < yB; y++) push_row(A, job, y, lane);
      continue;
    }
    fast_rows<kOutRec, kRecNB, kRecRowXT, kAgain>(J, A, nullptr, job, yA, yB, S, lane);
  }
}

// The rows k_scene_rec handed on (list 0): up to 512 crossings -- stroke
// outlines overlap themselves hundreds of times a row -- with fewer warps; the
// rest to list 1.
constexpr int kBigNB = 512, kBigXT = 1024, kBigWarps = 4;
__global__ void __launch_bounds__(kBigWarps * 32) k_scene_big(PathJob* jobs, Arena A) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  FastRow<kBigNB, kBigXT>& S = reinterpret_cast<FastRow<kBigNB, kBigXT>*>(rsm)[warp];
  init_fast_row(S, lane);
  pdl_trigger();
  pdl_wait();
  const long long n = (long long)min((unsigned long long)A.ovf_cap, A.counters[kCtrOvfRows]);
#pragma unroll 1
  for (long long i = (long long)blockIdx.x * kBigWarps + warp; i < n; i += (long long)gridDim.x * kBigWarps) {
    const long long v = A.ovf_rows[i];
    const int job = (int)(v >> 32), y = (int)(v & 0xffffffffLL);
    const PathJob& J = jobs[job];
    if (J.W >= fast_max_w(kBigNB)) push_row(A, job, y, lane, 1);
    else fast_rows<kOutRec, kBigNB, kBigXT, kAgain, 1>(J, A, nullptr, job, y, y + 1, S, lane);
  }
}

// List 1: up to 2048 crossings, a CTA per row and a warp per sample line, for
// these rows are few and each takes long (a warp each, the widest rows of a
// 240-path scene took 347 us, this way 74); the rest to list 2.
// (By a CTA per row the rows of up to 512 crossings of 240 local paths take 135
// us instead of 157, but those of 2000 paths over 1024 x 1024 1156 instead of
// 944: warp 0's share of a row leaves the other warps idle.)
constexpr int kHugeNB = 2048, kHugeXT = 1024;
__global__ void __launch_bounds__(kLineWarps * 32) k_scene_huge(PathJob* jobs, Arena A) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LineRow<kHugeNB, kHugeXT>& S = *reinterpret_cast<LineRow<kHugeNB, kHugeXT>*>(rsm);
  pdl_trigger();
  pdl_wait();
  if (warp > 0) {
    line_warps<false>(S, warp, lane);
    return;
  }
  init_fast_row(S.row, lane);
  const long long n = (long long)min((unsigned long long)A.ovf_cap, A.counters[kCtrOvfRows2]);
#pragma unroll 1
  for (long long i = blockIdx.x; i < n; i += gridDim.x) {
    const long long v = A.ovf_rows[A.ovf_cap + i];
    const int job = (int)(v >> 32), y = (int)(v & 0xffffffffLL);
    const PathJob& J = jobs[job];
    if (J.W >= fast_max_w(kHugeNB)) push_row(A, job, y, lane, 2);
    else fast_rows<kOutRec, kHugeNB, kHugeXT, kAgain, 2, true>(J, A, nullptr, job, y, y + 1, S.row, lane, &S.work, S.line);
  }
  line_warps_end(S.work, lane);
}

// The rows k_scene_huge handed on (list 2), by the general row code; those with
// more than MAXH crossings take a per-warp global scratch.
constexpr int kRecXT = 256;  // coverage tile of the general recording code
template <int MAXH, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_scene_rest(PathJob* jobs, Arena A, unsigned char* wide,
                                                           long long wideSlots) {
  extern __shared__ __align__(16) unsigned char rsm[];
  using Scratch = RowScratch<MAXH, kRecXT>;
  using Wide = RowScratch<kWideMaxH, kWideXT>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  Scratch& S = reinterpret_cast<Scratch*>(rsm)[warp];
  const long long gw = (long long)blockIdx.x * WARPS + warp;
  const long long n = (long long)min((unsigned long long)A.ovf_cap, A.counters[kCtrOvfRows3]);
  for (long long i = gw; i < n; i += (long long)gridDim.x * WARPS) {
    const long long v = A.ovf_rows[2 * A.ovf_cap + i];
    const int lo = (int)(v >> 32);
    const long long y = v & 0xffffffffLL;
    const PathJob& J = jobs[lo];
    bool ok = process_row<MAXH, kRecXT, false, true>(J, A, nullptr, lo, y, S, lane, 0, J.W);
    if (!ok && gw < wideSlots) {
      __syncwarp();
      ok = process_row<kWideMaxH, kWideXT, false, true>(J, A, nullptr, lo, y, reinterpret_cast<Wide*>(wide)[gw],
                                                        lane, 0, J.W);
    }
    if (!ok && lane == 0) atomicMin(&A.counters[kCtrRowErr], (unsigned long long)lo);
    __syncwarp();
  }
}

// A recorded program (RecKind) drawn within [xa, xb) of a row by the general
// code; out of line, for rows are rarely recorded so.  Returns the number of
// blends.
template <int XT>
static __device__ __noinline__ unsigned draw_program(RowPx<false> row, int mode, const uint8_t* tbl, uint32_t rgbx,
                                                     const int4* prog, int lo, int hi, long long y, int W, int xa,
                                                     int xb, int* acc, int lane) {
  unsigned cnt = 0;
  const int4 g = prog[0];
  if (g.x == kRecCov) {
    apply_cov<false, XT>(row, mode, tbl, rgbx, reinterpret_cast<const int2*>(prog + 1), g.y, g.z, max(lo, xa),
                         min(hi, xb), acc, lane, &cnt);
  } else if (g.x == kRecHits) {
    apply_hits<false>(row, mode, tbl, rgbx, reinterpret_cast<const int2*>(prog + 1), g.y, xa, xb, lane, &cnt);
  } else if (g.x == kRecTrap) {
#pragma unroll 1
    for (int t = 0; t < g.y; t++) {
      const int4 e = prog[1 + 2 * t], u = prog[2 + 2 * t];
      apply_trap_pair<false>(row, mode, tbl, rgbx, y, W, __int_as_float(e.x), __int_as_float(e.y), __int_as_float(e.z),
                             __int_as_float(e.w), __int_as_float(u.x), __int_as_float(u.y), __int_as_float(u.z),
                             __int_as_float(u.w), xa, xb, lane, &cnt);
    }
  }
  return __reduce_add_sync(0xffffffffu, cnt);
}

// The drawing pass.  What bounds it: issue -- a blend is 40 to 250 instructions
// a pixel and the modes of a scene differ path by path -- and the latency of
// one warp's path sequence.  A lane keeps PPL pixels of a step (pixels lane,
// lane + 32, ...) in registers while the launch's paths are applied, so a path
// costs its coverage bytes (one word per lane, requested a path ahead, dealt
// out by shuffles) and no pixel traffic; 32-pixel groups a path does not touch
// are skipped, and each mode's blend exists once (the lane's pixels rotate
// through it), which keeps the kernel within the instruction cache.  What a
// path costs besides its blends -- 250 of 290 us for 100 paths of one mode over
// 1024 x 1024 before, 200 of 240 now -- is kept in two words worked out for 32
// paths at once, groups of full coverage take the colour as it is, Normal runs
// through its groups without a branch on the pixels, and steps that were opaque
// take blend_opaque: 2000 paths 9.65 -> 8.45 ms, 240 local ones 0.16 -> 0.138,
// Color of 100 paths 0.66 -> 0.54, Screen 0.34 -> 0.31.  PPL = 4;
// PPL = 1 for launches with too few rows to fill the GPU, where a path's time
// on its warp matters and not the instructions per pixel.
template <int PPL, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 4) k_scene(const SceneRun* runs, int nruns, long long totalItems,
                                                         Arena A, const uint8_t* tbl, int sliceW) {
  constexpr int SW = 32 * PPL;          // pixels of a step
  __shared__ int accs[WARPS][SW + 1];   // recorded programs: a coverage tile and the step's pixels
  __shared__ uint32_t pix[WARPS][SW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  if (A.counters[kCtrProgFull]) return;  // programs incomplete: the host reruns the launch
#pragma unroll 1
  while (true) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(&A.counters[kCtrQueue2], 1ull);
    const long long item = (long long)__shfl_sync(0xffffffffu, q, 0);
    if (item >= totalItems) break;
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (runs[mid].row_off <= item) lo = mid;
      else hi = mid - 1;
    }
    const SceneRun& R = runs[lo];
    const int W = (int)R.W, njobs = R.j1 - R.j0;
    const long long ns = (R.W + sliceW - 1) / sliceW;
    const long long local = item - R.row_off;
    const int y = (int)(local / ns);
    const int xs = (int)(local % ns) * sliceW, xe = min(xs + sliceW, W);
    uint32_t* grow = reinterpret_cast<uint32_t*>(R.img) + (long long)y * W;
    const int4* hdr = A.rowhdr + R.ri_base + (long long)y * njobs;
    const uint2* info = A.pinfo + R.j0;
    unsigned painted = 0;  // pixel blends of this item (reported as a launch counter)
#pragma unroll 1
    for (int xa = xs; xa < xe; xa += SW) {
      const int xb = min(xa + SW, xe);
      uint32_t p[PPL];
#pragma unroll
      for (int i = 0; i < PPL; i++) p[i] = xa + i * 32 + lane < xb ? grow[xa + i * 32 + lane] : 0xFF000000u;
      // whether every pixel of the step is opaque: the colour modes leave it so,
      // a mask mode ends it
      bool solid = true;
#pragma unroll
      for (int i = 0; i < PPL; i++) solid &= p[i] >= 0xFF000000u;
      solid = __all_sync(0xffffffffu, solid);
      // 32 paths at a time: each lane loads one path's row header (contiguous
      // over the paths) and colour, then the warp applies them in path order.
      // Rows with more to them than coverage leave the loop, and it is entered
      // again behind them (path `from` of the 32): with their calls inside it,
      // its state went through local memory.
      int c0 = 0, from = 0;
#pragma unroll 1
      while (c0 < njobs) {
        int stop = -1;
        uint2 in = make_uint2(0u, (uint32_t)kNothing << 8);
        int4 h = make_int4(0, 0, 0, 0);
        if (c0 + lane < njobs) {
          in = info[c0 + lane];
          h = hdr[c0 + lane];
        }
        // the first failed path stops the run: it and the paths after it draw nothing
        const int st = (int)(in.y >> 8);
        const unsigned bad = __ballot_sync(0xffffffffu, st != kOk && st != kNothing);
        const int lim = bad ? __ffs(bad) - 1 : 32;
        const bool draws = lane >= from && lane < lim && st == kOk && h.x != 0 && h.z < xb && h.w > xa;
        unsigned dm = __ballot_sync(0xffffffffu, draws);
        // what the warp needs of a path, in two words: the step's pixels it may
        // touch, kind, mode, whether its colour is premultiplied and whether it
        // meets opaque pixels besides (decided for the step and not for each 32
        // pixels, for warps that go through both forms of the blends wait for
        // instructions); and where its coverage would begin at the multiple of 16
        // pixels up to the step's first (16-byte units: rows of coverage begin at
        // such multiples and hold whole units, the bytes past the last pixel 0)
        const int mode0 = (int)(in.y & 255u);
        const bool plain0 = mode0 < kMask && premultiplied(in.x);
        const unsigned masks = __ballot_sync(0xffffffffu, draws && mode0 >= kMask);
        int unit0 = h.y, kind0 = h.x;
        if (draws && kind0 == kRecCov8Z) {
          const int4 g = A.prog[(unsigned)h.y];
          unit0 = g.x;
          if (g.z >= xb || g.w < xa) kind0 = kRecCov8;  // its listed pixels are in other steps
        }
        const uint32_t pack0 = (uint32_t)max(h.z - xa, 0) | ((uint32_t)min(h.w - xa, xb - xa) << 8) |
                               ((uint32_t)kind0 << 16) | ((uint32_t)mode0 << 20) | (plain0 ? 1u << 30 : 0u) |
                               (plain0 && solid && (masks & ((1u << lane) - 1)) == 0 ? 1u << 31 : 0u);
        solid &= masks == 0;
        unit0 += ((xa & ~15) - h.z) >> 4;
        int next = -1;      // the path after the current one, and its coverage
        uint32_t nextCov = 0, nextPack = 0;
#pragma unroll 1
        while (dm || next >= 0) {
          const int cur = next;
          const uint32_t cov = nextCov, pk = nextPack;
          next = -1;
          if (dm) {
            next = __ffs(dm) - 1;
            dm &= dm - 1;
            nextPack = __shfl_sync(0xffffffffu, pack0, next);
            const unsigned unit = (unsigned)__shfl_sync(0xffffffffu, unit0, next);
            const int kind = (int)(nextPack >> 16) & 15, lo = (int)(nextPack & 255u), hi = (int)(nextPack >> 8) & 255;
            const int x = 4 * lane;
            nextCov = 0;
            if (kind == kRecFill) {
              const int b0 = min(max(lo - x, 0), 4), b1 = min(max(hi - x, 0), 4);
              if (b1 > b0) nextCov = (uint32_t)((1ull << (8 * b1)) - (1ull << (8 * b0)));
            } else if (kind != kRecProg && x >= lo && x < hi) {
              const int xu = x + (xa & 15);
              nextCov = *reinterpret_cast<const uint32_t*>(A.cov8 + ((long long)(unit + (xu >> 4)) << 4) + (xu & 15));
            }
          }
          if (cur < 0) continue;
          const uint32_t col = __shfl_sync(0xffffffffu, in.x, cur);
          const int mode = (int)(pk >> 20) & 255;
          // the lanes with coverage, and with nothing but 255: eight lanes' words
          // cover a group of 32 pixels
          unsigned some = __ballot_sync(0xffffffffu, cov != 0), full = __ballot_sync(0xffffffffu, cov == 0xffffffffu);
          painted += __popc((((cov & 0x7f7f7f7fu) + 0x7f7f7f7fu) | cov) & 0x80808080u);  // its bytes above 0
          if (((pk >> 20) & 0x4ffu) == 0x400u) {  // Normal, premultiplied
            if (some) {
#pragma unroll
              for (int i = 0; i < PPL; i++) {
                if (((some >> (8 * i)) & 255u) == 0) continue;
                uint32_t k = 255, s = col;
                if (((full >> (8 * i)) & 255u) != 255u) {
                  k = (__shfl_sync(0xffffffffu, cov, i * 8 + (lane >> 2)) >> (8 * (lane & 3))) & 255u;
                  s = mul_c_flat(col, k);
                }
                p[i] = blend_normal_flat(p[i], s, k != 0);
              }
            }
          } else if (some) {
#pragma unroll 1
            for (int i = 0; i < PPL; i++) {
              uint32_t v = p[0];
              if (some & 255u) {
                const uint32_t k = (__shfl_sync(0xffffffffu, cov, i * 8 + (lane >> 2)) >> (8 * (lane & 3))) & 255u;
                const uint32_t s = (full & 255u) == 255u ? col : mul_c_flat(col, k);
                if (k) v = (int)pk < 0 ? blend_opaque(mode, tbl, v, s) : blend_px(mode, tbl, v, s);
              }
              some >>= 8;
              full >>= 8;
#pragma unroll
              for (int t = 0; t + 1 < PPL; t++) p[t] = p[t + 1];
              p[PPL - 1] = v;
            }
          }
          const int ck = (int)(pk >> 16) & 15;
          if (ck == kRecCov8Z || ck == kRecProg) {
            stop = cur;
            break;
          }
        }
        if (stop < 0) {
          if (bad) break;
          c0 += 32;
          from = 0;
          continue;
        }
        // the general code, on the step's pixels in shared memory
        const int path = c0 + stop;
        from = stop + 1;  // 32: nothing of these paths is left
#pragma unroll
        for (int i = 0; i < PPL; i++) pix[warp][i * 32 + lane] = p[i];
        __syncwarp();
        const int4 ph = hdr[path];
        const uint2 pi = info[path];
        const int pmode = (int)(pi.y & 255u);
        if (ph.x == kRecCov8Z) {  // the listed pixels (no two the same)
          if (lane < A.prog[ph.y].y) {
            const int2 e = reinterpret_cast<const int2*>(A.prog + ph.y + 1)[lane];
            if (e.x >= xa && e.x < xb) {
              ++painted;
              pix[warp][e.x - xa] = blend_any(pmode, tbl, pix[warp][e.x - xa], mul_f(pi.x, __int_as_float(e.y)));
            }
          }
        } else {
          const RowPx<false> row{reinterpret_cast<unsigned char*>(pix[warp]), xa};
          const unsigned drawn = draw_program<SW>(row, pmode, tbl, pi.x, A.prog + ph.y, ph.z, ph.w, y, W, xa, xb,
                                                  accs[warp], lane);
          if (lane == 0) painted += drawn;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < PPL; i++) p[i] = pix[warp][i * 32 + lane];
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i < PPL; i++)
        if (xa + i * 32 + lane < xb) grow[xa + i * 32 + lane] = p[i];
    }
    painted = __reduce_add_sync(0xffffffffu, painted);
    if (lane == 0 && painted) atomicAdd(&A.counters[kCtrPainted], (unsigned long long)painted);
  }
}

// Scene kernels: the general recording code holds 128 crossings per row in
// shared memory (8 warps per CTA).
constexpr int kRecMaxH = 128, kRecWarps = 8, kSceneWarps = 8;
const void* scene_rec_kernel() { return (const void*)k_scene_rec; }
size_t scene_rec_smem() { return sizeof(FastRow<kRecNB, kRecRowXT>) * kRecRowWarps; }
int scene_rec_warps() { return kRecRowWarps; }
// the kernels of wide rows: 0 k_scene_big, 1 k_scene_huge
const void* scene_big_kernel(int v) { return v ? (const void*)k_scene_huge : (const void*)k_scene_big; }
size_t scene_big_smem(int v) { return v ? sizeof(LineRow<kHugeNB, kHugeXT>) : sizeof(FastRow<kBigNB, kBigXT>) * kBigWarps; }
int scene_big_threads(int v) { return (v ? kLineWarps : kBigWarps) * 32; }
int scene_big_rows(int v) { return v ? 1 : kBigWarps; }  // per CTA
void launch_scene_big(int v, unsigned blocks, cudaStream_t st, PathJob* jobs, const Arena& A) {
  launch_pdl(v ? k_scene_huge : k_scene_big, dim3(blocks), dim3(scene_big_threads(v)), scene_big_smem(v), st, jobs, A);
}
const void* scene_rest_kernel() { return (const void*)k_scene_rest<kRecMaxH, kRecWarps>; }
size_t scene_rest_smem() { return sizeof(RowScratch<kRecMaxH, kRecXT>) * kRecWarps; }
int scene_rest_warps() { return kRecWarps; }
const void* scene_kernel(int ppl) {
  return ppl == 1 ? (const void*)k_scene<1, kSceneWarps> : (const void*)k_scene<4, kSceneWarps>;
}
int scene_warps() { return kSceneWarps; }
void launch_scene_rec(unsigned blocks, cudaStream_t st, PathJob* jobs, const RecOrder* order, int njobs,
                      long long items, int rpi, const Arena& A) {
  launch_pdl(k_scene_rec, dim3(blocks), dim3(kRecRowWarps * 32), scene_rec_smem(), st, jobs, order, njobs, items, rpi,
             A);
}
void launch_scene_rest(unsigned blocks, cudaStream_t st, PathJob* jobs, const Arena& A, unsigned char* wide,
                       long long slots) {
  launch_pdl(k_scene_rest<kRecMaxH, kRecWarps>, dim3(blocks), dim3(kRecWarps * 32), scene_rest_smem(), st, jobs, A,
             wide, slots);
}
void launch_scene(int ppl, unsigned blocks, cudaStream_t st, const SceneRun* runs, int nruns, long long items,
                  const Arena& A, const uint8_t* tbl, int sliceW) {
  launch_pdl(ppl == 1 ? k_scene<1, kSceneWarps> : k_scene<4, kSceneWarps>, dim3(blocks), dim3(kSceneWarps * 32), 0, st,
             runs, nruns, items, A, tbl, sliceW);
}

// Dynamic shared memory of k_setup for a launch whose images have at most
// maxBands bands: per band of a window a count, an anti-aliasing flag and a
// place, per warp a count and a lane mask, and the step records.
size_t setup_smem(int maxBands) {
  const int stride = std::min(maxBands, kBandWindow) + 1;
  return (size_t)((3 + 2 * kSetupWarps) * stride) * 4 + kStepBytes;
}
// CTAs per job: the longest job's time shrinks with them, while each CTA of a
// launch beyond the first four per SM costs a wave's fixed part.  In
// microseconds, as measured: 0.014 per unit of work, 15.2 per wave, 4 for the
// cluster's barriers.  One heart: 10 us with 1 CTA, 15
// with 8; 64 cubics: 90 and 38; a 14,540-primitive stroke: 600 and 83; 4096
// glyphs: 100 with 1, 243 with 2; 240 local paths: 970 and 175; 2000 paths over
// 1024 x 1024: 6400 and 2250.
int setup_cluster(long long njobs, long long maxWork, int nsm) {
  const double cta = 15.2 / (4.0 * nsm);
  int best = 1;
  double cost = 0;
  for (int c = 1; c <= 8; c *= 2) {
    const double t = 0.014 * (double)maxWork / c + cta * (double)njobs * c + (c > 1 ? 4.0 : 0.0);
    if (c == 1 || t < cost) {
      best = c;
      cost = t;
    }
  }
  return best;
}
cudaError_t launch_setup(int njobs, int C, int maxBands, cudaStream_t st, PathJob* jobs, const Arena& A) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(njobs * C));
  cfg.blockDim = dim3(kSetupThreads);
  cfg.dynamicSmemBytes = setup_smem(maxBands);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_setup, jobs, A, maxBands, C);
}

size_t scene_wide_bytes() { return sizeof(RowScratch<kWideMaxH, kWideXT>); }

size_t rows_smem_wide() { return sizeof(RowScratch<kWideMaxH, kWideXT>); }

// Whether every row of a job fits one tile of the row engine (which begins up to
// 3 pixels before the row's first: RGBX images).
bool rows_narrow(long long W) { return W + 3 <= kRowsXT; }
const void* rows_lines_kernel(bool narrow) {
  return narrow ? (const void*)k_rows_lines<kNoTiles> : (const void*)k_rows_lines<kOnce>;
}
size_t rows_lines_smem() { return sizeof(LineRow<kRowsNB, kRowsXT>); }
int rows_lines_threads() { return kRowsLineThreads; }
void launch_rows_lines(bool narrow, unsigned blocks, cudaStream_t st, PathJob* jobs, const long long* offs, int njobs,
                       const Arena& A, const uint8_t* tbl, long long items) {
  launch_pdl(narrow ? k_rows_lines<kNoTiles> : k_rows_lines<kOnce>, dim3(blocks), dim3(kRowsLineThreads), rows_lines_smem(), st, jobs, offs, njobs, A, tbl,
             items);
}
const void* rows_huge_kernel(bool narrow) {
  return narrow ? (const void*)k_rows_huge<kNoTiles> : (const void*)k_rows_huge<kOnce>;
}
size_t rows_huge_smem() { return sizeof(LineRow<kWideMaxH, kWideXT>); }
void launch_rows_huge(bool narrow, unsigned blocks, cudaStream_t st, PathJob* jobs, const Arena& A,
                      const uint8_t* tbl) {
  launch_pdl(narrow ? k_rows_huge<kNoTiles> : k_rows_huge<kOnce>, dim3(blocks), dim3(kRowsLineThreads), rows_huge_smem(), st, jobs, A, tbl);
}

// Row kernel variants: 0 = RGBX images, 1 = masks of small paths such as
// glyphs (64 crossings and 256-px tiles, a quarter of the shared memory per
// warp), 2 = the general code, 3 = masks, 4 = RGBX images whose rows fit a tile.
constexpr auto kRowsRgbx = k_rows_fast<kOutRgbx, kRowsNB, kRowsXT, kRowsWarps, kOnce>;
constexpr auto kRowsNarrow = k_rows_fast<kOutRgbx, kRowsNB, kRowsXT, kRowsWarps, kNoTiles>;
constexpr auto kRowsGlyph = k_rows_fast<kOutA8, kGlyphNB, kGlyphXT, kGlyphWarps, kAgain>;
constexpr auto kRowsMask = k_rows_fast<kOutA8, kRowsNB, kRowsXT, kRowsWarps, kOnce>;
constexpr auto kRowsGeneral = k_rows<kFastMaxH, kFastXT, kFastWarps>;
const void* rows_kernel(int v) {
  return v == 0   ? (const void*)kRowsRgbx
         : v == 1 ? (const void*)kRowsGlyph
         : v == 2 ? (const void*)kRowsGeneral
         : v == 3 ? (const void*)kRowsMask
                  : (const void*)kRowsNarrow;
}
size_t rows_smem(int v) {
  return v == 1   ? sizeof(FastRow<kGlyphNB, kGlyphXT>) * kGlyphWarps
         : v == 2 ? sizeof(RowScratch<kFastMaxH, kFastXT>) * kFastWarps
                  : sizeof(FastRow<kRowsNB, kRowsXT>) * kRowsWarps;
}
int rows_warps(int v) { return v == 1 ? kGlyphWarps : v == 2 ? kFastWarps : kRowsWarps; }
// Whether a job's rows can take the row engine (every variant but 2).
bool rows_fast(int mode, long long W) { return mode != kMask && W < fast_max_w(kRowsNB); }
void launch_rows(int v, unsigned blocks, cudaStream_t st, PathJob* jobs, const long long* offs, int njobs,
                 const Arena& A, const uint8_t* tbl, long long items, int rpi) {
  const dim3 b(blocks), t(rows_warps(v) * 32);
  const size_t sm = rows_smem(v);
  if (v == 0) launch_pdl(kRowsRgbx, b, t, sm, st, jobs, offs, njobs, A, tbl, items, rpi);
  else if (v == 1) launch_pdl(kRowsGlyph, b, t, sm, st, jobs, offs, njobs, A, tbl, items, rpi);
  else if (v == 2) launch_pdl(kRowsGeneral, b, t, sm, st, jobs, offs, njobs, A, tbl, items, rpi);
  else if (v == 3) launch_pdl(kRowsMask, b, t, sm, st, jobs, offs, njobs, A, tbl, items, rpi);
  else launch_pdl(kRowsNarrow, b, t, sm, st, jobs, offs, njobs, A, tbl, items, rpi);
}

}  // namespace pxg
