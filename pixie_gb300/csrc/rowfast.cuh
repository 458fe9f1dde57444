// The row engine of the fill kernels: a warp draws (or records) consecutive
// rows of one path with the rows' crossings in shared memory and registers.
//
// What bounds it: instruction fetch, issue and the latency of one warp's chain
// (a band's entry list, divisions, a sort, a walk), not memory.  The general
// row code (process_row) inlines to 140-180 KB per kernel, and its warps, each
// at another place of it, wait for instructions most of the time; unrolled
// sorting networks at 480-810 KB were 4x slower still.  So everything here is
// a rolled loop with one copy of each part.  A sample line's crossings are
// gathered in the row's order (sorted once per row), settled into exact order
// by a few exchange passes, walked 32 at a time with the winding prefix as two
// population counts, and the spans of all the lines added together into a
// 16-bit difference array, whose prefix sum gives the row's coverage.
// Trapezoid rows and filled spans go through the same array, so there is one
// writer.  A band's entries are clipped once for the rows of a chunk (a band
// is 4-7 rows high for all but the tallest shapes).
//
// Measured against process_row (GB300, kernel times): recording 2000 paths on
// 1024 x 1024 (2 M rows) 21.3 -> 6.6 ms, with 1.0 ms for the rows of more than
// 128 crossings; the rows of 4096 glyphs 1.23 -> 0.38 ms; of one 512 x 512
// path of 64 cubics 46 -> 30 us.  The recording kernel's hot code is at the
// instruction cache's edge: 49 KB of it run at 6.6 ms, 54 KB (with the groups
// of cov_samples) at 8.6 ms.
//
// Included by raster.cu after the shared row helpers (make_entry, blends, the
// trapezoid areas).
#pragma once

namespace pxg {

// A sort key is a pixel position in 24.8 fixed point over the crossing's index
// (log2 NB bits) and winding (1 bit): images narrower than fast_max_w(NB).
constexpr int tag_bits(int nb) { return nb <= 64 ? 7 : nb <= 128 ? 8 : nb <= 256 ? 9 : nb <= 512 ? 10 : 12; }
constexpr int fast_max_w(int nb) { return 1 << (24 - tag_bits(nb)); }
static_assert(tag_bits(2048) == 12 && fast_max_w(256) == 32768, "a key holds NB crossings");
constexpr uint32_t kNoKey = 0xffffffffu;
constexpr int kZeroCap = 32;  // pixels of a trapezoid row listed apart: what a byte of coverage cannot say
enum RowOut { kOutRgbx = 0, kOutA8 = 1, kOutRec = 2 };

template <int NB, int XT>
struct __align__(16) FastRow {
  float ent[4][NB];               // the chunk's entries, in segment order: ay, by, m, b
  float key[NB];                  // a sample line's sort keys; midpoints of a trapezoid row
  float t0[NB], t1[NB];           // a trapezoid row's crossings with its top and bottom; else sample spans
  uint32_t diff[(XT + 272) / 2];  // coverage differences, two pixels per word; kDiffZero between rows
  uint16_t idx[NB], perm[NB];     // the row's entries; their order by midpoint
  uint8_t wp[NB];                 // winding +1
  float ends[2][2];               // clipped x of a two-entry band's entries (top, bottom)
  int nzero, zero[kZeroCap];
  __device__ __forceinline__ float& ay(int j) { return ent[0][j]; }
  __device__ __forceinline__ float& by(int j) { return ent[1][j]; }
  __device__ __forceinline__ float& m(int j) { return ent[2][j]; }
  __device__ __forceinline__ float& b(int j) { return ent[3][j]; }
};
// Two signed 16-bit sums per word.  Words add modulo 2^32 in any order, so only a
// pixel's final difference has to fit: a sample line's spans are disjoint and their
// bytes rounded down, a trapezoid row's pixels lie in one edge or span each, so a
// pixel's sum is within 0..511 (256 + 255) and a difference within +-511; one at a
// tile's edge, which takes what lies beyond, is a pixel's sum itself.  The lower
// half begins at 0x4000, so its final value is positive and borrows nothing.
constexpr uint32_t kDiffZero = 0x4000u;

// A loop-invariant value the compiler is not to specialise loops for: a copy
// of a loop per value of a flag doubles the code.
__device__ __forceinline__ int opaque(int v) {
  asm volatile("" : "+r"(v));
  return v;
}
// nim_int(f) limited to [lo, hi] (0 <= lo <= hi < 2^23): NaN and values
// outside int64 count as its minimum.
__device__ __forceinline__ int nim_clamp(float f, int lo, int hi) {
  if (!(f < 9223372036854775808.0f)) return lo;
  return min(max((int)fminf(fmaxf(f, -1.0f), 8388608.0f), lo), hi);
}
// nim_int(f) as a float, for comparisons of such values
__device__ __forceinline__ float nim_trunc(float f) {
  return f >= -9223372036854775808.0f && f < 9223372036854775808.0f ? truncf(f) : -9223372036854775808.0f;
}

// The sort keys of a sample line, K per lane in lane order (element lane * K +
// k), so that most exchanges of the networks below stay within a lane.
template <int K>
__device__ __forceinline__ void load_keys(const uint32_t* keys, uint32_t (&v)[K], int lane) {
  if (K == 2) {
    const uint2 q = reinterpret_cast<const uint2*>(keys)[lane];
    v[0] = q.x;
    v[1] = q.y;
  } else {
#pragma unroll
    for (int k = 0; k < K; k += 4) {
      const uint4 q = reinterpret_cast<const uint4*>(keys)[(lane * K + k) >> 2];
      v[k] = q.x;
      v[k + 1] = q.y;
      v[(k + 2) % K] = q.z;
      v[(k + 3) % K] = q.w;
    }
  }
}
template <int K>
__device__ __forceinline__ void store_keys(uint32_t* keys, const uint32_t (&v)[K], int lane) {
  if (K == 2) {
    reinterpret_cast<uint2*>(keys)[lane] = make_uint2(v[0], v[1]);
  } else {
#pragma unroll
    for (int k = 0; k < K; k += 4)
      reinterpret_cast<uint4*>(keys)[(lane * K + k) >> 2] = make_uint4(v[k], v[k + 1], v[(k + 2) % K], v[(k + 3) % K]);
  }
}
__device__ __forceinline__ void cmp_swap(uint32_t& a, uint32_t& b) {
  const uint32_t t = min(a, b);
  b = max(a, b);
  a = t;
}
// Sorts 32 K keys ascending: a bitonic network (descending runs are sorted
// complemented, so every exchange within a lane is a min and a max), stages
// for sizes that hold no more than padding past the first n skipped.
template <int K>
__device__ __forceinline__ void bitonic_keys(uint32_t (&v)[K], int n, int lane) {
#pragma unroll 1
  for (int size = 2; size < 2 * n; size <<= 1) {
    const uint32_t flip = size >= K && ((lane * K) & size) ? 0xffffffffu : 0u;
    if (size >= K) {
#pragma unroll
      for (int k = 0; k < K; k++) v[k] ^= flip;
#pragma unroll 1
      for (int d = size >> 1; d >= K; d >>= 1) {
        const bool mx = ((lane * K) & d) != 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v[k], d / K);
          v[k] = mx ? max(v[k], o) : min(v[k], o);
        }
      }
#pragma unroll
      for (int d = K / 2; d >= 1; d >>= 1)
#pragma unroll
        for (int k = 0; k < K; k++)
          if (!(k & d)) cmp_swap(v[k], v[k | d]);
#pragma unroll
      for (int k = 0; k < K; k++) v[k] ^= flip;
    } else {  // runs within a lane, alternating directions
#pragma unroll
      for (int s = 2; s < K; s <<= 1) {
        if (size != s) continue;
#pragma unroll
        for (int d = s / 2; d >= 1; d >>= 1)
#pragma unroll
          for (int k = 0; k < K; k++)
            if (!(k & d)) {
              if (k & s) cmp_swap(v[k | d], v[k]);
              else cmp_swap(v[k], v[k | d]);
            }
      }
    }
  }
}
// Sorts the 32 K keys (n of them valid).  Unless they are in no known order
// (fresh), passes of odd-even transposition until nothing moves; the bitonic
// network when that takes more than a few.
template <int K>
__device__ __forceinline__ void sort_keys(uint32_t* keys, int n, bool fresh, int lane) {
  uint32_t v[K];
  load_keys<K>(keys, v, lane);
  bool done = false;
#pragma unroll 1
  for (int pass = fresh ? 6 : 0; pass < 6; pass++) {
    bool moved = false;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int k = p; k + 1 < K; k += 2) {
        moved |= v[k] > v[k + 1];
        cmp_swap(v[k], v[k + 1]);
      }
    const uint32_t up = __shfl_down_sync(0xffffffffu, v[0], 1), dn = __shfl_up_sync(0xffffffffu, v[K - 1], 1);
    moved |= lane < 31 && v[K - 1] > up;
    if (lane > 0) v[0] = max(v[0], dn);
    if (lane < 31) v[K - 1] = min(v[K - 1], up);
    if (!__any_sync(0xffffffffu, moved)) {
      done = true;
      break;
    }
  }
  if (!done) bitonic_keys<K>(v, n, lane);
  store_keys<K>(keys, v, lane);
}

// The same in shared memory, for more keys than registers hold.
__device__ __forceinline__ void sort_keys_shared(uint32_t* keys, int n, bool fresh, int lane) {
  bool done = false;
#pragma unroll 1
  for (int pass = fresh ? 12 : 0; pass < 12; pass++) {  // even, then odd pairs
    bool moved = false;
#pragma unroll 1
    for (int i = 2 * lane + (pass & 1); i + 1 < n; i += 64) {
      const uint32_t a = keys[i], b = keys[i + 1];
      if (a > b) {
        keys[i] = b;
        keys[i + 1] = a;
        moved = true;
      }
    }
    __syncwarp();
    if (!__any_sync(0xffffffffu, moved)) {
      if (done) return;  // neither parity moved
      done = true;
    } else {
      done = false;
    }
  }
#pragma unroll 1
  for (int size = 2; size < 2 * n; size <<= 1)
#pragma unroll 1
    for (int d = size >> 1; d >= 1; d >>= 1) {
      // a reversed first exchange per merge keeps every run ascending, so
      // elements past n (larger than all) never move and need no storage
      const bool first = d == size >> 1;
#pragma unroll 1
      for (int p = lane; p < n; p += 32) {
        const int i = (p / d) * 2 * d + p % d, o = first ? i ^ (size - 1) : i + d;
        if (o < n) {
          const uint32_t a = keys[i], b = keys[o];
          if (a > b) {
            keys[i] = b;
            keys[o] = a;
          }
        }
      }
      __syncwarp();
    }
}

// Where the coverage of a row goes: pixels [t0, t1), difference index i at
// pixel x0 + i.  lo/hi: the pixels touched so far (per lane).
struct CovTile {
  int x0, t0, t1, lo, hi;
};

// diff[x] += v: contributions left of the tile carry into its first pixel,
// those right of it end at its last.
__device__ __forceinline__ void cov_add(uint32_t* diff, const CovTile& T, int x, int v) {
  const int i = min(max(x, T.t0), T.t1) - T.x0;
  atomicAdd(&diff[i >> 1], (uint32_t)v << ((i & 1) << 4));
}
// pixels [a, b) += v
__device__ __forceinline__ void cov_range(uint32_t* diff, const CovTile& T, int a, int b, int v) {
#pragma unroll 1
  for (int s = 0; s < 2; s++) {
    cov_add(diff, T, s ? b : a, v);
    v = -v;
  }
}
// One sample span (prevAt, at) of computeCoverage (paths.nim:1398-1431) in
// 24.8 fixed point: coverage 51 per sample (255 / 5) with anti-aliasing, else
// the pixels [prevAt / 256, at / 256) of a fillHits span at 255.  SKIP: spans
// outside the tile, whose differences cancel at its edge, are left out.
template <bool SKIP>
__device__ __forceinline__ void cov_span(uint32_t* diff, CovTile& T, int prevAt, int at, bool aa) {
  const int pi = prevAt >> 8, ai = at >> 8;
  if (SKIP && (ai < T.t0 || pi >= T.t1)) return;
  // differences at pi, pi + 1, ai, ai + 1; one pixel's span lies within it
  int d0, d1, d2 = 0, d3 = 0;
  if (!aa) {
    if (ai <= pi) return;
    d0 = 255;
    d1 = 0;
    d2 = -255;
  } else if (ai == pi) {
    d0 = ((at - prevAt) * 51) >> 8;
    d1 = -d0;
  } else {
    d0 = ((256 - (prevAt & 255)) * 51) >> 8;
    d1 = 51 - d0;
    d3 = -(((at & 255) * 51) >> 8);
    d2 = -d3 - 51;
  }
  T.lo = min(T.lo, pi);
  T.hi = max(T.hi, ai + 1);
  int x = pi;
#pragma unroll 1
  for (int s = 0; s < 4; s++) {
    if (d0) cov_add(diff, T, x, d0);
    x = s == 1 ? ai : x + 1;
    d0 = d1;
    d1 = d2;
    d2 = d3;
    d3 = 0;
  }
}

// 32 crossings of computeCoverage's walk over a sample line's nh sorted ones
// (paths.nim:1298-1334), for one line or for several with a group of lanes
// each; the spans it draws are appended to sp.  A crossing's
// winding count is the number of +1 minus -1 crossings before it.  What the
// walk does at one position -- draws a span up to it, only moves prevAt
// there, or neither -- is decided by the first of its crossings that does
// either (a second span there would be empty), which the lane of the
// position's first crossing finds: crossings that cancel their successor are
// skipped with it, and a nonzero count that stays nonzero does nothing.
// i: the lane's crossing (keys[i]; none at or past nh); group: the lanes of the
// same line; count and prevAt: the walk's before them, moved past them unless
// the line ends with them.
template <int TAG>
__device__ __forceinline__ void walk_step(const uint32_t* keys, int i, int nh, unsigned group, bool last, int& count,
                                          int& prevAt, int winding, int2* sp, int& ns, int lane) {
  const unsigned lt = (1u << lane) - 1, before = lt & group;
  const bool valid = i < nh;
  uint32_t key = valid ? keys[i] : kNoKey;
  const uint32_t prev = valid && i > 0 ? keys[i - 1] : kNoKey;
  const int at = (int)(key >> TAG);
  const unsigned V = __ballot_sync(0xffffffffu, valid), P = __ballot_sync(0xffffffffu, valid && (key & 1));
  int c = count + 2 * __popc(P & before) - __popc(V & before);
  bool span = false, upd = false;
  const bool nonzero = opaque(winding) == 0;
  if (valid && at > 0 && ((key ^ prev) >> TAG) != 0) {
#pragma unroll 1
    while (true) {
      if ((nonzero ? c : c & 1) == 0) {
        upd = true;
        break;
      }
      const uint32_t nx = i + 1 < nh ? keys[i + 1] : kNoKey;
      const int w = (key & 1) ? 1 : -1;
      if (((key ^ nx) >> TAG) == 0 && ((key ^ nx) & 1)) {
        i += 2;
        key = i < nh ? keys[i] : kNoKey;
      } else if (nonzero && i < nh - 1 && c + w != 0) {
        c += w;
        i++;
        key = nx;
      } else {
        span = upd = true;
        break;
      }
      if ((int)(key >> TAG) != at) break;
    }
  }
  const unsigned um = __ballot_sync(0xffffffffu, upd), below = um & before;
  const unsigned em = __ballot_sync(0xffffffffu, span);
  const int pa = __shfl_sync(0xffffffffu, at, below ? 31 - __clz(below) : lane);
  if (span) sp[ns + __popc(em & lt)] = make_int2(below ? pa : prevAt, at);
  ns += __popc(em);
  if (!last) {
    count += 2 * __popc(P) - __popc(V);
    const int moved = __shfl_sync(0xffffffffu, at, um ? 31 - __clz(um) : 0);
    if (um) prevAt = moved;
  }
}

// A line's key for the row's entry e (the chunk's j): where it crosses yLine,
// over its place among equals and its winding.
template <int TAG, int NB, int XT>
__device__ __forceinline__ uint32_t crossing_key(FastRow<NB, XT>& S, int j, int e, float yLine, float Wf) {
  const float m = S.m(j), b = S.b(j);
  const float x = m == 0 ? b : (yLine - b) / m;
  const int fx = nim_i32(nmin(x, Wf) * 256.0f);
  // crossings at or left of 0 only add to the winding count, in any order
  return ((uint32_t)max(fx, 0) << TAG) | ((uint32_t)e << 1) | S.wp[j];
}
// The sample lines of row y (:1350-1397): the row's n entries (S.idx) against
// each line, sorted, walked, accumulated into S.diff over the tile T.
// Up to kGroupN entries -- most rows of drawn shapes have 2 to 8 -- the lanes
// take as many lines at once as fit, a group of n lanes each, and a crossing's
// rank is counted (GROUPED; the recording kernel is faster without the code).
// With more, the entries are ordered once by where they cross the middle of the
// row (or end nearest to it); a line's crossings, gathered in that order, are
// then nearly sorted.  Only the exact sort of a line's own keys decides.
// held: the row's spans left by the call for its first tile, which those for the
// others take as they are; -1 before that, and where they were too many.  A
// stroke of 300 points on 16384 x 512, 16 tiles a row, takes 1080 us with lines
// and trapezoids gone through for each, 348 so.
constexpr int kGroupN = 16;
// Rows in several tiles: none (the images are narrower than one), or gone through
// again for each (recording, whose code is at the instruction cache's edge, and
// glyphs, seldom so wide), or worked out once.  A call on 60000 rows of 16 pixels
// takes 134 us with the code for none, 152 with that for the last.
enum Tiles { kNoTiles = 0, kAgain = 1, kOnce = 2 };
template <bool GROUPED, bool HOLD, int NB, int XT>
__device__ __forceinline__ void cov_samples(FastRow<NB, XT>& S, int n, int y, float Wf, int winding, bool aa,
                                            CovTile& T, int lane, int& held) {
  constexpr int TAG = tag_bits(NB);
  const unsigned lt = (1u << lane) - 1;
  uint32_t* keys = reinterpret_cast<uint32_t*>(S.key);
  int2* sp = reinterpret_cast<int2*>(S.t0);
  const int lines = aa ? 5 : 1;
  const float offset = aa ? 1.0f / 5.0f : 1.0f;
  const float initialOffset = offset / 2 + kEps;
  float yLine = (float)y + initialOffset - offset;
  const bool grouped = GROUPED && n <= kGroupN;
  const int sets = grouped ? 32 / n : 1;
  // the lane's place: line s of a step, entry i of its group, keys from kb on
  const int s = grouped ? lane / n : 0, kb = s * n, i = lane - kb;
  const unsigned group = grouped ? ((1u << n) - 1) << kb : 0xffffffffu;
  static_assert(NB <= 512, "a line's keys are sorted in registers");
  const int cap = NB <= 64 || n <= 64 ? 64 : NB;
  int ns = 0, done = grouped ? 0 : -1;  // lines done (-1: the ordering is to come)
  bool all = true;                            // every span so far is still there
  if (HOLD && held >= 0) {
    ns = held;
    done = lines;
  }
  const auto draw = [&]() {
#pragma unroll 1
    for (int k = lane; k < ns; k += 32) cov_span<HOLD>(S.diff, T, sp[k].x, sp[k].y, opaque(aa) != 0);
    __syncwarp();
  };
  if (grouped) {                        // the first step's lines are s ahead
#pragma unroll 1
    for (int k = 0; k < min(s, lines); k++) yLine += offset;
  }
#pragma unroll 1
  while (HOLD || done < lines) {
    if (HOLD && (ns > NB - max(n / 2, 16) || done >= lines)) {  // a step has at most n / 2 spans (16 by groups)
      draw();
      if (done >= lines) break;
      ns = 0;
      all = false;
    }
    const bool ordering = !grouped && opaque(done) < 0;
    int nh = 0;  // the crossings of the lane's line
    if (!ordering) yLine += offset;
    if (grouped) {
      const int j = S.idx[i];
      const bool hit = s < sets && done + s < lines && S.ay(j) <= yLine && S.by(j) >= yLine;
      const uint32_t key = hit ? crossing_key<TAG>(S, j, i, yLine, Wf) : kNoKey;
      int rank = 0;
#pragma unroll 1
      for (int d = 1, o = i + 1; d < n; d++, o++) {
        if (o == n) o = 0;
        rank += __shfl_sync(0xffffffffu, key, kb + o) < key;
      }
      nh = __popc(__ballot_sync(0xffffffffu, hit) & group);
      if (hit) keys[kb + rank] = key;
      // the lane's next line is `sets` further on: sets - 1 of them here
#pragma unroll 1
      for (int k = 1; k < sets && done + sets < lines; k++) yLine += offset;
    } else {
#pragma unroll 1
      for (int e0 = 0; e0 < n; e0 += 32) {
        const int at = min(e0 + lane, n - 1), e = ordering ? at : S.perm[at], j = S.idx[e];
        const float ay = S.ay(j), by = S.by(j);
        const float yl = ordering ? fminf(fmaxf((float)y + 0.5f, ay), by) : yLine;
        const bool hit = e0 + lane < n && (ordering || (ay <= yl && by >= yl));
        const unsigned msk = __ballot_sync(0xffffffffu, hit);
        if (hit) keys[nh + __popc(msk & lt)] = crossing_key<TAG>(S, j, e, yl, Wf);
        nh += __popc(msk);
      }
#pragma unroll 1
      for (int k = nh + lane; k < cap; k += 32) keys[k] = kNoKey;
      __syncwarp();
      if (cap == 64) sort_keys<2>(keys, nh, ordering, lane);
      else sort_keys<NB / 32>(keys, nh, ordering, lane);
    }
    __syncwarp();
    if (ordering) {
#pragma unroll 1
      for (int k = lane; k < nh; k += 32) S.perm[k] = (uint16_t)((keys[k] >> 1) & ((1u << (TAG - 1)) - 1));
    } else {
      int count = 0, prevAt = 0;  // after the 32 crossings before
#pragma unroll 1
      for (int c0 = 0; c0 < (grouped ? 1 : nh); c0 += 32)
        walk_step<TAG>(keys + kb, c0 + i, nh, group, grouped, count, prevAt, winding, sp, ns, lane);
    }
    __syncwarp();
    done += sets;
    if (!HOLD && (ns > NB / 2 || done >= lines)) {  // a line has at most NB / 2 spans, and there is room for NB
      draw();
      ns = 0;
    }
  }
  if (HOLD) held = all ? ns : -1;
}

// Rows whose time on one warp is what a launch waits for: a warp per sample
// line.  The row's warp (0) orders the entries and publishes the row; warps
// 1 .. 4 take the other lines with keys and spans of their own, all into the
// row's difference array.
constexpr int kLineWarps = 5;
template <int NB>
struct __align__(16) LineScratch {
  uint32_t keys[NB];
  int2 spans[NB / 2 + 32];
  int ns;  // spans of the row's last tile: the same for its others
};
struct LineWork {  // what warp 0 publishes (n < 0: no more rows), and the warps' touched pixels
  int n, y, winding, lines, x0, t0, t1, held;
  float Wf;
  int lo[kLineWarps], hi[kLineWarps];
};
template <int NB, int XT>
struct LineRow {  // a CTA's row
  FastRow<NB, XT> row;
  LineScratch<NB> line[kLineWarps];
  LineWork work;
};
__device__ __forceinline__ void line_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kLineWarps * 32) : "memory"); }

template <int K>
__device__ __forceinline__ void sort_padded(uint32_t* keys, int n, bool fresh, int lane) {
#pragma unroll 1
  for (int k = n + lane; k < 32 * K; k += 32) keys[k] = kNoKey;
  __syncwarp();
  sort_keys<K>(keys, n, fresh, lane);
}
// n keys of up to NB, in the registers of the warp where they fit.
template <int NB>
static __device__ __noinline__ void sort_line(uint32_t* keys, int n, bool fresh, int lane) {
  if (NB <= 256 && n <= 64) sort_padded<2>(keys, n, fresh, lane);
  else if (n <= (NB < 1024 ? NB : 1024)) sort_padded<(NB < 1024 ? NB : 1024) / 32>(keys, n, fresh, lane);
  else sort_keys_shared(keys, n, fresh, lane);
  __syncwarp();
}

template <bool SKIP, int NB, int XT>
__device__ __forceinline__ void one_line(FastRow<NB, XT>& S, LineWork& L, LineScratch<NB>& K, int q, int lane) {
  constexpr int TAG = tag_bits(NB);
  const unsigned lt = (1u << lane) - 1;
  CovTile T{L.x0, L.t0, L.t1, INT_MAX, INT_MIN};
  const int n = L.n;
  const bool aa = L.lines == 5;
  if (q < L.lines && !L.held) {
    const float offset = aa ? 1.0f / 5.0f : 1.0f;
    const float initialOffset = offset / 2 + kEps;
    float yLine = (float)L.y + initialOffset - offset;
#pragma unroll 1
    for (int k = 0; k <= q; k++) yLine += offset;
    int nh = 0;
#pragma unroll 1
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = S.perm[min(e0 + lane, n - 1)], j = S.idx[e];
      const bool hit = e0 + lane < n && S.ay(j) <= yLine && S.by(j) >= yLine;
      const unsigned msk = __ballot_sync(0xffffffffu, hit);
      if (hit) K.keys[nh + __popc(msk & lt)] = crossing_key<TAG>(S, j, e, yLine, L.Wf);
      nh += __popc(msk);
    }
    __syncwarp();
    sort_line<NB>(K.keys, nh, false, lane);
    int count = 0, prevAt = 0, ns = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < nh; c0 += 32)
      walk_step<TAG>(K.keys, c0 + lane, nh, 0xffffffffu, false, count, prevAt, L.winding, K.spans, ns, lane);
    if (lane == 0) K.ns = ns;
    __syncwarp();
  }
  if (q < L.lines) {
#pragma unroll 1
    for (int k = lane; k < K.ns; k += 32) cov_span<SKIP>(S.diff, T, K.spans[k].x, K.spans[k].y, opaque(aa) != 0);
  }
  const int lo = __reduce_min_sync(0xffffffffu, T.lo), hi = __reduce_max_sync(0xffffffffu, T.hi);
  if (lane == 0) {
    L.lo[q] = lo;
    L.hi[q] = hi;
  }
}
// cov_samples by kLineWarps warps (called by warp 0; a line's spans always fit).
template <bool SKIP, int NB, int XT>
__device__ __forceinline__ void cov_lines(FastRow<NB, XT>& S, LineWork& L, LineScratch<NB>& K, int n, int y, float Wf,
                                          int winding, bool aa, CovTile& T, int lane, int& held) {
  constexpr int TAG = tag_bits(NB);
  if (held < 0) {
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      const int j = S.idx[i];
      K.keys[i] = crossing_key<TAG>(S, j, i, fminf(fmaxf((float)y + 0.5f, S.ay(j)), S.by(j)), Wf);
    }
    __syncwarp();
    sort_line<NB>(K.keys, n, true, lane);
#pragma unroll 1
    for (int i = lane; i < n; i += 32) S.perm[i] = (uint16_t)((K.keys[i] >> 1) & ((1u << (TAG - 1)) - 1));
  }
  if (lane == 0) {
    L.held = held >= 0;
    L.n = n;
    L.y = y;
    L.winding = winding;
    L.lines = aa ? 5 : 1;
    L.x0 = T.x0;
    L.t0 = T.t0;
    L.t1 = T.t1;
    L.Wf = Wf;
  }
  held = 0;
  line_barrier();
  one_line<SKIP>(S, L, K, 0, lane);
  line_barrier();
#pragma unroll 1
  for (int q = 0; q < kLineWarps; q++) {
    T.lo = min(T.lo, L.lo[q]);
    T.hi = max(T.hi, L.hi[q]);
  }
}

__device__ __forceinline__ int warp_scan_incl(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}
// Takes the difference array from index i0 (a multiple of 8) through iEnd,
// leaving it at zero, 2 N pixels (N = 2 or 4 words) per lane: out(i, f) gets the
// prefix sums of indices i .. i + 2 N - 1, two per word.  A word's two prefix
// sums are w + (w << 16), the sum before it is added to both halves at once;
// the sums themselves are not negative, so the halves come out exact.  SPARSE:
// steps of pixels that nothing covers are passed over (a wide row of a stroke is
// mostly those).
template <int N, bool SPARSE, class Out>
__device__ __forceinline__ void flush_diff(uint32_t* diff, int i0, int iEnd, int lane, Out&& out) {
  int carry = 0;
#pragma unroll 1
  for (int i = i0; i <= iEnd; i += 64 * N) {
    const int ii = i + lane * 2 * N;
    uint32_t w[N];
    if (SPARSE && N == 2 && carry == 0) {
      const uint2 q = *reinterpret_cast<const uint2*>(diff + (ii >> 1));
      if (!__any_sync(0xffffffffu, q.x != kDiffZero || q.y != kDiffZero)) continue;
    }
    if (N == 4) {
      uint4* p = reinterpret_cast<uint4*>(diff + (ii >> 1));
      const uint4 q = *p;
      *p = make_uint4(kDiffZero, kDiffZero, kDiffZero, kDiffZero);
      w[0] = q.x;
      w[1] = q.y;
      w[N - 2] = q.z;
      w[N - 1] = q.w;
    } else {
      uint2* p = reinterpret_cast<uint2*>(diff + (ii >> 1));
      const uint2 q = *p;
      *p = make_uint2(kDiffZero, kDiffZero);
      w[0] = q.x;
      w[1] = q.y;
    }
    int sum[N];  // through word k
#pragma unroll
    for (int k = 0; k < N; k++) {
      sum[k] = ((int)w[k] >> 16) + (int)(w[k] & 0xffffu) - (int)kDiffZero + (k ? sum[k - 1] : 0);
      w[k] -= kDiffZero;
      w[k] += w[k] << 16;
    }
    const int incl = warp_scan_incl(sum[N - 1], lane);
    const int base = carry + incl - sum[N - 1];
    carry += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
    for (int k = 0; k < N; k++) w[k] += (uint32_t)(base + (k ? sum[k - 1] : 0)) * 0x00010001u;
    out(ii, w);
  }
  __syncwarp();
}
// the low bytes of four prefix sums
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x6420); }

// Loads the entries of a band that overlap the rows [c0, c1) into S, in segment
// order; returns their number, or -1 when they exceed NB.  A band of exactly two entries that
// are two non-intersecting spanning edges (:1250-1262) sets two and orders them
// left to right.
template <int NB, int XT>
__device__ __forceinline__ int load_chunk(const PathJob& J, const Arena& A, const Band& bd, float top, float bottom,
                                          float c0, float c1, FastRow<NB, XT>& S, int lane, bool& two) {
  const float4* SG = A.segs + J.seg_off;
  const int* SW = A.segw + J.seg_off;
  const int* BL = A.bandseg + bd.off;
  const unsigned lt = (1u << lane) - 1;
  const int nb = bd.count;
  int n = 0;
#pragma unroll 1
  for (int j0 = 0; j0 < nb; j0 += 32) {
    const int j = j0 + lane;
    bool pred = false;
    Entry e;
    if (j < nb) {
      const int i = BL[j];
      e = make_entry(SG[i], SW[i], top, bottom);
      pred = opaque(nb) == 2 || !(e.by <= c0 || e.ay >= c1);
    }
    const unsigned msk = __ballot_sync(0xffffffffu, pred);
    const int p = n + __popc(msk & lt);
    if (pred && p < NB) {
      S.ay(p) = e.ay;
      S.by(p) = e.by;
      S.m(p) = e.m;
      S.b(p) = e.b;
      S.wp[p] = e.w > 0;
      if (p < 2) {
        S.ends[p][0] = e.ax;
        S.ends[p][1] = e.bx;
      }
    }
    n += __popc(msk);
  }
  __syncwarp();
  two = false;
  if (n > NB) return -1;
  if (nb == 2) {
    const V2 a0{S.ends[0][0], S.ay(0)}, b0{S.ends[0][1], S.by(0)}, a1{S.ends[1][0], S.ay(1)}, b1{S.ends[1][1], S.by(1)};
    two = !intersectsInside(a0, b0, a1, b1) && a0.y <= top && b0.y >= bottom && a1.y <= top && b1.y >= bottom;
    if (two && (a0.x + b0.x) * 0.5f > (a1.x + b1.x) * 0.5f) {
      const int p = lane & 1;
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = S.ent[k][p];
      const uint8_t t = S.wp[p];
      const float x = S.ends[p][0];
      __syncwarp();
      if (lane < 2) {
#pragma unroll
        for (int k = 0; k < 4; k++) S.ent[k][1 - p] = v[k];
        S.wp[1 - p] = t;
        S.ends[1 - p][0] = x;
      }
      __syncwarp();
    }
  }
  return n;
}

// Hands row y of the job on, to list 0, 1 or 2 (which a later kernel takes): more
// crossings than this instance holds, or a coverage arena that ran out.
__device__ __forceinline__ void push_row(const Arena& A, int job, int y, int lane, int list = 0) {
  if (lane == 0) {
    const unsigned long long slot = atomicAdd(&A.counters[list == 0 ? kCtrOvfRows : list == 1 ? kCtrOvfRows2 : kCtrOvfRows3], 1ull);
    if ((long long)slot < A.ovf_cap) A.ovf_rows[list * A.ovf_cap + slot] = ((long long)job << 32) | y;
  }
}

__device__ __forceinline__ float entry_x(float m, float b, float y) {  // solveX :1137-1141
  return m == 0 ? b : (y - b) / m;
}

// The trapezoid test of a row whose n entries all span it (:1695-1750): their
// crossings with its top and bottom in S.t0/t1, their order by midpoint in
// S.perm; whether they form simple pairs.  ordered: every position is exact as
// an integer's floor and ceiling, so simple pairs lie one behind the other.
template <bool ORDERED, int NB, int XT>
__device__ __forceinline__ bool trap_row(FastRow<NB, XT>& S, int n, float yTop, float yBottom, int winding, int lane,
                                         bool& ordered) {
  const unsigned le = 0xffffffffu >> (31 - lane);
  bool nan = false, far = false;
#pragma unroll 1
  for (int i = lane; i < n; i += 32) {
    const int j = S.idx[i];
    const float m = S.m(j), b = S.b(j);
    const float t0 = entry_x(m, b, yTop), t1 = entry_x(m, b, yBottom), key = (t0 + t1) * 0.5f;
    S.t0[i] = t0;
    S.t1[i] = t1;
    S.key[i] = key;
    nan |= isnan(key);
    if (ORDERED) far |= !(fabsf(t0) < 1e18f && fabsf(t1) < 1e18f);
  }
  if (ORDERED) ordered = !__any_sync(0xffffffffu, far);
  nan = __any_sync(0xffffffffu, nan);
  __syncwarp();
  if (!nan) {
#pragma unroll 1
    for (int i = lane; i < n; i += 32) S.perm[stable_rank_f(S.key, n, i)] = (uint16_t)i;
  } else if (lane == 0) {  // NaN compares false: the reference's insertion sort itself (:1710-1719)
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      const float kv = S.key[i];
      int j = i - 1;
#pragma unroll 1
      for (; j >= 0 && S.key[j] > kv; j--) {
        S.key[j + 1] = S.key[j];
        S.perm[j + 1] = S.perm[j];
      }
      S.key[j + 1] = kv;
      S.perm[j + 1] = (uint16_t)i;
    }
  }
  __syncwarp();
  bool bad = false;
  int carry = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const bool valid = i < n;
    const int j = S.perm[min(i, n - 1)], q = S.perm[min(i + 1, n - 1)];
    // partial coverage of neighbours must not overlap (:1721-1731)
    if (i + 1 < n) bad |= nim_trunc(ceilf(nmax(S.t0[j], S.t1[j]))) > nim_trunc(nmin(S.t0[q], S.t1[q]));
    // and pairs must be simple fills (:1733-1750)
    const bool up = S.wp[S.idx[j]] != 0;
    const unsigned P = __ballot_sync(0xffffffffu, valid && up);
    const unsigned N = __ballot_sync(0xffffffffu, valid && !up);
    const int count = carry + __popc(P & le) - __popc(N & le);  // after this entry
    if (valid) bad |= ((opaque(winding) == 0 ? count : count & 1) != 0) != ((i & 1) == 0);
    carry += __popc(P) - __popc(N);
  }
  return !__any_sync(0xffffffffu, bad);
}

// The pixels of a simple trapezoid row (:1752-1835) over tile T into S.diff:
// 256 + the multiplier (0..255) its area rounds to, so that pixels blended
// with nothing stay distinct from untouched ones (listed in S.zero, their area in
// S.key, free by now, when ZERO, where only the multiplier is kept).  Returns
// true where a multiplier is above 255, which list_odd lists, or the list is
// full: the general code's.  dry: no more than that.
// from: the first entry that reaches the tile or those to its right (advanced
// where the entries are ordered: of 200 a row's 16 tiles have a dozen each).
template <bool ZERO, bool ORDERED, int NB, int XT>
__device__ __forceinline__ bool trap_cov(FastRow<NB, XT>& S, int n, int y, const CovTile& T, int lane, bool dry,
                                         bool ordered, int& from) {
  constexpr int kBase = ZERO ? 0 : 256;
  bool odd = false;
#pragma unroll 1
  for (int s = ORDERED ? from : 0; s < n; s++) {
    const int i = S.perm[s], j = S.idx[i];
    const float m = S.m(j), b = S.b(j), t0 = S.t0[i], t1 = S.t1[i];
    const float lo = nmin(t0, t1), end = ceilf(nmax(t0, t1));
    if (ORDERED && ordered && !dry) {
      if (!(s & 1) && lo >= (float)T.t1) break;
      if ((s & 1) && end <= (float)T.t1) from = s + 1;
    }
    const long long xs = nim_int(lo);
    const int x1 = nim_clamp(end, T.t0, T.t1);
#pragma unroll 1
    for (int x = nim_clamp(lo, T.t0, T.t1) + lane; x < x1; x += 32) {
      const float area = (s & 1) ? trap_right_area(m, b, t0, t1, x, xs, y) : trap_left_area(m, b, t0, t1, x, xs, y);
      const uint32_t v = area == 0.0f ? 0u : nim_u32(roundf(area * 255.0f));
      if (v > 255) odd = true;
      else if (!ZERO && dry) continue;
      else if (!ZERO || v) cov_range(S.diff, T, x, x + 1, kBase + (int)v);
      else {
        const int z = atomicAdd(&S.nzero, 1);
        if (z < kZeroCap) {
          S.zero[z] = x;
          S.key[z] = 0.0f;
        } else {
          odd = true;
        }
      }
    }
    if (!(s & 1) && lane == 0 && !(!ZERO && dry)) {  // the fully covered middle up to the next edge
      const int r = S.perm[s + 1];
      const int fe = nim_clamp(nmin(S.t0[r], S.t1[r]), T.t0, T.t1);
      if (fe > x1) cov_range(S.diff, T, x1, fe, kBase + 255);
    }
  }
  return __any_sync(0xffffffffu, odd) != 0;
}

// Lists the pixels of [dl, dh) whose multipliers are above 255, with their areas,
// in S.zero and S.key; true if there is no room for them.  Where an edge crosses
// the image's left side between pixels -1 and 0, pixel 0 has an area above 1, so
// a shape that leaves the image there has such a pixel in many of its rows; as
// rows handed on they cost a wait for the host or three kernels: 1000 edges on
// 1500 x 1000 222 us, 120 so, 200 of them in a scene 10.99 ms and 1.48.  Out of
// line, and a walk of its own: a list made in trap_cov took a fifth of the time of
// rows that have none (50 lines on 2000 x 1500 96 us, 123).
template <int NB, int XT>
static __device__ __noinline__ bool list_odd(FastRow<NB, XT>* S, int n, int y, int dl, int dh, bool fresh, int lane) {
  __syncwarp();
  if (fresh && lane == 0) S->nzero = 0;
  __syncwarp();
#pragma unroll 1
  for (int s = 0; s < n; s++) {
    const int i = S->perm[s], j = S->idx[i];
    const float m = S->m(j), b = S->b(j), t0 = S->t0[i], t1 = S->t1[i], lo = nmin(t0, t1);
    const long long xs = nim_int(lo);
    const int x1 = nim_clamp(ceilf(nmax(t0, t1)), dl, dh);
#pragma unroll 1
    for (int x = nim_clamp(lo, dl, dh) + lane; x < x1; x += 32) {
      const float area = (s & 1) ? trap_right_area(m, b, t0, t1, x, xs, y) : trap_left_area(m, b, t0, t1, x, xs, y);
      if (area == 0.0f || nim_u32(roundf(area * 255.0f)) <= 255) continue;
      const int z = atomicAdd(&S->nzero, 1);
      if (z < kZeroCap) {
        S->zero[z] = x;
        S->key[z] = area;
      }
    }
  }
  __syncwarp();
  return S->nzero > kZeroCap;
}
// The listed pixels, drawn as the general code draws them.
template <int OUT, int NB, int XT>
static __device__ __noinline__ void draw_odd(FastRow<NB, XT>* S, uint8_t* base, int mode, const uint8_t* tbl,
                                             uint32_t rgbx, int lane) {
  if (lane < S->nzero) {
    const int x = S->zero[lane];
    const uint32_t c = mul_f(rgbx, S->key[lane]);
    uint32_t* p = reinterpret_cast<uint32_t*>(base) + x;
    if (OUT == kOutA8) base[x] = (uint8_t)(c >> 24);
    else *p = blend_any(mode, tbl, *p, c);
  }
  __syncwarp();
}

// Rows [yA, yB) of job J (non-MaskBlend, narrower than fast_max_w(NB), within the
// path's rows), drawn into an RGBX image or an 8-bit mask, or recorded; rows it
// does not take are handed on to list LIST.
template <int OUT, int NB, int XT, int TILES, int LIST = 0, bool LINES = false>
__device__ __forceinline__ void fast_rows(const PathJob& J, const Arena& A, const uint8_t* tbl, int job, int yA,
                                          int yB, FastRow<NB, XT>& S, int lane, LineWork* L = nullptr,
                                          LineScratch<NB>* K = nullptr) {
  constexpr bool REC = OUT == kOutRec, ONCE = TILES == kOnce;
  const unsigned lt = (1u << lane) - 1;
  const int W = (int)J.W, startY = (int)J.startY, pathHeight = (int)J.pathHeight, ph = (int)J.ph;
  const int winding = J.winding, nb = J.nb;
  const bool flat = J.mode == kOverwrite || (J.mode == kNormal && (J.rgbx >> 24) == 255);  // covers what it is drawn on
  int cnt = 0, validTo = yA;  // validTo: the rows the loaded entries serve
  bool aa = false, two = false;
#pragma unroll 1
  for (int y = yA; y < yB; y++) {
    if (y >= validTo) {
      const int k = min((y - startY) / ph, nb - 1);
      const Band bd = A.bands[J.band_off + k];
      const int bt = startY + k * ph;  // the band's top and bottom (:1178-1190)
      const int bb = k == nb - 1 ? pathHeight : bt + ph;
      aa = (bd.flags & kBandAA) != 0;
      validTo = min(bb, yB);
#pragma unroll 1
      while (true) {  // too many entries for the chunk: this row's alone
        __syncwarp();
        cnt = load_chunk<NB, XT>(J, A, bd, (float)bt, (float)bb, (float)y, (float)validTo, S, lane, two);
        if (cnt >= 0 || validTo == y + 1) break;
        validTo = y + 1;
      }
    }
    if (cnt < 0) {
      push_row(A, job, y, lane, LIST);
      continue;
    }
    const float yTop = (float)y, yBottom = (float)(y + 1);
    int n = 0;
    int kind = 0;             // 0: sample lines, 1: trapezoids, 2: a filled span
    bool ordered = false;     // the trapezoids, one behind the other
    int dl = 0, dh = W;       // the pixels the row may touch
    if (two && !aa) {
      // (i) non-AA band with two spanning vertical edges (:1644-1668)
      kind = 2;
      dl = nim_clamp(S.ends[0][0], 0, W);
      dh = nim_clamp(S.ends[1][0], 0, W);
    } else {
      // entries overlapping the scanline, in band order (:1677-1693)
      bool allSpan = true;
      __syncwarp();
      if (two) {
        n = 2;
        if (lane < 2) S.idx[lane] = (uint16_t)lane;
      } else {
#pragma unroll 1
        for (int j0 = 0; j0 < cnt; j0 += 32) {
          const int j = j0 + lane;
          const float ay = j < cnt ? S.ay(j) : yBottom, by = j < cnt ? S.by(j) : yTop;
          const bool pred = !(by <= yTop || ay >= yBottom);
          const unsigned msk = __ballot_sync(0xffffffffu, pred);
          if (pred) S.idx[n + __popc(msk & lt)] = (uint16_t)j;
          if (__any_sync(0xffffffffu, pred && (ay > yTop || by < yBottom))) allSpan = false;
          n += __popc(msk);
        }
      }
      __syncwarp();
      if (n == 0) continue;
      // (ii) trapezoid fast path (:1695-1872), else (iii) computeCoverage
      // (:1350-1431) + fillCoverage / fillHits
      if (allSpan && (n & 1) == 0) {
        if (trap_row<ONCE>(S, n, yTop, yBottom, winding, lane, ordered)) {
          kind = 1;
          // the pixels the pairs touch (the path's bounds do not limit them)
          int lo = W, hi = 0;
#pragma unroll 1
          for (int i = lane; i < n; i += 32) {
            const float t0 = S.t0[i], t1 = S.t1[i];
            const int a = nim_clamp(nmin(t0, t1), 0, W), c = nim_clamp(ceilf(nmax(t0, t1)), 0, W);
            lo = min(lo, min(a, c));
            hi = max(hi, max(a, c));
          }
          dl = __reduce_min_sync(0xffffffffu, lo);
          dh = __reduce_max_sync(0xffffffffu, hi);
        } else {
          // the sample lines see the sorted entries
#pragma unroll 1
          for (int i = lane; i < n; i += 32) S.perm[i] = S.idx[S.perm[i]];
          __syncwarp();
#pragma unroll 1
          for (int i = lane; i < n; i += 32) S.idx[i] = S.perm[i];
          __syncwarp();
        }
      }
      if (kind == 0 && aa) {  // fillHits draws anywhere on the row, coverage within the path's bounds
        dl = (int)J.startX;
        dh = (int)min(J.W, J.startX + J.pathWidth);
      }
    }
    if (dh <= dl) continue;
    int4* hdr = REC ? A.rowhdr + J.ri_off + (long long)y * J.ri_stride : nullptr;
    if (REC && kind == 2) {
      if (lane == 0) *hdr = make_int4(kRecFill, 0, dl, dh);
      continue;
    }
    uint8_t* base = J.img + (long long)y * W * (OUT == kOutA8 ? 1 : 4);  // pixel 0 of the row
    const int off = REC ? dl & 15
                        : OUT == kOutA8 ? (int)((reinterpret_cast<uintptr_t>(base) + dl) & 7)
                                        : (int)(((reinterpret_cast<uintptr_t>(base) >> 2) + dl) & 3);
    const bool tiled = TILES != kNoTiles && dh - (dl - off) > XT;  // wider than the difference array
    long long cov = -1;                       // REC: the row's bytes in cov8
    unsigned covBytes = 0;
    int covX = dl - off, covHi = dh;
    bool failed = false;
    // a row in several tiles whose trapezoids might be the general code's is
    // gone through once, whole, before any of it is drawn
    bool dry = !REC && tiled && kind == 1;
    int held = -1, from = 0;  // what the tiles before found: the row's spans, its first trapezoid to come
    bool listed = false;      // the row's odd multipliers are in S.zero
    if (REC && lane == 0) S.nzero = 0;
    __syncwarp();
#pragma unroll 1
    for (int xt = dl - off; !failed; xt += XT) {
      if (xt >= dh) break;
      CovTile T{xt, max(dl, xt), dry ? dh : min(dh, xt + XT), INT_MAX, INT_MIN};
      if (kind == 0) {
        if constexpr (LINES && (REC || NB > 512)) {
          cov_lines<!REC>(S, *L, *K, n, y, (float)W, winding, aa, T, lane, held);
        } else {
          bool byLines = false;
          if constexpr (LINES) {
            byLines = n > kGroupN;
            if (byLines) cov_lines<!REC>(S, *L, *K, n, y, (float)W, winding, aa, T, lane, held);
          }
          if (!byLines) cov_samples<!REC, ONCE, NB, XT>(S, n, y, (float)W, winding, aa, T, lane, held);
        }
      } else {
        if (kind == 1) {
          if (trap_cov<REC, ONCE>(S, n, y, T, lane, dry, ordered, from) && !listed) {
            listed = true;
            failed = list_odd(&S, n, y, dl, dh, !REC, lane);
          }
        } else if (lane == 0) cov_range(S.diff, T, dl, dh, 255);
        T.lo = T.t0;
        T.hi = T.t1;
        if (!REC && dry) {
          dry = false;
          xt -= XT;
          continue;
        }
      }
      __syncwarp();
      const int lo = max(__reduce_min_sync(0xffffffffu, T.lo), T.t0);
      const int hi = min(__reduce_max_sync(0xffffffffu, T.hi), T.t1);
      int i0 = 0, iEnd = T.t1 - xt;
      if (!tiled || ONCE) {
        if (hi <= lo) {  // every difference cancelled or was dropped
          if (ONCE && tiled) continue;
          break;
        }
        i0 = (lo - xt) & ~15;
        iEnd = hi - xt;
      }
      if (REC && cov < 0 && !failed) {  // the row's bytes: what it touches, or all tiles
        covX = xt + i0;
        covHi = tiled ? dh : hi;
        covBytes = (unsigned)(covHi - covX + 15) & ~15u;
        unsigned long long cb = 0;
        if (lane == 0) cb = atomicAdd(&A.counters[kCtrCov8], (unsigned long long)covBytes);
        cb = __shfl_sync(0xffffffffu, cb, 0);
        cov = (long long)cb;
        failed = (long long)(cb + covBytes) > A.cov8_cap;
      }
      uint8_t* dst = REC ? A.cov8 + cov : base;
      flush_diff<OUT == kOutRgbx ? 2 : 4, ONCE>(S.diff, i0, iEnd, lane, [&](int i, const uint32_t* f) {
        if (REC) {
          const int o = xt + i - covX;
          if (i < XT && o < (int)covBytes && !failed)
            *reinterpret_cast<uint2*>(dst + o) = make_uint2(pack4(f[0], f[1]), pack4(f[2], f[3]));
        } else if (OUT == kOutA8) {
          // a mask job paints white, opaque, Normal onto a cleared mask, each
          // pixel once: the blended alpha is the multiplier
          const uint32_t a = pack4(f[0], f[1]), b = pack4(f[2], f[3]);
          const int x = xt + i;
          if (failed || (a | b) == 0) return;
          if (x >= 0 && x + 8 <= W) {
            *reinterpret_cast<uint2*>(dst + x) = make_uint2(a, b);
          } else {
#pragma unroll 1
            for (int q = 0; q < 8; q++) {
              const uint32_t v = ((q < 4 ? a : b) >> ((q & 3) * 8)) & 255u;
              if (v && x + q >= 0 && x + q < W) dst[x + q] = (uint8_t)v;
            }
          }
        } else {
          const uint32_t c[4] = {f[0] & 0xffffu, f[0] >> 16, f[1] & 0xffffu, f[1] >> 16};
          const int x = xt + i;
          uint32_t* p = reinterpret_cast<uint32_t*>(base) + x;
          const bool vec = x >= 0 && x + 4 <= W, some = !failed && (f[0] | f[1]) != 0;
          const bool whole = vec && (f[0] & f[1] & 0x00ff00ffu) == 0x00ff00ffu;
          // a step within a span, where it is Normal: no blend for parts of it (a
          // translucent heart on 3000 x 3000 111 -> 100 us)
          if (!LINES && J.mode == kNormal && !flat && !__any_sync(0xffffffffu, some && !whole)) {
            if (!some) return;
            uint4 v = *reinterpret_cast<const uint4*>(p);
            v.x = blendNormal(v.x, J.rgbx);
            v.y = blendNormal(v.y, J.rgbx);
            v.z = blendNormal(v.z, J.rgbx);
            v.w = blendNormal(v.w, J.rgbx);
            *reinterpret_cast<uint4*>(p) = v;
            return;
          }
          if (!some) return;
          // what a full coverage replaces is not read (a heart that overwrites 8192 x
          // 8192: 368 us reading, 183 not)
          if (whole && flat) {
            *reinterpret_cast<uint4*>(p) = make_uint4(J.rgbx, J.rgbx, J.rgbx, J.rgbx);
            return;
          }
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (vec) {
            v = *reinterpret_cast<const uint4*>(p);
          } else {
            if (c[0] && x >= 0 && x < W) v.x = p[0];
            if (c[1] && x >= -1 && x + 1 < W) v.y = p[1];
            if (c[2] && x >= -2 && x + 2 < W) v.z = p[2];
            if (c[3] && x >= -3 && x + 3 < W) v.w = p[3];
          }
          uint32_t c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
#pragma unroll 1
          for (int q = 0; q < 4; q++) {  // one copy of the blend: the pixels rotate through it
            uint32_t r = v.x;
            if (c0) r = blend_row(J.mode, tbl, r, mul_c(J.rgbx, c0 & 255u));
            v = make_uint4(v.y, v.z, v.w, r);
            const uint32_t t = c0;
            c0 = c1;
            c1 = c2;
            c2 = c3;
            c3 = t;
          }
          if (vec) {
            *reinterpret_cast<uint4*>(p) = v;
          } else {
            if (c0 && x >= 0 && x < W) p[0] = v.x;
            if (c1 && x >= -1 && x + 1 < W) p[1] = v.y;
            if (c2 && x >= -2 && x + 2 < W) p[2] = v.z;
            if (c3 && x >= -3 && x + 3 < W) p[3] = v.w;
          }
        }
      });
    }
    if (failed) {
      push_row(A, job, y, lane, LIST);
    } else if (!REC) {
      if (listed) draw_odd<OUT>(&S, base, J.mode, tbl, J.rgbx, lane);
    } else if (cov >= 0) {
      const int nz = S.nzero;
      if (nz > kZeroCap) {
        push_row(A, job, y, lane, LIST);
      } else if (nz == 0) {
        if (lane == 0) *hdr = make_int4(kRecCov8, (int)(cov >> 4), covX, covHi);
      } else {
        const long long at = rec_alloc(J, A, y, kRecCov8Z, 1 + (nz + 1) / 2, covX, covHi, lane);
        const int x = S.zero[min(lane, nz - 1)];
        const int lo = __reduce_min_sync(0xffffffffu, x), hi = __reduce_max_sync(0xffffffffu, x);
        if (at >= 0) {
          if (lane == 0) A.prog[at] = make_int4((int)(cov >> 4), nz, lo, hi);
          if (lane < nz) reinterpret_cast<int2*>(A.prog + at + 1)[lane] = make_int2(x, __float_as_int(S.key[lane]));
        }
      }
    }
  }
}

// The warps of a CTA that take a row's other sample lines, until warp 0 has no
// more rows; what warp 0 calls then.
template <bool SKIP, int NB, int XT>
__device__ __forceinline__ void line_warps(LineRow<NB, XT>& S, int warp, int lane) {
#pragma unroll 1
  while (true) {
    line_barrier();
    if (S.work.n < 0) break;
    one_line<SKIP>(S.row, S.work, S.line[warp], warp, lane);
    line_barrier();
  }
}
__device__ __forceinline__ void line_warps_end(LineWork& W, int lane) {
  if (lane == 0) W.n = -1;
  line_barrier();
}

template <int NB, int XT>
__device__ __forceinline__ void init_fast_row(FastRow<NB, XT>& S, int lane) {
#pragma unroll 1
  for (int i = lane; i < (XT + 272) / 2; i += 32) S.diff[i] = kDiffZero;
  __syncwarp();
}

}  // namespace pxg
