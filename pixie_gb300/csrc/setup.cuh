// The setup kernel of the fill pipeline: flatten -> segments -> bounds ->
// partitions, for one job per thread-block cluster.
//
// What bounds it: the latency of one job's chain.  A stroke's outline is tens
// of thousands of primitives and a curve's adaptive steps follow one another,
// while most SMs have nothing to do: on one CTA per job a 14,540-primitive
// stroke took 515 us, and the longest path of a 240-path scene 770 us of its
// 2.2 ms.  So a job is shared out over a cluster of CTAs, each owning a
// contiguous run of primitives and the segments they emit; sums, bounds and
// band counts are exchanged through distributed shared memory.  A curve with
// 8 or more lanes has several steps tested at once (flatten_chain).  Loops are
// rolled: the 61 KB of the unrolled kernel did not fit the instruction cache.
//
// Included by raster.cu after the flattening and segment helpers.
#pragma once
#include <cooperative_groups.h>

namespace pxg {

constexpr int kSetupThreads = 256, kSetupWarps = kSetupThreads / 32;
constexpr int kStepBytes = 16384;  // accepted levels or points of a CTA's curves, shared out over its groups

// One test of addCubic/addQuadratic's error margin (paths.nim:677-762): the
// segment from prev to the curve's point at t + sk.
struct StepTest {
  V2 nx;
  bool accept, invalid;
};
struct CurvePts {
  V2 at, c1, c2, to;
  bool cubic;
};
__device__ __forceinline__ V2 curve_at(const CurvePts& c, float t) {
  return c.cubic ? cubicAt(c.at, c.c1, c.c2, c.to, t) : quadAt(c.at, c.c1, c.c2, t);
}
__device__ __forceinline__ StepTest test_step(const CurvePts& c, float ems, V2 prev, float t, float sk) {
  StepTest r;
  r.invalid = sk <= FLT_EPSILON;
  const float sh = sk * 0.5f;
  r.nx = curve_at(c, t + sk);
  const V2 halfway = curve_at(c, t + sh);
  const V2 midpoint = (prev + r.nx) / 2;
  const float error = lengthSq(midpoint - halfway);
  if (c.cubic) {
    const V2 lineTangent = midpoint - prev;
    const V2 curveTangent = cubicDeriv(c.at, c.c1, c.c2, c.to, t + sh);
    const V2 scaled = (curveTangent / length(curveTangent)) * length(lineTangent);
    r.accept = !(error + lengthSq(lineTangent - scaled) > ems);
  } else {
    r.accept = !(error > ems);
  }
  return r;
}

// The reference's adaptive loop (addCubic, addQuadratic): after a segment is
// accepted it tries steps s0, s0/2, s0/4, ... until one passes the error test
// (or drops to float32 epsilon, which raises).  Every quantity the test at
// level k reads depends only on (t, s0, prev): halving a normal float is
// exact, so the sequential loop's recomputed `next = halfway` and `t + step/4`
// equal these values bit for bit, and the first level that passes is the one
// the sequential loop stops at.
__device__ __forceinline__ float next_s0(bool cubic, bool halfStepping, float step, float t) {
  return (!cubic && halfStepping) ? nmin(step, 1 - t) : nmin(step * 2, 1 - t);
}
__device__ __forceinline__ void load_curve(const Prim& q, CurvePts& c) {
  c.cubic = q.kind == kPrimCubic;
  c.at = V2{q.x[0], q.y[0]};
  c.c1 = V2{q.x[1], q.y[1]};
  c.c2 = V2{q.x[2], q.y[2]};
  c.to = V2{c.cubic ? q.x[3] : q.x[2], c.cubic ? q.y[3] : q.y[2]};
}

// Flattens the curves p0 + gid, p0 + gid + NG, ... < p1 of a job (lines are
// skipped), a group of G = 1, 2 or 4 lanes each: G levels of a step at once.
// The groups of a warp step together.  The accepted levels go to rec (cap
// bytes; *nrec counts them), from which a second call with replay set takes
// them without testing.  emit(p, prev, next) is called by every lane of the
// group for each segment addSegment keeps (zero-length ones dropped,
// :669-675), done(p) after a curve.  Returns the group's error status for the
// first failing curve it met (kOk if none), its index in errp.
template <class Emit, class Done>
__device__ __forceinline__ int flatten_small(const Prim* P, int p0, int p1, float ems, int G, int gid, int NG, int gl,
                                             int leader, bool replay, uint8_t* rec, int cap, int* nrec, int& errp,
                                             Emit&& emit, Done&& done) {
  const unsigned gbits = (1u << G) - 1;
  int p = p0 + gid, n = 0, status = kOk, base = 0;
  CurvePts c{V2{0, 0}, V2{0, 0}, V2{0, 0}, V2{0, 0}, false};
  V2 prev{0, 0};
  float t = 0, s0 = 1;
  bool halfStepping = false, fresh = true;  // fresh: p is the next primitive to look at
  long long rounds = 0;
#pragma unroll 1
  while (true) {
    if (fresh) {
#pragma unroll 1
      while (p < p1 && P[p].kind == kPrimLine) p += NG;
      if (p < p1) load_curve(P[p], c);
      prev = c.at;
      t = 0;
      s0 = 1;
      halfStepping = false;
      base = 0;
      rounds = 0;
      fresh = false;
    }
    const bool active = p < p1;
    if (!__any_sync(0xffffffffu, active)) break;
    int level;
    V2 next;
    if (replay) {
      level = active ? rec[n] : 0;
      next = curve_at(c, t + s0 * pow2neg(level));
    } else {
      const int k = base + gl;
      const StepTest a = test_step(c, ems, prev, t, k < 100 ? s0 * pow2neg(k) : 0.0f);
      const unsigned hit = (__ballot_sync(0xffffffffu, active && (a.invalid || a.accept)) >> leader) & gbits;
      const int src = leader + (hit ? __ffs(hit) - 1 : 0);
      next.x = __shfl_sync(0xffffffffu, a.nx.x, src);
      next.y = __shfl_sync(0xffffffffu, a.nx.y, src);
      const bool invalid = __shfl_sync(0xffffffffu, (int)a.invalid, src) != 0;
      if (active && (++rounds > kIterCap || (hit && invalid))) {
        status = rounds > kIterCap ? kErrIterLimit : c.cubic ? kErrCubic : kErrQuad;
        errp = p;
        p = p1;
        continue;
      }
      if (active && !hit) {
        base += G;
        continue;
      }
      level = base + src - leader;
      if (active && n < cap && gl == 0) rec[n] = (uint8_t)level;
    }
    if (!active) continue;
    ++n;
    const float step = s0 * pow2neg(level);
    if (prev.x - next.x != 0.0f || prev.y - next.y != 0.0f) emit(p, prev, next);
    t += step;
    if (t == 1) {
      done(p);
      p += NG;
      fresh = true;
      continue;
    }
    prev = next;
    if (level > 0) halfStepping = true;
    s0 = next_s0(c.cubic, halfStepping, step, t);
    base = 0;
  }
  *nrec = n;
  return status;
}

// The same with G = 8, 16 or 32 lanes a curve, several steps at once.  Nine
// steps in ten of a cubic keep the step before (level 1: the doubled step
// fails, its half passes), and a quadratic that has halved once stays at level
// 0.  So lane pair d tests levels 0 and 1 of the d-th step from here as it is
// if every step before it takes that level; the steps up to the first that
// does not are accepted together (its own, too, if it takes the other level;
// else its further levels are tested, G at once).  A random cubic of 46 steps
// takes 8 rounds.  The points go to buf (cap of them) and the lanes turn them
// into segments together: seg(p, valid, a, b) is called by the whole warp.  Where the
// group had one curve whose points fit, *kept is their number and a second
// call with kept >= 0 for the whole warp takes them as they are.
template <class Seg, class Done>
__device__ __forceinline__ int flatten_chain(const Prim* P, int p0, int p1, float ems, int G, int gid, int NG, int gl,
                                             int leader, V2* buf, int cap, int* kept, int& errp, Seg&& seg,
                                             Done&& done) {
  const unsigned gbits = G == 32 ? 0xffffffffu : ((1u << G) - 1);
  const int D = G / 2;
  int p = p0 + gid, n = 0, status = kOk, base = 0, keep = 0, curves = 0;
  const bool again = __all_sync(0xffffffffu, *kept >= 0);
  CurvePts c{V2{0, 0}, V2{0, 0}, V2{0, 0}, V2{0, 0}, false};
  V2 prev{0, 0};
  float t = 0, s0 = 1;
  bool halfStepping = false, fresh = true;
  long long rounds = 0;
#pragma unroll 1
  while (true) {
    if (fresh) {
#pragma unroll 1
      while (p < p1 && P[p].kind == kPrimLine) p += NG;
      if (p < p1) {
        load_curve(P[p], c);
        if (gl == 0) buf[0] = c.at;  // (a kept curve's first point is the same)
      }
      prev = c.at;
      t = 0;
      s0 = 1;
      halfStepping = false;
      base = 0;
      rounds = 0;
      n = 1;
      fresh = false;
    }
    const bool active = p < p1;
    if (!__any_sync(0xffffffffu, active)) break;
    bool finished = false;
    if (again) {
      n = *kept;
      finished = active;
    } else {
      // the lane's step: depth steps ahead at the usual level, or level base + gl of this one
      const bool chain = base == 0;
      const int usual = c.cubic || !halfStepping ? 1 : 0;
      const int len = c.cubic || halfStepping ? D : 1;
      const int depth = chain ? gl >> 1 : 0, level = chain ? gl & 1 : base + gl;
      float td = t, sd = s0;
#pragma unroll 1
      for (int i = 0; i < depth; i++) {
        const float step = usual ? sd * 0.5f : sd;
        td += step;
        sd = next_s0(c.cubic, true, step, td);
      }
      const V2 from = depth > 0 ? curve_at(c, td) : prev;
      const float sk = level < 100 ? sd * pow2neg(level) : 0.0f;
      const StepTest a = test_step(c, ems, from, td, sk);
      const bool inChain = active && depth < len && (depth == 0 || td < 1);
      const unsigned hit = (__ballot_sync(0xffffffffu, inChain && (a.invalid || a.accept)) >> leader) & gbits;
      const unsigned inv = (__ballot_sync(0xffffffffu, inChain && a.invalid) >> leader) & gbits;
      unsigned take = 0;  // the lanes whose steps are accepted
      bool deeper = false;  // the step after them passes neither level 0 nor 1
      if (chain) {
        const unsigned h0 = hit & 0x55555555u, h1 = (hit >> 1) & 0x55555555u;  // per depth, at bit 2 depth
        const unsigned asUsual = usual ? h1 & ~h0 : h0;
        const unsigned stop = ~asUsual & 0x55555555u & gbits;
        const unsigned before = stop ? (stop & (0u - stop)) - 1 : gbits;  // bits of the depths before the stop
        take = (asUsual & before) << usual;
        const unsigned at = stop & (0u - stop);  // the first depth that does not take the usual level
        if (usual ? (h0 & at) : (h1 & at)) take |= usual ? at : at << 1;
        else deeper = true;
      } else {
        take = hit & (0u - hit);
      }
      if (active && (++rounds > kIterCap || (inv & take))) {
        status = rounds > kIterCap ? kErrIterLimit : c.cubic ? kErrCubic : kErrQuad;
        errp = p;
        p = p1;
      }
      const int last = take ? 31 - __clz(take) : 0, taken = __popc(take);
      if (active && p < p1 && ((take >> gl) & 1)) buf[n + depth] = a.nx;
      const float tl = __shfl_sync(0xffffffffu, td + sk, leader + last);
      const float step = __shfl_sync(0xffffffffu, sk, leader + last);
      const float nx = __shfl_sync(0xffffffffu, a.nx.x, leader + last);
      const float ny = __shfl_sync(0xffffffffu, a.nx.y, leader + last);
      if (active && p < p1) {
        if (taken == 0) {
          base += chain ? 2 : G;
        } else {
          n += taken;
          t = tl;
          prev = V2{nx, ny};
          // level above 0: outside a chain, at an odd lane, or usual before the last
          if (!chain || (last & 1) || (usual && taken > 1)) halfStepping = true;
          s0 = next_s0(c.cubic, halfStepping, step, t);
          finished = t == 1;
          // (a chain that ran out of lanes says nothing about the step after it)
          base = chain && deeper && taken < len && !finished ? 2 : 0;
        }
      }
    }
    const bool flush = active && p < p1 && (finished || n + D > cap);
    if (__any_sync(0xffffffffu, flush)) {
      __syncwarp();
#pragma unroll 1
      for (int i = 1; __any_sync(0xffffffffu, flush && i < n); i += G) {
        const int j = i + gl;
        const bool valid = flush && j < n;
        const V2 u = buf[valid ? j - 1 : 0], v = buf[valid ? j : 0];
        seg(p, valid && (u.x - v.x != 0.0f || u.y - v.y != 0.0f), u, v);
      }
      __syncwarp();
      if (flush) {
        keep = finished && keep == 0 && ++curves == 1 ? n : -1;
        if (!finished && gl == 0) buf[0] = prev;
        n = 1;
      }
      __syncwarp();
    }
    if (finished) {
      done(p);
      p += NG;
      fresh = true;
    }
  }
  *kept = keep;
  return status;
}

// Sum of the values before this thread's, and the block's total.
__device__ __forceinline__ long long block_scan_excl(long long v, long long* s_warp, long long& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  long long before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kSetupWarps; w++) {
    if (w < warp) before += s_warp[w];
    total += s_warp[w];
  }
  return before + x - v;
}

// The job's outcome: for the host, and with its colour and mode for the
// drawing pass.
__device__ __forceinline__ void set_status(PathJob& J, const Arena& A, int job, int st) {
  J.status = st;
  A.pinfo[job] = make_uint2(J.rgbx, (uint32_t)J.mode | ((uint32_t)st << 8));
}

// C: CTAs per job (the cluster size; 1: a plain launch).
__global__ void __launch_bounds__(kSetupThreads, 4) k_setup(PathJob* jobs, Arena A, int maxBands, int C) {
  namespace cg = cooperative_groups;
  pdl_trigger();  // the row kernel may be set up while this runs; it waits for the segments
  pdl_wait();
  extern __shared__ int dsm[];
  // per band of a window of at most kBandWindow: the CTA's counts and places, and
  // each warp's own
  const int wb = min(maxBands, kBandWindow), stride = wb + 1;
  int* bandc = dsm;              // this CTA's entries
  int* bandf = dsm + stride;     // entries that need anti-aliasing (differences, then sums)
  int* bandx = bandf + stride;   // place of this CTA's first entry in the window's list
  int* wc = bandx + stride;      // [warp][band]: entries, then each warp's next place
  uint32_t* wm = reinterpret_cast<uint32_t*>(wc + kSetupWarps * stride);  // [warp][band]: lanes of a batch
  uint8_t* recs = reinterpret_cast<uint8_t*>(wm + kSetupWarps * stride);
  __shared__ long long s_err, s_base, s_bandbase, s_listbase, s_tot, s_warp[kSetupWarps];
  __shared__ int s_status;
  __shared__ float s_red[4][kSetupWarps], s_bounds[4];
  __shared__ int s_hdr[6];
  auto cluster = cg::this_cluster();
  auto sync = [&]() {
    if (C > 1) cluster.sync();
    else __syncthreads();
  };
  auto at = [&](auto* p, int q) { return C > 1 ? cluster.map_shared_rank(p, q) : p; };

  const int job = (int)blockIdx.x / C, rank = (int)blockIdx.x % C;
  PathJob& J = jobs[job];
  const int tid = threadIdx.x, T = kSetupThreads, lane = tid & 31, warp = tid >> 5;
  const unsigned lt32 = (1u << lane) - 1;
  if (tid == 0) {
    s_err = LLONG_MAX;
    s_status = kOk;
  }
  __syncthreads();

  const Prim* P = J.prims + J.prim_off;
  const int np = J.nprims, per = (np + C - 1) / C, p0 = min(np, rank * per), p1 = min(np, p0 + per);
  int* PC = A.primcnt + J.pc_off;
  SegMat M;
  M.identity = J.identity;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    M.mx[i] = J.mat[3 * i];
    M.my[i] = J.mat[3 * i + 1];
  }
  // lanes per curve: the CTA's threads shared out over the curves it may have
  // (chains need room for their points)
  const int most = min(per, (J.curves + C - 1) / C + 1);
  int G = 1;
  while (G < 32 && most * G * 2 <= T) G *= 2;
  const int NG = T / G, gid = tid / G, gl = tid % G, leader = lane - gl;
  const int cap = kStepBytes / NG;
  uint8_t* rec = recs + gid * cap;

  // Two passes: count the segments each primitive emits, then -- their places
  // known -- emit them in order and reduce the bounds (:1098-1117).
  long long segbase = 0;
  int off = 0, nseg = 0, mysegs = 0, nrec = 0, kept = -1;  // (places and counts fit once the total does)
  float xmin = INFINITY, xmax = -INFINITY, ymin = INFINITY, ymax = -INFINITY;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    const bool emitting = opaque(pass) == 1;
    auto put = [&](long long o, float4 s, int w) {
      A.segs[o] = s;
      A.segw[o] = w;
      xmin = nmin(xmin, nmin(s.x, s.z));
      xmax = nmax(xmax, nmax(s.x, s.z));
      ymin = nmin(ymin, s.y);
      ymax = nmax(ymax, s.w);
    };
#pragma unroll 1
    for (int p = p0 + tid; p < p1; p += T) {
      const Prim& q = P[p];
      if (q.kind != kPrimLine) continue;
      float4 s;
      int w;
      const V2 a{q.x[0], q.y[0]}, b{q.x[1], q.y[1]};
      const bool keep = (a.x - b.x != 0.0f || a.y - b.y != 0.0f) && make_seg(M, a, b, s, w);
      if (!emitting) PC[p] = keep ? 1 : 0;
      else if (keep) put(segbase + PC[p], s, w);
    }
    int cnt = 0, errp = 0, st;
    auto done = [&](int p) {
      if (!emitting && gl == 0) PC[p] = cnt;
      cnt = 0;
    };
    if (G >= 8) {
      const unsigned gbits = G == 32 ? 0xffffffffu : ((1u << G) - 1);
      st = flatten_chain(
          P, p0, p1, J.ems, G, gid, NG, gl, leader, reinterpret_cast<V2*>(rec), cap / (int)sizeof(V2), &kept, errp,
          [&](int p, bool valid, V2 a, V2 b) {
            float4 s;
            int w;
            const bool keep = valid && make_seg(M, a, b, s, w);
            const unsigned kept = (__ballot_sync(0xffffffffu, keep) >> leader) & gbits;
            if (emitting && keep) put(segbase + PC[p] + cnt + __popc(kept & ((1u << gl) - 1)), s, w);
            cnt += __popc(kept);
          },
          done);
    } else {
      // replay where every group of the warp kept its whole record, else search again
      const bool replay = emitting && __all_sync(0xffffffffu, nrec <= cap);
      st = flatten_small(
          P, p0, p1, J.ems, G, gid, NG, gl, leader, replay, rec, cap, &nrec, errp,
          [&](int p, V2 a, V2 b) {
            float4 s;
            int w;
            if (make_seg(M, a, b, s, w)) {
              if (emitting && gl == 0) put(segbase + PC[p] + cnt, s, w);
              cnt++;
            }
          },
          done);
    }
    if (emitting) break;
    if (st != kOk && gl == 0)  // the reference raises at the first failing primitive
      atomicMin(reinterpret_cast<unsigned long long*>(&s_err), (unsigned long long)(((long long)errp << 8) | st));
    __syncthreads();
    // exclusive prefix of the counts, in primitive order
    const int m = (p1 - p0 + T - 1) / T, q0 = min(p1, p0 + tid * m), q1 = min(p1, q0 + m);
    long long sum = 0, mine = 0, ahead = 0;
    if (s_err == LLONG_MAX) {
#pragma unroll 1
      for (int p = q0; p < q1; p++) sum += PC[p];
    }
    const long long first = block_scan_excl(sum, s_warp, mine);
    if (tid == 0) s_tot = mine;
    sync();
    long long err = LLONG_MAX, total = 0;
#pragma unroll 1
    for (int q = 0; q < C; q++) {
      err = min(err, *at(&s_err, q));
      const long long v = *at(&s_tot, q);
      if (q < rank) ahead += v;
      total += v;
    }
    if (rank == 0 && tid == 0) {
      s_base = 0;
      if (err != LLONG_MAX) s_status = (int)(err & 255);
      else if (total > INT_MAX) s_status = kErrTooManyEntries;
      else {
        s_base = (long long)atomicAdd(&A.counters[kCtrSegs], (unsigned long long)total);
        if (s_base + total > A.seg_cap) s_status = kErrArenaFull;
      }
    }
    sync();
    const int status = *at(&s_status, 0);
    segbase = *at(&s_base, 0);
    nseg = (int)total;
    if (status != kOk) {
      if (rank == 0 && tid == 0) set_status(J, A, job, status);
      sync();  // no CTA leaves while another may read its shared memory
      return;
    }
    off = (int)ahead;
    mysegs = (int)mine;
    int run = (int)(ahead + first);
#pragma unroll 1
    for (int p = q0; p < q1; p++) {
      const int v = PC[p];
      PC[p] = run;
      run += v;
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    xmin = nmin(xmin, __shfl_xor_sync(0xffffffffu, xmin, o));
    xmax = nmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
    ymin = nmin(ymin, __shfl_xor_sync(0xffffffffu, ymin, o));
    ymax = nmax(ymax, __shfl_xor_sync(0xffffffffu, ymax, o));
  }
  if (lane == 0) {
    s_red[0][warp] = xmin;
    s_red[1][warp] = xmax;
    s_red[2][warp] = ymin;
    s_red[3][warp] = ymax;
  }
  __syncthreads();
  if (tid < 4) {
    const bool mx = tid & 1;
    float v = mx ? -INFINITY : INFINITY;
#pragma unroll 1
    for (int w = 0; w < kSetupWarps; w++) v = mx ? nmax(v, s_red[tid][w]) : nmin(v, s_red[tid][w]);
    s_bounds[tid] = v;
  }
  sync();

  // bounds -> pixel window, partition geometry (:1602-1619, :1172-1192); every
  // CTA for itself
  if (tid == 0) {
    float x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
#pragma unroll 1
    for (int q = 0; q < C; q++) {
      const float* b = at(s_bounds, q);
      x0 = nmin(x0, b[0]);
      x1 = nmax(x1, b[1]);
      y0 = nmin(y0, b[2]);
      y1 = nmax(y1, b[3]);
    }
    float bx = 0, by = 0, bw = 0, bh = 0;
    if (!(isnan(x0) || isnan(x1) || isnan(y0) || isnan(y1))) {
      bx = x0;
      by = y0;
      bw = x1 - x0;
      bh = y1 - y0;
    }
    const long long W = J.W, H = J.H;
    float sx = floorf(bx), sw = ceilf(bx + bw) - sx;  // snapToPixels common.nim:92-101
    float sy = floorf(by), sh = ceilf(by + bh) - sy;
    long long startX = max(0LL, nim_int(sx)), startY = max(0LL, nim_int(sy));
    long long pathWidth = startX < W ? min(nim_int(sw), W - startX) : 0LL;
    long long pathHeight = min(H, nim_int(sy + sh));
    int status = kOk;
    if (pathWidth == 0) status = kNothing;
    else if (pathWidth < 0) status = kErrIntOverflow;
    // A path wholly above or below the image, or one whose end is past 2^63 (the
    // conversion's minimum then), draws no row and needs no partition.  The row
    // kernels hold rows in 32 bits: theirs are within the image from here on.
    if (pathHeight <= startY) startY = pathHeight = 0;
    const long long height = pathHeight - startY;
    uint32_t maxP = (uint32_t)max(1LL, height / 4);
    uint32_t numP = min(maxP, (uint32_t)max(1, nseg / 2));
    uint32_t ph = max(1u, (uint32_t)height / numP);
    if (status == kOk && numP > (uint32_t)maxBands) status = kErrArenaFull;
    s_hdr[0] = status;
    s_hdr[1] = (int)numP;
    s_hdr[2] = (int)ph;
    s_hdr[3] = (int)(uint32_t)startY;
    if (rank == 0) {
      J.seg_off = segbase;
      J.nseg = nseg;
      J.startX = startX;
      J.startY = startY;
      J.pathWidth = pathWidth;
      J.pathHeight = pathHeight;
      J.nb = (int)numP;
      J.ph = ph;
      if (status == kOk) {  // the bands' records
        s_bandbase = (long long)atomicAdd(&A.counters[kCtrBands], (unsigned long long)numP);
        if (s_bandbase + numP > A.band_cap) s_status = kErrArenaFull;
        J.band_off = s_bandbase;
      }
    }
  }
  __syncthreads();
  if (s_hdr[0] != kOk) {
    if (rank == 0 && tid == 0) set_status(J, A, job, s_hdr[0]);
    sync();
    return;
  }
  const uint32_t numP = (uint32_t)s_hdr[1], ph = (uint32_t)s_hdr[2];
  const float fStartY = (float)(uint32_t)s_hdr[3];
  auto bandRange = [&](float4 s) {  // partitionRange :1201-1213
    uint2 r = make_uint2(0u, 0u);
    if (numP > 1) {
      r.x = min(nim_u32(nmax(0.0f, s.y - fStartY)) / ph, numP - 1);
      r.y = min(nim_u32(nmax(0.0f, s.w - fStartY)) / ph, numP - 1);
    }
    return r;
  };

  // Windows of bands, one for images of up to 4096 rows: what the per-warp arrays
  // hold.  Each has a list of its own, so a tall image costs a pass over the
  // segments' ranges per window and nothing else.
  //
  // A window's entry counts and anti-aliasing flags (:1215-1234): every warp
  // owns a contiguous run of the CTA's segments and counts them as differences
  // over the bands, so a segment costs two additions however tall it is.  A
  // range may be empty (its first band above its last): a y of 2^32 or more
  // wraps in partitionRange's conversion, and the segment is in no band.
  int* mine = wc + warp * stride;
  uint32_t* mask = wm + warp * stride;
  const int perw = ((mysegs + kSetupWarps - 1) / kSetupWarps + 31) / 32 * 32;
  const int ws0 = min(mysegs, warp * perw), ws1 = min(mysegs, ws0 + perw);
  const long long seg0 = segbase + off;  // the CTA's first segment
  long long etotal = 0;  // a job of more than INT_MAX entries is an error: their places are 32 bits
  int status = kOk;
#pragma unroll 1
  for (int b0 = 0; b0 < (int)numP; b0 += wb) {
    const int nw = min(wb, (int)numP - b0);  // bands b0 .. b0 + nw - 1
#pragma unroll 1
    for (int k = tid; k <= nw; k += T) bandf[k] = 0;
#pragma unroll 1
    for (int k = lane; k <= nw; k += 32) {
      mine[k] = 0;
      mask[k] = 0u;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = ws0 + lane; i < ws1; i += 32) {
      const float4 sg = A.segs[seg0 + i];
      const uint2 r = bandRange(sg);
      if (b0 == 0) A.segband[seg0 + i] = r;
      const int x = max((int)r.x - b0, 0), y = min((int)r.y - b0, nw - 1);
      if (x > y || r.x > r.y) continue;
      atomicAdd(&mine[x], 1);
      atomicAdd(&mine[y + 1], -1);
      if (segRequiresAA(sg)) {
        atomicAdd(&bandf[x], 1);
        atomicAdd(&bandf[y + 1], -1);
      }
    }
    __syncthreads();
    // differences -> counts: each warp its own, warp 0 the flags
#pragma unroll 1
    for (int w = 0; w < 2; w++) {
      int* d = w == 0 ? mine : warp == 0 ? bandf : nullptr;
      if (!d) continue;
      int carry = 0;
#pragma unroll 1
      for (int k0 = 0; k0 < nw; k0 += 32) {
        const int k = k0 + lane;
        int v = k < nw ? d[k] : 0;
        v = carry + warp_scan_incl(v, lane);
        if (k < nw) d[k] = v;
        carry = __shfl_sync(0xffffffffu, v, 31);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int k = tid; k < nw; k += T) {
      int c = 0;
#pragma unroll 1
      for (int w = 0; w < kSetupWarps; w++) c += wc[w * stride + k];
      bandc[k] = c;
    }
    sync();
    // the bands' places in the list, in band order; within a band the CTAs in
    // rank order, so the list holds a band's segments ascending -- the order in
    // which partitionSegments appends them (:1215-1234)
    long long wtotal = 0;
#pragma unroll 1
    for (int k0 = 0; k0 < nw; k0 += T) {
      const int k = k0 + tid;
      int v = 0, before = 0, aa = 0;
      if (k < nw) {
#pragma unroll 1
        for (int q = 0; q < C; q++) {
          const int c = at(bandc, q)[k];
          if (q < rank) before += c;
          v += c;
          aa |= at(bandf, q)[k];
        }
      }
      long long tot;
      const long long ex = wtotal + block_scan_excl(v, s_warp, tot);
      if (k < nw) bandx[k] = (int)(ex + before);
      if (rank == 0 && k < nw && s_status == kOk) {
        Band bd;
        bd.off = ex;  // relative until the base is known
        bd.count = v;
        bd.flags = aa ? kBandAA : 0;
        A.bands[s_bandbase + b0 + k] = bd;
      }
      wtotal += tot;
    }
    etotal += wtotal;
    if (etotal > INT_MAX) {
      status = kErrTooManyEntries;
      break;
    }
    if (rank == 0 && tid == 0) {
      s_listbase = (long long)atomicAdd(&A.counters[kCtrBandSegs], (unsigned long long)wtotal);
      if (s_listbase + wtotal > A.bandseg_cap) s_status = kErrArenaFull;
    }
    sync();
    // (a workspace that is too small is told how much the other windows take)
    status = *at(&s_status, 0);
    if (status != kOk) continue;
    const long long listbase = *at(&s_listbase, 0);
    int* L = A.bandseg + listbase;
    if (rank == 0) {
#pragma unroll 1
      for (int k = tid; k < nw; k += T) A.bands[s_bandbase + b0 + k].off += listbase;
    }
    // each warp's start in every band: the CTA's plus the earlier warps' entries
#pragma unroll 1
    for (int k = tid; k < nw; k += T) {
      int run = bandx[k];
#pragma unroll 1
      for (int w = 0; w < kSetupWarps; w++) {
        const int t = wc[w * stride + k];
        wc[w * stride + k] = run;
        run += t;
      }
    }
    __syncthreads();
    // per batch of 32 segments, where they lie close together (a path's
    // neighbours mostly do), a lane owns a band of the batch's range and walks
    // the 32 segments; scattered short ones go the other way round: every lane
    // marks the bands its segment touches in the warp's band masks, and a
    // segment's place in band k is the warp's next place plus the number of
    // lower lanes in k's mask (2,700 segments of 64 cubics in 8 x 8 warps: 12,400
    // cycles with masks alone, 4,600 so).
#pragma unroll 1
    for (int c0 = ws0; c0 < ws1; c0 += 32) {
      const int i = c0 + lane;
      uint2 r = make_uint2(0xffffffffu, 0u);  // empty range
      if (i < ws1) {
        const uint2 g = A.segband[seg0 + i];
        const int x = max((int)g.x - b0, 0), y = min((int)g.y - b0, nw - 1);
        if (x <= y && g.x <= g.y) r = make_uint2((uint32_t)x, (uint32_t)y);
      }
      const uint32_t kmin = __reduce_min_sync(0xffffffffu, r.x), kmax = __reduce_max_sync(0xffffffffu, r.y);
      if (kmin > kmax) continue;
      const uint32_t tallest = __reduce_max_sync(0xffffffffu, r.x <= r.y ? r.y - r.x : 0u);
      if ((kmax - kmin) / 32 <= 1 + tallest / 2) {
#pragma unroll 1
        for (uint32_t k = kmin + lane; k - lane <= kmax; k += 32) {
          int pos = k <= kmax ? mine[k] : 0;
          const int end = min(32, ws1 - c0);
#pragma unroll 4
          for (int j = 0; j < end; j++) {
            const uint32_t a = __shfl_sync(0xffffffffu, r.x, j), b = __shfl_sync(0xffffffffu, r.y, j);
            if (a <= k && k <= b) L[pos++] = off + c0 + j;
          }
          if (k <= kmax) mine[k] = pos;
        }
        __syncwarp();
        continue;
      }
      const uint32_t bit = 1u << lane;
#pragma unroll 1
      for (uint32_t k = r.x; k <= r.y; k++) atomicOr(&mask[k], bit);
      __syncwarp();
#pragma unroll 1
      for (uint32_t k = r.x; k <= r.y; k++) L[mine[k] + __popc(mask[k] & lt32)] = off + i;
      __syncwarp();
      // each band's lowest lane advances the place and clears the mask
#pragma unroll 1
      for (uint32_t k = r.x; k <= r.y; k++) {
        const uint32_t m = mask[k];
        if (m && !(m & lt32)) {
          mine[k] += __popc(m);
          mask[k] = 0u;
        }
      }
      __syncwarp();
    }
    __syncthreads();  // the next window's counts take the places' room
  }
  if (rank == 0 && tid == 0) set_status(J, A, job, status);
  sync();  // no CTA leaves while another may read its shared memory
}

}  // namespace pxg
