// Separable filters: gaussian blur (src/pixie/images.nim:304-365), spread
// (images.nim:700-758) and shadow (images.nim:760-776).
//
// blur: the X pass quantises each channel to uint8 (v div 256 div 255) before
// the Y pass, exactly as the reference's transposed intermediate does; taps
// outside the image take the outOfBounds colour.  Sums are exact uint32
// (255 * sum(weights) < 2^24).  Both passes stage a tile plus its halo in
// shared memory and run one output pixel per thread.
// shadow: MaskBlend reads only the mask's alpha and spread writes
// rgbx(0,0,0,v), so the whole shadow runs on one uint8 alpha plane.
#include <algorithm>

#include "pxg_device.cuh"

namespace pxg {

void note_launch();

constexpr int kBX = 256;       // X pass: outputs per CTA
constexpr int kTX = 32;        // Y pass: tile width
constexpr int kTY = 64;        // Y pass: tile height
constexpr int kYThreadsY = 8;  // Y pass: block is 32 x 8

__device__ __forceinline__ void mac4(uint32_t s[4], uint32_t p, uint32_t w) {
  s[0] += (p & 255u) * w;
  s[1] += ((p >> 8) & 255u) * w;
  s[2] += ((p >> 16) & 255u) * w;
  s[3] += (p >> 24) * w;
}
__device__ __forceinline__ uint32_t quant4(const uint32_t s[4]) {
  return pack(s[0] / 256 / 255, s[1] / 256 / 255, s[2] / 256 / 255, s[3] / 256 / 255);
}

// ---- RGBX blur --------------------------------------------------------------
__global__ void __launch_bounds__(kBX) k_blur_x(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                long long W, long long H, int r,
                                                const uint16_t* __restrict__ kern, uint32_t oob) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint32_t* px = reinterpret_cast<uint32_t*>(sm);
  uint16_t* kw = reinterpret_cast<uint16_t*>(px + kBX + 2 * r);
  const long long y = blockIdx.y, x0 = (long long)blockIdx.x * kBX;
  const uint32_t* row = in + y * W;
  for (int i = threadIdx.x; i < kBX + 2 * r; i += kBX) {
    long long gx = x0 - r + i;
    px[i] = (gx >= 0 && gx < W) ? row[gx] : oob;
  }
  for (int i = threadIdx.x; i < 2 * r + 1; i += kBX) kw[i] = kern[i];
  __syncthreads();
  const long long x = x0 + threadIdx.x;
  if (x >= W) return;
  uint32_t s[4] = {0, 0, 0, 0};
  for (int k = 0; k <= 2 * r; k++) mac4(s, px[threadIdx.x + k], kw[k]);
  out[y * W + x] = quant4(s);
}

__global__ void __launch_bounds__(kTX * kYThreadsY) k_blur_y(const uint32_t* __restrict__ in,
                                                             uint32_t* __restrict__ out, long long W,
                                                             long long H, int r,
                                                             const uint16_t* __restrict__ kern,
                                                             uint32_t oob) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint32_t* px = reinterpret_cast<uint32_t*>(sm);  // (kTY + 2r) x kTX
  uint16_t* kw = reinterpret_cast<uint16_t*>(px + (kTY + 2 * r) * kTX);
  const long long x0 = (long long)blockIdx.x * kTX, y0 = (long long)blockIdx.y * kTY;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTX + tx;
  const long long x = x0 + tx;
  for (int i = ty; i < kTY + 2 * r; i += kYThreadsY) {
    long long gy = y0 - r + i;
    uint32_t v = oob;
    if (gy >= 0 && gy < H) v = x < W ? in[gy * W + x] : 0u;
    px[i * kTX + tx] = v;
  }
  for (int i = tid; i < 2 * r + 1; i += kTX * kYThreadsY) kw[i] = kern[i];
  __syncthreads();
  if (x >= W) return;
  for (int oy = ty; oy < kTY; oy += kYThreadsY) {
    long long y = y0 + oy;
    if (y >= H) break;
    uint32_t s[4] = {0, 0, 0, 0};
    for (int k = 0; k <= 2 * r; k++) mac4(s, px[(oy + k) * kTX + tx], kw[k]);
    out[y * W + x] = quant4(s);
  }
}


// ---- RGBX blur, float32 path ------------------------------------------------
// Every tap product and every partial sum is an integer below 2^24
// (255 * sum(weights) <= 255 * 65345), so float32 multiply-adds give the
// exact uint32 sums of the reference.  Pixels are staged in shared memory as
// float4 (converted once per load) and each thread accumulates one output
// with one 128-bit shared load and four FFMAs per tap.
constexpr int kFX = 256;             // X pass: outputs per row per CTA
constexpr int kFXRows = 2;           // X pass: rows per CTA
constexpr int kFYT = 64;             // Y pass: output rows per CTA
constexpr int kFYThreads = 8;        // Y pass: block is 32 x 8

__device__ __forceinline__ float4 px4(uint32_t p) {
  return make_float4((float)(p & 255u), (float)((p >> 8) & 255u), (float)((p >> 16) & 255u),
                     (float)(p >> 24));
}
__device__ __forceinline__ uint32_t quantf(float4 s) {  // v div 256 div 255 of the exact sums
  return pack((uint32_t)s.x / 65280u, (uint32_t)s.y / 65280u, (uint32_t)s.z / 65280u,
              (uint32_t)s.w / 65280u);
}

__global__ void __launch_bounds__(kFX) k_blurf_x(const uint32_t* __restrict__ in,
                                                 uint32_t* __restrict__ out, long long W,
                                                 long long H, int r,
                                                 const uint16_t* __restrict__ kern, uint32_t oob) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int span = kFX + 2 * r;
  float4* px = reinterpret_cast<float4*>(sm);                 // kFXRows x span
  float* kw = reinterpret_cast<float*>(px + kFXRows * span);  // 2r + 1
  const long long x0 = (long long)blockIdx.x * kFX, y0 = (long long)blockIdx.y * kFXRows;
  const float4 o = px4(oob);
  for (int rr = 0; rr < kFXRows; rr++) {
    long long y = y0 + rr;
    if (y >= H) break;
    const uint32_t* row = in + y * W;
    for (int i = threadIdx.x; i < span; i += kFX) {
      long long gx = x0 - r + i;
      px[rr * span + i] = (gx >= 0 && gx < W) ? px4(row[gx]) : o;
    }
  }
  for (int i = threadIdx.x; i < 2 * r + 1; i += kFX) kw[i] = (float)kern[i];
  __syncthreads();
  const long long x = x0 + threadIdx.x;
  if (x >= W) return;
  for (int rr = 0; rr < kFXRows; rr++) {
    long long y = y0 + rr;
    if (y >= H) break;
    const float4* p = px + rr * span + threadIdx.x;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k <= 2 * r; k++) {
      float4 v = p[k];
      float w = kw[k];
      a.x = fmaf(v.x, w, a.x);
      a.y = fmaf(v.y, w, a.y);
      a.z = fmaf(v.z, w, a.z);
      a.w = fmaf(v.w, w, a.w);
    }
    out[y * W + x] = quantf(a);
  }
}

__global__ void __launch_bounds__(32 * kFYThreads) k_blurf_y(const uint32_t* __restrict__ in,
                                                             uint32_t* __restrict__ out, long long W,
                                                             long long H, int r,
                                                             const uint16_t* __restrict__ kern,
                                                             uint32_t oob) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int span = kFYT + 2 * r;
  float4* px = reinterpret_cast<float4*>(sm);            // span x 32
  float* kw = reinterpret_cast<float*>(px + span * 32);  // 2r + 1
  const long long x0 = (long long)blockIdx.x * 32, y0 = (long long)blockIdx.y * kFYT;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const long long x = x0 + tx;
  const float4 o = px4(oob);
  for (int i = ty; i < span; i += kFYThreads) {
    long long gy = y0 - r + i;
    float4 v = o;
    if (gy >= 0 && gy < H) v = x < W ? px4(in[gy * W + x]) : make_float4(0.f, 0.f, 0.f, 0.f);
    px[i * 32 + tx] = v;
  }
  for (int i = ty * 32 + tx; i < 2 * r + 1; i += 32 * kFYThreads) kw[i] = (float)kern[i];
  __syncthreads();
  if (x >= W) return;
  for (int oy = ty; oy < kFYT; oy += kFYThreads) {
    long long y = y0 + oy;
    if (y >= H) break;
    const float4* p = px + oy * 32 + tx;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k <= 2 * r; k++) {
      float4 v = p[k * 32];
      float w = kw[k];
      a.x = fmaf(v.x, w, a.x);
      a.y = fmaf(v.y, w, a.y);
      a.z = fmaf(v.z, w, a.z);
      a.w = fmaf(v.w, w, a.w);
    }
    out[y * W + x] = quantf(a);
  }
}

size_t blurf_x_smem(int r) { return (size_t)kFXRows * (kFX + 2 * r) * 16 + (size_t)(2 * r + 1) * 4 + 16; }
size_t blurf_y_smem(int r) { return (size_t)(kFYT + 2 * r) * 32 * 16 + (size_t)(2 * r + 1) * 4 + 16; }


// ---- RGBX blur, register-blocked float32 path ---------------------------------
// The tile lives in shared memory as [position along the filter axis][lane],
// where the 32 lanes are 32 rows (X pass) or 32 columns (Y pass), so every
// warp-wide 128-bit load is conflict-free.  Each thread produces 8
// consecutive outputs along the axis from a 16-pixel register window that
// advances 8 taps at a time: 16 shared loads feed 256 FFMAs.
constexpr int kBT = 64;   // outputs along the filter axis per CTA
constexpr int kBP = 8;    // outputs per thread (and taps per block)
constexpr int kBWarps = kBT / kBP;

__host__ __device__ constexpr int blockblur_span(int r) { return kBT + 2 * r + kBP; }
size_t blockblur_smem(int r) {
  return (size_t)blockblur_span(r) * 32 * 16 + (size_t)(2 * r + 1 + kBP) * 4 + 16;
}

template <bool XPASS>
__global__ void __launch_bounds__(kBWarps * 32, 2)
    k_blurb(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, long long W, long long H,
            int r, const uint16_t* __restrict__ kern, uint32_t oob) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int span = blockblur_span(r);
  const int ntap = 2 * r + 1;
  float4* px = reinterpret_cast<float4*>(sm);            // span x 32
  float* kw = reinterpret_cast<float*>(px + span * 32);  // taps, zero-padded to a multiple of 8
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // tile origin: along the axis (a0) and across it (c0)
  const long long a0 = (long long)blockIdx.x * kBT, c0 = (long long)blockIdx.y * 32;
  const long long alen = XPASS ? W : H, clen = XPASS ? H : W;
  const float4 o = px4(oob), zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // Stage the tile: 8 loads per thread in flight before any is converted, so
  // the staging does not wait on L2/HBM latency one pixel at a time.
  constexpr int kU = 8;
  const int total = span * 32;
  for (int i0 = tid; i0 < total; i0 += kU * kBWarps * 32) {
    uint32_t raw[kU];
    int kind[kU];  // 0: zero padding, 1: out of bounds, 2: pixel
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int i = i0 + u * kBWarps * 32;
      int p, c;
      if (XPASS) {  // consecutive threads read consecutive x of one row
        c = i / span;
        p = i - c * span;
      } else {  // consecutive threads read consecutive x of one row
        p = i >> 5;
        c = i & 31;
      }
      const long long ga = a0 - r + p, gc = c0 + c;
      kind[u] = 0;
      raw[u] = 0u;
      if (i < total && p < kBT + 2 * r && gc < clen) {
        if (ga >= 0 && ga < alen) {
          raw[u] = XPASS ? in[gc * W + ga] : in[ga * W + gc];
          kind[u] = 2;
        } else {
          kind[u] = 1;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int i = i0 + u * kBWarps * 32;
      if (i >= total) break;
      int p, c;
      if (XPASS) {
        c = i / span;
        p = i - c * span;
      } else {
        p = i >> 5;
        c = i & 31;
      }
      px[p * 32 + c] = kind[u] == 2 ? px4(raw[u]) : (kind[u] == 1 ? o : zero);
    }
  }
  for (int i = tid; i < ntap + kBP; i += kBWarps * 32) kw[i] = i < ntap ? (float)kern[i] : 0.f;
  __syncthreads();

  const int p0 = warp * kBP;  // this thread's first output along the axis
  float4 acc[kBP];
#pragma unroll
  for (int j = 0; j < kBP; j++) acc[j] = zero;
  for (int kb = 0; kb < ntap; kb += kBP) {
    float4 win[2 * kBP];
#pragma unroll
    for (int i = 0; i < 2 * kBP; i++) win[i] = px[(p0 + kb + i) * 32 + lane];
#pragma unroll
    for (int kk = 0; kk < kBP; kk++) {
      const float w = kw[kb + kk];
#pragma unroll
      for (int j = 0; j < kBP; j++) {
        acc[j].x = fmaf(win[j + kk].x, w, acc[j].x);
        acc[j].y = fmaf(win[j + kk].y, w, acc[j].y);
        acc[j].z = fmaf(win[j + kk].z, w, acc[j].z);
        acc[j].w = fmaf(win[j + kk].w, w, acc[j].w);
      }
    }
  }
  const long long gc = c0 + lane;
  if (XPASS) {
    // stage through shared memory so the row-major stores are coalesced
    __syncthreads();
    uint32_t* st = reinterpret_cast<uint32_t*>(sm);  // 32 rows x kBT
#pragma unroll
    for (int j = 0; j < kBP; j++) st[lane * kBT + p0 + j] = quantf(acc[j]);
    __syncthreads();
    for (int i = tid; i < 32 * kBT; i += kBWarps * 32) {
      int c = i / kBT, p = i - c * kBT;
      long long gy = c0 + c, gx = a0 + p;
      if (gy < H && gx < W) out[gy * W + gx] = st[i];
    }
  } else {
    if (gc < W) {
#pragma unroll
      for (int j = 0; j < kBP; j++) {
        long long gy = a0 + p0 + j;
        if (gy < H) out[gy * W + gc] = quantf(acc[j]);
      }
    }
  }
}

void* blurb_kernel(bool x) { return x ? (void*)k_blurb<true> : (void*)k_blurb<false>; }

// Direct (untiled) passes for radii whose halo does not fit in shared memory.
__global__ void k_blur_x_direct(const uint32_t* in, uint32_t* out, long long W, long long H, int r,
                                const uint16_t* kern, uint32_t oob) {
  const long long n = W * H;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long y = i / W, x = i - y * W;
    uint32_t s[4] = {0, 0, 0, 0};
    for (int k = 0; k <= 2 * r; k++) {
      long long gx = x - r + k;
      mac4(s, (gx >= 0 && gx < W) ? in[y * W + gx] : oob, kern[k]);
    }
    out[i] = quant4(s);
  }
}
__global__ void k_blur_y_direct(const uint32_t* in, uint32_t* out, long long W, long long H, int r,
                                const uint16_t* kern, uint32_t oob) {
  const long long n = W * H;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long y = i / W, x = i - y * W;
    uint32_t s[4] = {0, 0, 0, 0};
    for (int k = 0; k <= 2 * r; k++) {
      long long gy = y - r + k;
      mac4(s, (gy >= 0 && gy < H) ? in[gy * W + x] : oob, kern[k]);
    }
    out[i] = quant4(s);
  }
}

// ---- alpha-plane passes (shadow) -------------------------------------------
// mask.draw(image, translate(offset), OverwriteBlend), alpha only
__global__ void k_alpha_offset(const uint32_t* src, uint8_t* a, long long W, long long H,
                               long long ox, long long oy) {
  const long long n = W * H;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long y = i / W, x = i - y * W;
    long long sx = x - ox, sy = y - oy;
    a[i] = (sx >= 0 && sx < W && sy >= 0 && sy < H) ? (uint8_t)(src[sy * W + sx] >> 24) : 0;
  }
}
// spread: running max (grow) or min (shrink) over [c - s, c + s] clipped to
// the image, along x (dir 0) or y (dir 1)
__global__ void k_spread(const uint8_t* in, uint8_t* out, long long W, long long H, int s, int grow,
                         int dir) {
  const long long n = W * H;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long y = i / W, x = i - y * W;
    long long c = dir == 0 ? x : y, len = dir == 0 ? W : H;
    long long lo = c - s < 0 ? 0 : c - s, hi = c + s > len - 1 ? len - 1 : c + s;
    uint32_t v = grow ? 0u : 255u;
    for (long long t = lo; t <= hi; t++) {
      uint32_t p = dir == 0 ? in[y * W + t] : in[t * W + x];
      v = grow ? (p > v ? p : v) : (p < v ? p : v);
    }
    out[i] = (uint8_t)v;
  }
}
__global__ void k_blur_a(const uint8_t* in, uint8_t* out, long long W, long long H, int r,
                         const uint16_t* kern, uint32_t oobA, int dir) {
  const long long n = W * H;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long y = i / W, x = i - y * W;
    long long c = dir == 0 ? x : y, len = dir == 0 ? W : H;
    uint32_t s = 0;
    for (int k = 0; k <= 2 * r; k++) {
      long long t = c - r + k;
      uint32_t p = (t >= 0 && t < len) ? (dir == 0 ? in[y * W + t] : in[t * W + x]) : oobA;
      s += p * kern[k];
    }
    out[i] = (uint8_t)(s / 256 / 255);
  }
}
// result.fill(color); result.draw(mask, MaskBlend)  -> color * a / 255
__global__ void k_shadow_out(const uint8_t* a, uint32_t* out, long long n, uint32_t color) {
  Px c = unpack(color);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    uint32_t k = a[i];
    out[i] = pack((c.r * k) / 255, (c.g * k) / 255, (c.b * k) / 255, (c.a * k) / 255);
  }
}
// spread on an RGBX image: writes rgbx(0, 0, 0, v)
__global__ void k_alpha_to_rgbx(const uint8_t* a, uint32_t* out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = (uint32_t)a[i] << 24;
}
__global__ void k_rgbx_alpha(const uint32_t* in, uint8_t* a, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    a[i] = (uint8_t)(in[i] >> 24);
}

static unsigned grid_for(long long n, int nsm) {
  long long b = (n + 255) / 256, cap = (long long)nsm * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

size_t blur_x_smem(int r) { return (size_t)(kBX + 2 * r) * 4 + (size_t)(2 * r + 1) * 2 + 16; }
size_t blur_y_smem(int r) { return (size_t)(kTY + 2 * r) * kTX * 4 + (size_t)(2 * r + 1) * 2 + 16; }

// in -> tmp (X pass) -> in (Y pass); float32 tiles when they fit, then the
// integer tiles, then the direct kernels.


void launch_blur(uint32_t* img, uint32_t* tmp, long long W, long long H, int r,
                 const uint16_t* kern, uint32_t oob, int nsm, size_t maxSmem, cudaStream_t st) {
  // radius >= 8: register-blocked tiles; smaller radii stay on the one-output
  // float32 tiles, where the blocked kernel's 8-tap granularity and halo cost
  // more than they save.
  if (r >= 8 && blockblur_smem(r) <= maxSmem && (H + 31) / 32 <= 65535 && (W + 31) / 32 <= 65535) {
    dim3 gx((unsigned)((W + kBT - 1) / kBT), (unsigned)((H + 31) / 32));
    k_blurb<true><<<gx, kBWarps * 32, blockblur_smem(r), st>>>(img, tmp, W, H, r, kern, oob); note_launch();
    dim3 gy((unsigned)((H + kBT - 1) / kBT), (unsigned)((W + 31) / 32));
    k_blurb<false><<<gy, kBWarps * 32, blockblur_smem(r), st>>>(tmp, img, W, H, r, kern, oob); note_launch();
    return;
  }
  if (blurf_x_smem(r) <= maxSmem && (H + kFXRows - 1) / kFXRows <= 65535) {
    dim3 g((unsigned)((W + kFX - 1) / kFX), (unsigned)((H + kFXRows - 1) / kFXRows));
    k_blurf_x<<<g, kFX, blurf_x_smem(r), st>>>(img, tmp, W, H, r, kern, oob); note_launch();
  } else if (blur_x_smem(r) <= maxSmem && H <= 65535) {
    dim3 g((unsigned)((W + kBX - 1) / kBX), (unsigned)H);
    k_blur_x<<<g, kBX, blur_x_smem(r), st>>>(img, tmp, W, H, r, kern, oob); note_launch();
  } else {
    k_blur_x_direct<<<grid_for(W * H, nsm), 256, 0, st>>>(img, tmp, W, H, r, kern, oob); note_launch();
  }
  if (blurf_y_smem(r) <= maxSmem && (H + kFYT - 1) / kFYT <= 65535) {
    dim3 g((unsigned)((W + 31) / 32), (unsigned)((H + kFYT - 1) / kFYT));
    k_blurf_y<<<g, dim3(32, kFYThreads), blurf_y_smem(r), st>>>(tmp, img, W, H, r, kern, oob); note_launch();
  } else if (blur_y_smem(r) <= maxSmem && (H + kTY - 1) / kTY <= 65535) {
    dim3 g((unsigned)((W + kTX - 1) / kTX), (unsigned)((H + kTY - 1) / kTY));
    k_blur_y<<<g, dim3(kTX, kYThreadsY), blur_y_smem(r), st>>>(tmp, img, W, H, r, kern, oob); note_launch();
  } else {
    k_blur_y_direct<<<grid_for(W * H, nsm), 256, 0, st>>>(tmp, img, W, H, r, kern, oob); note_launch();
  }
}

void launch_spread(uint32_t* img, uint8_t* a0, uint8_t* a1, long long W, long long H, int s,
                   int nsm, cudaStream_t st) {
  long long n = W * H;
  int grow = s > 0, m = s > 0 ? s : -s;
  k_rgbx_alpha<<<grid_for(n, nsm), 256, 0, st>>>(img, a0, n); note_launch();
  k_spread<<<grid_for(n, nsm), 256, 0, st>>>(a0, a1, W, H, m, grow, 0); note_launch();
  k_spread<<<grid_for(n, nsm), 256, 0, st>>>(a1, a0, W, H, m, grow, 1); note_launch();
  k_alpha_to_rgbx<<<grid_for(n, nsm), 256, 0, st>>>(a0, img, n); note_launch();
}

// Shadow in one pass over tiles of 64 columns and th rows: the tile and a halo of
// |spread| + radius (at most kShadowHalo) of the offset alpha plane are staged
// in shared memory and the reference's stages run there in order -- spread
// along x then y (a running max or min over the window clipped to the image:
// positions outside the image hold the neutral value), blur along x then y
// (taps outside the image read 0; integer sums and v div 256 div 255 as the
// blur passes), then colour * alpha / 255 (the MaskBlend draw of the filled
// result) written once.
//
// What bounds it is instructions: at 1237 x 1001, spread 4 and radius 12 a
// byte at a time took 31 us of which the image's bytes are 1.5.  So four
// neighbours are handled at once.  A shrink is a grow of the complement.  A
// window's four results share its middle.  A blur's are dot products of 16-bit
// weight pairs with byte pairs of the staged words (dp2a: two taps an
// instruction, exact), the weights of the four shifts read from one table of
// pairs (w[d], w[d + 1]); along y the same code runs on a transposed copy.
// Rows and columns of words have odd pitches, so lanes down a column fall on
// different banks.  At 1237 x 1001 (spread, radius): (4, 12) 29.7 -> 14.5 us,
// (0, 12) 18.3 -> 11.1, (4, 0) 15.6 -> 9.4, (0, 4) 13.3 -> 9.0, (0, 32) 37 ->
// 20.7, (16, 16) 59 -> 24.6.  Three CTAs an SM: at the 56 registers the
// compiler would take only two fit, and one tile in twenty runs a second wave.
//
// 4 Q is the radius rounded up to whole words: what a window's words reach
// beyond it meets zero weights.
constexpr int kShadowTile = 64, kShadowHalo = 32, kShadowThreads = 512, kShadowMaxRows = 96;
struct ShadowDims {  // in shared memory: two byte planes, the weight pairs, the colours by alpha
  int rows, hx, pitch;  // staged rows, columns left of the tile, words from row to row
};
__host__ __device__ inline ShadowDims shadow_dims(int th, int m, int r) {
  ShadowDims d;
  d.rows = th + 2 * (m + r);
  d.hx = (m + 3) / 4 * 4 + (r + 3) / 4 * 4;
  d.pitch = ((kShadowTile + 2 * d.hx) / 4) | 1;
  return d;
}
// The second plane also takes the transposed columns (64 of th + 8 ceil(r / 4)
// bytes and a word).
__host__ __device__ inline int shadow_col_words(int th, int r) { return (th / 4 + 2 * ((r + 3) / 4)) | 1; }
size_t shadow_tile_smem(int th, int m, int r) {
  const ShadowDims d = shadow_dims(th, m, r);
  return (size_t)(2 * ((r + 3) / 4) + 1) * 16 + 256 * 4 + (size_t)d.rows * d.pitch * 4 +
         std::max((size_t)d.rows * d.pitch, (size_t)kShadowTile * shadow_col_words(th, r)) * 4;
}
// Rows of a tile, a multiple of 4: what the busiest SM does (its tiles, their
// rows and halo, 24 rows' worth before the first) is least.  With 64 rows
// always, 1237 x 1001 at (4, 12) is three tiles on the busiest of 152 SMs and
// 17.9 us, at 68 two and 14.5; (0, 32) 24.1 and 20.7.
int shadow_tile_rows(long long W, long long H, int m, int r, int nsm) {
  const long long cols = (W + kShadowTile - 1) / kShadowTile;
  long long best = 0;
  int th = 64;
  for (int t = kShadowMaxRows; t >= 16; t -= 4) {
    const long long tiles = cols * ((H + t - 1) / t), cost = (tiles + nsm - 1) / nsm * (t + 2 * (m + r) + 24);
    if (best == 0 || cost < best) {
      best = cost;
      th = t;
    }
  }
  return th;
}

// Four outputs' weighted sums over the words p[0 .. 2 Q]: output o takes the
// bytes from 4 Q - r + o on.  wq[k] holds the weight pairs at d - 1 .. d + 2
// with d = 4 k - (4 Q - r); those at d - 3 and d - 2 are the word before's.
template <int Q>
__device__ __forceinline__ void dot_words(const uint32_t* p, const uint4* wq, uint32_t (&a)[4]) {
  uint32_t p1 = 0, p2 = 0;
  a[0] = a[1] = a[2] = a[3] = 0;
#pragma unroll(Q <= 2 ? 2 * Q + 1 : 3)
  for (int k = 0; k <= 2 * Q; k++) {
    const uint32_t v = p[k];
    const uint4 t = wq[k];
    a[0] = __dp2a_hi(t.w, v, __dp2a_lo(t.y, v, a[0]));
    a[1] = __dp2a_hi(t.z, v, __dp2a_lo(t.x, v, a[1]));
    a[2] = __dp2a_hi(t.y, v, __dp2a_lo(p2, v, a[2]));
    a[3] = __dp2a_hi(t.x, v, __dp2a_lo(p1, v, a[3]));
    p1 = t.z;
    p2 = t.w;
  }
}
// floor(floor(a / 256) / 255) for a < 2^24
__device__ __forceinline__ uint32_t quot_65280(uint32_t a) { return ((a >> 8) * 0x8081u) >> 23; }

template <int Q>
__global__ void __launch_bounds__(kShadowThreads, 3) k_shadow_tile(const uint32_t* __restrict__ src,
                                                                uint32_t* __restrict__ out, int W, int H, int ox,
                                                                int oy, int th, int m, int r, int grow,
                                                                const uint16_t* __restrict__ kern, uint32_t color,
                                                                int late) {
  extern __shared__ __align__(16) unsigned char sh[];
  constexpr int kWarps = kShadowThreads / 32, kCols = kShadowTile / 4 + 2 * Q;  // word columns the blur reads
  const ShadowDims D = shadow_dims(th, m, r);
  const int S = D.rows, P = 4 * D.pitch, h = m + r;
  uint4* wq = reinterpret_cast<uint4*>(sh);
  uint32_t* lut = reinterpret_cast<uint32_t*>(wq + 2 * Q + 1);
  unsigned char* b0 = reinterpret_cast<unsigned char*>(lut + 256);
  unsigned char* b1 = b0 + S * P;
  const int gx0 = blockIdx.x * kShadowTile - D.hx, gy0 = blockIdx.y * th - h;  // staged [0][0]
  const int tid = threadIdx.x, wi = tid >> 5, ln = tid & 31;
  pdl_late_entry(late);
  if (Q > 0 && tid < 4 * (2 * Q + 1)) {
    const int d = 4 * (tid >> 2) - (4 * Q - r) - 1 + (tid & 3);
    const uint32_t w0 = d >= 0 && d <= 2 * r ? kern[d] : 0u, w1 = d + 1 >= 0 && d + 1 <= 2 * r ? kern[d + 1] : 0u;
    reinterpret_cast<uint32_t*>(wq)[tid] = w0 | (w1 << 16);
  }
  if (tid < 256) lut[tid] = mul_div255_px(color, (uint32_t)tid);
  const uint32_t flip = (m > 0 && !grow) ? 255u : 0u;
  // the offset alpha plane (k_alpha_offset), complemented for a shrink; 0
  // (neutral) outside the image.  A warp's rows are loaded eight at a time.
  const int in0 = max(0, -gy0), inN = max(0, min(S, H - gy0) - in0);  // staged rows in the image
  const int so0 = max(in0, oy - gy0), soN = max(0, min(in0 + inN, H + oy - gy0) - so0);  // those with a source row
  const bool whole = gx0 >= max(0, ox) && gx0 + kShadowTile + 2 * D.hx <= min(W, W + ox) && soN == S;
  for (int j = ln; j < kShadowTile + 2 * D.hx; j += 32) {
    const int gx = gx0 + j, sx = gx - ox;
    const bool inx = gx >= 0 && gx < W;
    const unsigned n = inx ? (unsigned)inN : 0u, nsrc = inx && sx >= 0 && sx < W ? (unsigned)soN : 0u;
    for (int i0 = wi; i0 < S; i0 += 8 * kWarps) {
      // the alpha bytes (only read where they lie in the image)
      const unsigned char* p = reinterpret_cast<const unsigned char*>(src + (long long)(gy0 + i0 - oy) * W + sx) + 3;
      const long long step = (long long)kWarps * W * 4;
      uint32_t v[8];
      if (whole) {
#pragma unroll
        for (int k = 0; k < 8; k++, p += step)
          if (i0 + k * kWarps < S) v[k] = *p;
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (i0 + k * kWarps < S) b0[(i0 + k * kWarps) * P + j] = (unsigned char)(v[k] ^ flip);
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++, p += step) v[k] = (unsigned)(i0 + k * kWarps - so0) < nsrc ? *p : 0u;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int i = i0 + k * kWarps;
          if (i < S) b0[i * P + j] = (unsigned)(i - in0) < n ? (unsigned char)(v[k] ^ flip) : 0;
        }
      }
    }
  }
  __syncthreads();
  if (m > 0) {
    // spread along x into b1 and along y back into b0 (rows [m, S - m)), the
    // word columns that the blur reads; of a window's 2 m + 4 inputs for four
    // outputs the middle ones are in all
    const int wc0 = (m + 3) / 4;
    for (int task = tid; task < S * kCols; task += kShadowThreads) {
      const int i = task / kCols, wc = wc0 + task - i * kCols;
      const unsigned char* p = b0 + i * P + 4 * wc - m;
      uint32_t c = 0;
      for (int t = 3; t <= 2 * m; t++) c = max(c, (uint32_t)p[t]);
      const uint32_t l0 = p[0], l1 = p[1], l2 = p[2], e1 = p[2 * m + 1], e2 = p[2 * m + 2], e3 = p[2 * m + 3];
      const uint32_t l12 = max(l1, l2), e12 = max(e1, e2);
      const uint32_t o0 = max(max(l0, l12), c), o1 = max(max(l12, c), e1), o2 = max(max(l2, c), e12),
                     o3 = max(max(c, e12), e3);
      reinterpret_cast<uint32_t*>(b1 + i * P)[wc] = o0 | (o1 << 8) | (o2 << 16) | (o3 << 24);
    }
    __syncthreads();
    const int rows = S - 2 * m;
    for (int task = tid; task < (rows + 3) / 4 * kCols; task += kShadowThreads) {
      const int rg = task / kCols, wc = wc0 + task - rg * kCols;
      const uint32_t* p = reinterpret_cast<const uint32_t*>(b1) + wc;
      const auto even = [&](int i) { return p[min(i, S - 1) * D.pitch] & 0x00FF00FFu; };
      const auto odd = [&](int i) { return (p[min(i, S - 1) * D.pitch] >> 8) & 0x00FF00FFu; };
      uint32_t ce = 0, co = 0;
      for (int t = 4 * rg + 3; t <= 4 * rg + 2 * m; t++) {
        const uint32_t v = p[t * D.pitch];
        ce = __vmaxu2(ce, v & 0x00FF00FFu);
        co = __vmaxu2(co, (v >> 8) & 0x00FF00FFu);
      }
      uint32_t res[4];
      const auto four = [&](auto get, uint32_t c, int s) {
        const int i = 4 * rg, e = i + 2 * m;
        const uint32_t l0 = get(i), l1 = get(i + 1), l2 = get(i + 2), e1 = get(e + 1), e2 = get(e + 2), e3 = get(e + 3);
        const uint32_t l12 = __vmaxu2(l1, l2), e12 = __vmaxu2(e1, e2);
        const uint32_t o[4] = {__vmaxu2(__vmaxu2(l0, l12), c), __vmaxu2(__vmaxu2(l12, c), e1),
                               __vmaxu2(__vmaxu2(l2, c), e12), __vmaxu2(__vmaxu2(c, e12), e3)};
#pragma unroll
        for (int k = 0; k < 4; k++) res[k] = s ? res[k] | (o[k] << 8) : o[k];
      };
      four(even, ce, 0);
      four(odd, co, 1);
      uint32_t in = 0;  // blur taps outside the image read 0
#pragma unroll
      for (int k = 0; k < 4; k++) in |= gx0 + 4 * wc + k >= 0 && gx0 + 4 * wc + k < W ? 255u << (8 * k) : 0u;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int i = m + 4 * rg + k, gy = gy0 + i;
        if (i < S - m)
          reinterpret_cast<uint32_t*>(b0)[i * D.pitch + wc] =
              gy >= 0 && gy < H ? (res[k] ^ (flip * 0x01010101u)) & in : 0u;
      }
    }
    __syncthreads();
  }
  const int bx = blockIdx.x * kShadowTile, by = blockIdx.y * th;
  if (Q > 0) {
    // blur along x: rows [m, S - m), the tile's columns, transposed into b1
    // (column c's bytes from 4 Q - r on; 0 outside the image).  A warp takes a
    // word column, its lanes the rows.
    const int tp = shadow_col_words(th, r);  // words from column to column (odd)
    static_assert(kWarps == kShadowTile / 4, "one warp for each word column");
    for (int t = ln; t < S - 2 * m; t += 32) {
      uint32_t a[4];
      dot_words<Q>(reinterpret_cast<const uint32_t*>(b0) + (m + t) * D.pitch + D.hx / 4 - Q + wi, wq, a);
      const int gy = gy0 + m + t;
      const bool in = gy >= 0 && gy < H;
#pragma unroll
      for (int o = 0; o < 4; o++)
        b1[(4 * wi + o) * 4 * tp + t + 4 * Q - r] = in ? (unsigned char)quot_65280(a[o]) : 0;
    }
    __syncthreads();
    // blur along y: lanes take columns, four rows each
    const int c = ln + 32 * (wi & 1);
    if (bx + c < W) {
#pragma unroll 1
      for (int yg = wi >> 1; yg < th / 4; yg += kWarps / 2) {
        uint32_t a[4];
        dot_words<Q>(reinterpret_cast<const uint32_t*>(b1) + c * tp + yg, wq, a);
#pragma unroll
        for (int o = 0; o < 4; o++) {
          const int gy = by + 4 * yg + o;
          if (gy < H) out[(long long)gy * W + bx + c] = lut[quot_65280(a[o]) & 255u];
        }
      }
    }
  } else {
    for (int idx = tid; idx < th * kShadowTile; idx += kShadowThreads) {
      const int y = idx / kShadowTile, x = idx % kShadowTile;
      if (bx + x < W && by + y < H) out[(long long)(by + y) * W + bx + x] = lut[b0[(h + y) * P + D.hx + x]];
    }
  }
  pdl_late_exit(late);
}
typedef void (*ShadowTileKernel)(const uint32_t*, uint32_t*, int, int, int, int, int, int, int, int, const uint16_t*,
                                 uint32_t, int);
template <int Q>
ShadowTileKernel shadow_tile_kernel(int r) {
  if constexpr (Q < kShadowHalo / 4)
    if (r > 4 * Q) return shadow_tile_kernel<Q + 1>(r);
  return k_shadow_tile<Q>;
}

void launch_shadow(const uint32_t* src, uint32_t* out, uint8_t* a0, uint8_t* a1, long long W,
                   long long H, long long ox, long long oy, int s, int r, const uint16_t* kern,
                   uint32_t color, int nsm, cudaStream_t st) {
  long long n = W * H;
  const int m = s > 0 ? s : -s;
  if (m + r <= kShadowHalo && W <= (1 << 24) && H <= (1 << 24) && ox > -(1 << 24) && ox < (1 << 24) &&
      oy > -(1 << 24) && oy < (1 << 24)) {
    const int th = shadow_tile_rows(W, H, m, r, nsm);
    const dim3 g((unsigned)((W + kShadowTile - 1) / kShadowTile), (unsigned)((H + th - 1) / th));
    const int late = dep_late(st, {Span{out, (size_t)(n * 4)}}, {Span{src, (size_t)(n * 4)}});
    launch_pdl(shadow_tile_kernel<0>(r), g, dim3(kShadowThreads), shadow_tile_smem(th, m, r), st, src, out, (int)W,
               (int)H, (int)ox, (int)oy, th, m, r, (int)(s > 0), kern, color, late);
    note_launch();
    return;
  }
  k_alpha_offset<<<grid_for(n, nsm), 256, 0, st>>>(src, a0, W, H, ox, oy); note_launch();
  if (s != 0) {
    int grow = s > 0, m = s > 0 ? s : -s;
    k_spread<<<grid_for(n, nsm), 256, 0, st>>>(a0, a1, W, H, m, grow, 0); note_launch();
    k_spread<<<grid_for(n, nsm), 256, 0, st>>>(a1, a0, W, H, m, grow, 1); note_launch();
  }
  if (r != 0) {
    k_blur_a<<<grid_for(n, nsm), 256, 0, st>>>(a0, a1, W, H, r, kern, 0u, 0); note_launch();
    k_blur_a<<<grid_for(n, nsm), 256, 0, st>>>(a1, a0, W, H, r, kern, 0u, 1); note_launch();
  }
  k_shadow_out<<<grid_for(n, nsm), 256, 0, st>>>(a0, out, n, color); note_launch();
}

}  // namespace pxg
