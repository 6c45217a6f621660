// k_post.cu — frame development on the GPU: the reference's `post` module
// (src/post.rs:25-160), which runs on the CPU there, for the path tracer's
// accumulated image.
//
//   mean + keys   accum (r, g, b sums, samples) -> mean radiance per pixel
//                 (sums / max(samples, 1)) and each pixel's luminance
//                 (post.rs:31-33) as an order-preserving 32-bit key
//   select        the k-th smallest luminance by a 4-pass radix select
//                 (8 bits per pass, device-side bin choice) -- the exact
//                 value np.partition / the reference's sort picks
//   scale         linear = mean * 2^exposure, formed where it is read
//   glare_h, _v   the glare's box filters with the reference's running sums
//                 (post.rs:109-160): one thread per row (column) and channel
//                 keeps the sum, so every sum is formed in the same order as
//                 on the CPU; the three scales run side by side, each in
//                 place in a buffer of its own
//   box_h, box_v  the same filters from global memory, for images whose rows
//                 do not fit the shared memory (wider than 9,016 pixels)
//   final         glare mix, ACES fit, sRGB, dither and 8-bit quantisation
//                 (post.rs:47-88)
//
// FP32 in the reference's expression order (the library is built without
// fused multiply-add contraction): everything up to the sRGB curve is bit
// for bit the CPU restatement; powf in the sRGB curve may differ from the
// host's in the last place, which can move an 8-bit value by one.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "kernels.h"

namespace pyro {

namespace {

// float -> unsigned key with the same order (negative values reversed)
__device__ __forceinline__ uint32_t fkey(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void __launch_bounds__(256) k_post_mean(const float4* __restrict__ acc,
                                                   float* __restrict__ img,
                                                   uint32_t* __restrict__ keys, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const float4 a = acc[i];
  const float s = fmaxf(a.w, 1.0f);
  const float r = a.x / s, g = a.y / s, b = a.z / s;
  img[3 * i] = r;
  img[3 * i + 1] = g;
  img[3 * i + 2] = b;
  keys[i] = fkey(0.2126f * r + 0.7152f * g + 0.0722f * b);
}

// Radix-select state (POST_SEL_WORDS words): [0] prefix, [1] mask, [2] rank
// still to skip, [3] the selected key (after the last pass), [4..260) the
// histogram of the pass.
constexpr int SEL_HIST = 4;

__global__ void k_sel_init(uint32_t* __restrict__ sel, uint32_t rank) {
  for (int t = threadIdx.x; t < POST_SEL_WORDS; t += blockDim.x) sel[t] = t == 2 ? rank : 0u;
}

__global__ void __launch_bounds__(256) k_sel_hist(const uint32_t* __restrict__ keys, int n,
                                                  uint32_t* __restrict__ sel, int shift) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t prefix = sel[0], mask = sel[1];
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const uint32_t k = keys[i];
    if ((k & mask) == prefix) atomicAdd(&h[(k >> shift) & 255u], 1u);
  }
  __syncthreads();
  if (h[threadIdx.x]) atomicAdd(&sel[SEL_HIST + threadIdx.x], h[threadIdx.x]);
}

// One block of 256 threads: the bin holding the rank, by an inclusive scan
// of the 256 counts.
__global__ void __launch_bounds__(256) k_sel_pick(uint32_t* __restrict__ sel, int shift) {
  __shared__ uint32_t c[256];
  const int t = threadIdx.x;
  const uint32_t mine = sel[SEL_HIST + t];
  c[t] = mine;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const uint32_t v = t >= o ? c[t - o] : 0u;
    __syncthreads();
    c[t] += v;
    __syncthreads();
  }
  const uint32_t rank = sel[2];
  const uint32_t below = c[t] - mine;  // keys of this prefix in lower bins
  __syncthreads();
  if (below <= rank && rank < c[t]) {
    sel[0] |= (uint32_t)t << shift;
    sel[1] |= 255u << shift;
    sel[2] = rank - below;
    if (shift == 0) sel[3] = sel[0];
  }
  sel[SEL_HIST + t] = 0u;
}

__global__ void __launch_bounds__(256) k_post_scale(const float* __restrict__ img, float gain,
                                                    float* __restrict__ lin, int n3) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n3) lin[i] = img[i] * gain;
}

// Box filter of radius r along x, clamp to edge (post.rs:109-133): thread
// (row, channel) runs the row's sum.
__global__ void __launch_bounds__(128) k_box_h(const float* __restrict__ b, float* __restrict__ out,
                                               int w, int h, int r) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= 3 * h) return;
  const int y = t / 3, c = t - 3 * y;
  const float* row = b + (size_t)y * w * 3 + c;
  float* o = out + (size_t)y * w * 3 + c;
  const float norm = 1.0f / (float)(2 * r + 1);
  float acc = 0.0f;
  const int m = min(r, w - 1);
  for (int i = 0; i <= m; i++) acc = acc + row[3 * i];
  acc = acc + row[0] * (float)r;
  for (int x = 0; x < w; x++) {
    o[3 * x] = acc * norm;
    acc = acc + (row[3 * min(x + r + 1, w - 1)] - row[3 * max(x - r, 0)]);
  }
}

// Along y (post.rs:135-160): thread (column, channel).
__global__ void __launch_bounds__(128) k_box_v(const float* __restrict__ b, float* __restrict__ out,
                                               int w, int h, int r) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= 3 * w) return;
  const size_t stride = (size_t)w * 3;
  const float* col = b + t;
  float* o = out + t;
  const float norm = 1.0f / (float)(2 * r + 1);
  float acc = 0.0f;
  const int m = min(r, h - 1);
  for (int i = 0; i <= m; i++) acc = acc + col[i * stride];
  acc = acc + col[0] * (float)r;
  for (int y = 0; y < h; y++) {
    o[y * stride] = acc * norm;
    acc = acc + (col[min(y + r + 1, h - 1) * stride] - col[max(y - r, 0) * stride]);
  }
}

// ---- the glare filters in shared memory
// A running sum is a chain of dependent additions, one per pixel of a row or
// column; nothing else has to wait.  box_h and box_v wait for two loads from
// L2 at every step (123 and 192 us per filter of a 1280 x 720 image).  Here
// the loads run ahead of the chain, and since the scales are independent,
// one launch does a step of all three (blockIdx.y).
struct GlareScales {
  float* buf[3];
  int r[3];
};
constexpr int GH_ROWS = 2;        // rows per block of glare_h, in one warp's chains
constexpr int GH_THREADS = 128;
constexpr int GH_BATCH = 16;      // loads in flight per thread
constexpr int GV_THREADS = 32;    // columns x channels per block of glare_v
constexpr int GV_GROUP = 16;      // rows per group of copies and of steps
constexpr int GV_DEPTH = 4;       // groups in flight
constexpr size_t GLARE_SMEM = 220 * 1024;

// words per row of glare_h: the row r + 1 pixels in, rounded up to 3 mod 32
// words so that the 6 chains read different banks
__host__ __device__ __forceinline__ int gh_pitch(int w, int r) {
  const int n = 3 * (w + r + 1);
  return (n + 28) / 32 * 32 + 3;
}

// rows of glare_v's ring, a power of two: those of 2 r + 1 steps, of the
// group of steps and of the copies ahead of it
__host__ __device__ __forceinline__ int gv_rows(int r) {
  int n = 64;
  while (n < 2 * r + GV_GROUP * (GV_DEPTH + 3)) n *= 2;
  return n;
}

// Box filter of radius r along x, src -> buf (or in place: src null).  The
// block's rows are staged in shared memory r + 1 pixels to the right of the
// results, so that a result overwrites the pixel whose last use was the step
// before.  Measured: 35 us for the three scales of 1280 x 720
// (their rows are 1.03 times what all SMs hold).
__global__ void __launch_bounds__(GH_THREADS) k_glare_h(const float* __restrict__ img, float gain,
                                                        GlareScales g, int w, int h) {
  extern __shared__ float sm[];
  const int r = g.r[blockIdx.y], pitch = gh_pitch(w, r), off = 3 * (r + 1);
  float* buf = g.buf[blockIdx.y];
  const int y0 = blockIdx.x * GH_ROWS, rows = min(GH_ROWS, h - y0), w3 = 3 * w;
  for (int y = 0; y < rows; y++) {
    const size_t o = (size_t)(y0 + y) * w3;
    float* d = sm + y * pitch + off;
    for (int i0 = threadIdx.x; i0 < w3; i0 += GH_THREADS * GH_BATCH) {
      float v[GH_BATCH];
#pragma unroll
      for (int k = 0; k < GH_BATCH; k++) {
        const int i = i0 + k * GH_THREADS;
        v[k] = i < w3 ? (img ? img[o + i] * gain : buf[o + i]) : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < GH_BATCH; k++)
        if (i0 + k * GH_THREADS < w3) d[i0 + k * GH_THREADS] = v[k];
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < 3 * rows) {
    const int y = threadIdx.x / 3, c = threadIdx.x - 3 * y;
    float* o = sm + y * pitch + c;   // results
    const float* row = o + off;      // pixels
    const float norm = 1.0f / (float)(2 * r + 1);
    float acc = 0.0f;
    const int m = min(r, w - 1);
    for (int i = 0; i <= m; i++) acc = acc + row[3 * i];
    acc = acc + row[0] * (float)r;
    constexpr int U = 16;
    auto step = [&](int x) {
      const float e = row[3 * min(x + r + 1, w - 1)], l = row[3 * max(x - r, 0)];
      o[3 * x] = acc * norm;
      acc = acc + (e - l);
    };
    int x = 0;
    for (; x < min(r, w); x++) step(x);
    // Inside (no clamped index), U steps with every load first.  The loads of
    // a group read pixels x - r .. x + U + r, and its stores end at the place
    // of pixel x + U - 1 - (r + 1): behind every pixel a later step loads.
    for (; x + U + r < w; x += U) {
      const float *pe = row + 3 * (x + r + 1), *pl = row + 3 * (x - r);
      float* po = o + 3 * x;
      float e[U], l[U];
#pragma unroll
      for (int j = 0; j < U; j++) {
        e[j] = pe[3 * j];
        l[j] = pl[3 * j];
      }
#pragma unroll
      for (int j = 0; j < U; j++) {
        po[3 * j] = acc * norm;
        acc = acc + (e[j] - l[j]);
      }
    }
    for (; x < w; x++) step(x);
  }
  __syncthreads();
  for (int y = 0; y < rows; y++) {
    float* o = buf + (size_t)(y0 + y) * w3;
    for (int i = threadIdx.x; i < w3; i += GH_THREADS) o[i] = sm[y * pitch + i];
  }
}

// Box filter of radius r along y, in place: thread per column and channel.
// Every pixel is copied once, asynchronously, into a ring in shared memory
// several groups of rows before it enters the sum, and is read again there
// when it leaves; a result is stored behind the last row copied.  No thread
// reads another's column, so there is no barrier.  Measured: 37 us for the
// three scales of 1280 x 720.
__global__ void __launch_bounds__(GV_THREADS) k_glare_v(GlareScales g, int w, int h) {
  extern __shared__ float sm[];
  const int t = blockIdx.x * GV_THREADS + threadIdx.x;
  if (t >= 3 * w) return;
  const int r = g.r[blockIdx.y], mask = gv_rows(r) - 1;
  const size_t stride = (size_t)w * 3;
  float* col = g.buf[blockIdx.y] + t;
  float* ring = sm + threadIdx.x;  // row i of the image at (i & mask) * GV_THREADS
  const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring);
  const int groups = (h + GV_GROUP - 1) / GV_GROUP;
  auto issue = [&](int k) {
    if (k < groups) {
      const float* p = col + (size_t)k * GV_GROUP * stride;
#pragma unroll
      for (int j = 0; j < GV_GROUP; j++) {
        const int i = k * GV_GROUP + j;
        if (i < h)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                           ring_a + (uint32_t)((i & mask) * GV_THREADS * 4)),
                       "l"(p + j * stride)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // step y: row min(y + r + 1, h - 1) enters and max(y - r, 0) leaves
  const float norm = 1.0f / (float)(2 * r + 1);
  float acc = 0.0f;
  int kk = (GV_GROUP + r) / GV_GROUP;  // the group of the last row a group of steps needs
  for (int k = 0; k < kk + GV_DEPTH; k++) issue(k);
  for (int y0 = 0; y0 < h; y0 += GV_GROUP, kk++) {
    issue(kk + GV_DEPTH);
    asm volatile("cp.async.wait_group %0;" ::"n"(GV_DEPTH) : "memory");  // groups 0 .. kk are in
    if (y0 == 0) {
      const int m = min(r, h - 1);
      for (int i = 0; i <= m; i++) acc = acc + ring[(i & mask) * GV_THREADS];
      acc = acc + ring[0] * (float)r;
    }
    float e[GV_GROUP], l[GV_GROUP];
#pragma unroll
    for (int j = 0; j < GV_GROUP; j++) {
      e[j] = ring[(min(y0 + j + r + 1, h - 1) & mask) * GV_THREADS];
      l[j] = ring[(max(min(y0 + j, h - 1) - r, 0) & mask) * GV_THREADS];
    }
    float* o = col + (size_t)y0 * stride;
#pragma unroll
    for (int j = 0; j < GV_GROUP; j++) {
      if (y0 + j < h) {
        o[j * stride] = acc * norm;
        acc = acc + (e[j] - l[j]);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// g = g + b * weight (the glare's sum over scales, post.rs:100-104)
__global__ void __launch_bounds__(256) k_post_axpy(const float* __restrict__ b, float wt,
                                                   float* __restrict__ g, int n3) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n3) g[i] = g[i] + b[i] * wt;
}

__device__ __forceinline__ float aces(float x) {
  x = x * 0.6f;
  const float num = x * (2.51f * x + 0.03f);
  const float den = x * (2.43f * x + 0.59f) + 0.14f;
  return fminf(fmaxf(num / den, 0.0f), 1.0f);
}
__device__ __forceinline__ float srgb(float x) {
  return x <= 0.0031308f ? 12.92f * x : 1.055f * powf(x, 1.0f / 2.4f) - 0.055f;
}
// PCG hash of the pixel index to [0, 1) with 24 bits (post.rs:83-88)
__device__ __forceinline__ float hash01(uint32_t v) {
  uint32_t x = v * 747796405u + 2891336453u;
  x = ((x >> ((x >> 28u) + 4u)) ^ x) * 277803737u;
  x = (x >> 22u) ^ x;
  return (float)(x >> 8u) / 16777216.0f;
}

// The three scales' weighted sum and the mix, from the filters' own buffers.
__global__ void __launch_bounds__(256) k_post_final3(const float* __restrict__ img, float gain,
                                                     GlareScales g, float w0, float w1, float w2,
                                                     float glare, uint8_t* __restrict__ out,
                                                     float* __restrict__ lin_out, int n) {
  const int p = blockIdx.x * 256 + threadIdx.x;
  if (p >= n) return;
  const float dith = (hash01((uint32_t)p) - 0.5f) / 255.0f;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int i = 3 * p + c;
    float gl = 0.0f + g.buf[0][i] * w0;
    gl = gl + g.buf[1][i] * w1;
    gl = gl + g.buf[2][i] * w2;
    const float v = (img[i] * gain) * (1.0f - glare) + gl * glare;
    if (lin_out) lin_out[i] = v;
    const float s = srgb(aces(v)) + dith;
    out[i] = (uint8_t)(fminf(fmaxf(s, 0.0f), 1.0f) * 255.0f + 0.5f);
  }
}

__global__ void __launch_bounds__(256) k_post_final(const float* __restrict__ lin,
                                                    const float* __restrict__ gl, float glare,
                                                    uint8_t* __restrict__ out,
                                                    float* __restrict__ lin_out, int n) {
  const int p = blockIdx.x * 256 + threadIdx.x;
  if (p >= n) return;
  const float dith = (hash01((uint32_t)p) - 0.5f) / 255.0f;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    float v = lin[3 * p + c];
    if (glare > 0.0f) v = v * (1.0f - glare) + gl[3 * p + c] * glare;
    if (lin_out) lin_out[3 * p + c] = v;
    const float s = srgb(aces(v)) + dith;
    out[3 * p + c] = (uint8_t)(fminf(fmaxf(s, 0.0f), 1.0f) * 255.0f + 0.5f);
  }
}

inline unsigned blocks(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t launch_post_select(const float* accum, int n, int k, float* img, uint32_t* keys,
                               uint32_t* sel, cudaStream_t st) {
  k_post_mean<<<blocks(n, 256), 256, 0, st>>>(reinterpret_cast<const float4*>(accum), img, keys,
                                               n);
  k_sel_init<<<1, 256, 0, st>>>(sel, (uint32_t)k);
  const unsigned hb = std::min(blocks(n, 256), 1184u);
  for (int shift = 24; shift >= 0; shift -= 8) {
    k_sel_hist<<<hb, 256, 0, st>>>(keys, n, sel, shift);
    k_sel_pick<<<1, 256, 0, st>>>(sel, shift);
  }
  return cudaGetLastError();
}

float post_key_value(uint32_t key) {
  const uint32_t u = (key & 0x80000000u) ? (key & 0x7FFFFFFFu) : ~key;
  float v;
  std::memcpy(&v, &u, 4);
  return v;
}

cudaError_t launch_post_develop(const float* img, int w, int h, float gain, float glare,
                                float* scratch, uint8_t* out, float* lin_out, cudaStream_t st) {
  const long n = (long)w * h, n3 = 3 * n;
  // (radius as a fraction of the width, weight), post.rs:93
  const float scales[3][2] = {{0.003f, 0.5f}, {0.012f, 0.3f}, {0.04f, 0.2f}};
  if (glare > 0.0f) {
    GlareScales g;
    size_t sh = 0, sv = 0;
    for (int k = 0; k < 3; k++) {
      g.buf[k] = scratch + (k + 1) * n3;
      g.r[k] = std::max((int)(scales[k][0] * (float)w), 1);
      sh = std::max(sh, (size_t)gh_pitch(w, g.r[k]) * std::min(h, GH_ROWS) * 4);
      sv = std::max(sv, (size_t)gv_rows(g.r[k]) * GV_THREADS * 4);
    }
    if (sh <= GLARE_SMEM && sv <= GLARE_SMEM) {
      cudaError_t e = cudaFuncSetAttribute(k_glare_h, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)GLARE_SMEM);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_glare_v, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)GLARE_SMEM);
      if (e != cudaSuccess) return e;
      const dim3 gh(blocks(h, GH_ROWS), 3), gv(blocks(3L * w, GV_THREADS), 3);
      for (int it = 0; it < 3; it++) {
        k_glare_h<<<gh, GH_THREADS, sh, st>>>(it == 0 ? img : nullptr, gain, g, w, h);
        k_glare_v<<<gv, GV_THREADS, sv, st>>>(g, w, h);
      }
      k_post_final3<<<blocks(n, 256), 256, 0, st>>>(img, gain, g, scales[0][1], scales[1][1],
                                                    scales[2][1], glare, out, lin_out, (int)n);
      return cudaGetLastError();
    }
  }
  float* lin = scratch;
  float* t1 = scratch + n3;
  float* t2 = scratch + 2 * n3;
  float* gl = scratch + 3 * n3;
  k_post_scale<<<blocks(n3, 256), 256, 0, st>>>(img, gain, lin, (int)n3);
  if (glare > 0.0f) {
    cudaError_t e = cudaMemsetAsync(gl, 0, n3 * 4, st);
    if (e != cudaSuccess) return e;
    for (const auto& sw : scales) {
      const int rad = std::max((int)(sw[0] * (float)w), 1);
      const float* src = lin;
      for (int it = 0; it < 3; it++) {
        k_box_h<<<blocks(3L * h, 128), 128, 0, st>>>(src, t1, w, h, rad);
        k_box_v<<<blocks(3L * w, 128), 128, 0, st>>>(t1, t2, w, h, rad);
        src = t2;
      }
      k_post_axpy<<<blocks(n3, 256), 256, 0, st>>>(t2, sw[1], gl, (int)n3);
    }
  }
  k_post_final<<<blocks(n, 256), 256, 0, st>>>(lin, gl, glare, out, lin_out, (int)n);
  return cudaGetLastError();
}

}  // namespace pyro
