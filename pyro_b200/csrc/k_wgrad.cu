// k_wgrad.cu — weight gradient of the 3x3x3 convolutions on the tcgen05
// tensor cores with TMA-staged operands.
//
//   dw[co][(dz, dy, dx)][ci] += sum_u x[u + (dy, dz)][ci] * g[u - dx][co]
//
// (u runs over the rows' positions, x and g are zero outside their volume),
// so the taps along y and z are shifts of the input and the taps along x are
// shifts of the output gradient.  As a matrix product the sum over voxels is
// K, the rows (M) are (dy, dz, input channel) and the columns (N) are (dx,
// output channel): 27 ci co sums in ceil(9 ci / 128) x (3 co) tiles.
//
// Both operands are MN-major (channels contiguous, K = voxels), which is how
// activations lie in memory: planes of 8 channels, 16 bytes per voxel, so 8
// consecutive voxels of a row are one 128-byte core matrix.  A stage holds,
// for a tile of BX x BY voxels of one z-plane,
//   x  [BY + 2 rows y][3 planes z][P channel planes][BX voxels]  (one box)
//   g  [BY rows y][ndx shifts][Q channel planes][BX voxels]      (a box per
//      row and shift; the tensor map's zero fill is the row's end)
// so that for every output row the 9 P core-matrix rows of (dy, dz, plane)
// follow one another at the stride of a row: an M tile is 16 of them at a
// uniform stride, no gather, and the rows past 9 P (the next rows' data)
// only feed rows of D that are never read.
//
// What bounds it: an MMA of 128 x 48 x 16 takes 45 cycles (measured; 128
// rows of A cost 32 cycles of shared-memory reads whatever N is), so 16 -> 16
// channels need 5.8 cycles per voxel and SM; the kernel issues one every 54.
// Measured on two 128^3 volumes: 16 -> 16 channels 16.4 ms -> 0.12 ms, 48 ->
// 16 47 ms -> 0.24 ms (before: each thread gathered its operand rows with
// 2-byte loads), all nine layers of the network 81 -> 0.92 ms.
//
// At the volume's edges values of x that belong to no tap meet the zeros
// outside it (u = 0 and g[-1], a tile's rows past ny), and zero times Inf or
// NaN is NaN.  A CTA that drains a sum that is not finite sets *bad, and the
// caller takes the gradient from the gather GEMM (k_conv.cu), whose products
// are those of the pairs inside the volume.
//
// The CTAs share the tiles round robin; each takes its own in turn into as many
// accumulators as the TMEM holds, and adds their sums to dw, in FP64, once.  A
// sum's error grows with the MMAs that add to it (1.8e-8 of it for each on
// normal inputs: 16 -> 16 channels on two 128^3 volumes 3.2e-5 with one
// accumulator of 1,771, 6.1e-6 with five), so no accumulator takes more of them
// than one of the gather GEMM's (k_conv.cu), whose error that bounds: past it
// there are more CTAs than SMs.  Warp 0 loads, warp 1 issues the MMAs, all four
// drain the sums.  Every wait is bounded; one that runs out sets *err, the
// copies in flight land (bounded again) and the TMEM is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cfloat>

#include "net.h"
#include "umma.cuh"

namespace pyro {

namespace {

using bf16 = __nv_bfloat16;

constexpr int WG_THREADS = 128;
constexpr int WG_MAX_STAGES = 8;
constexpr uint32_t WG_SMEM = 222u * 1024u;  // stages; + 1 KB of alignment

struct WgGeom {
  int nz, BX, BY, tiles_x, tiles_y, ntiles;
  int P, Q, ndx;        // planes of x and of g per CTA, x-shifts of g
  int mt, N;            // M tiles, columns
  int Cin, Cout;        // of dw
  int pack;             // 0; 1: g's channel is the x-shift; 2: x's channels are (x-shift, ci)
  int stages;
  int nacc;             // accumulators, taken in turn
  uint32_t xbytes, stage_bytes, ncols;
};

// MN-major operand without swizzle: core matrices of 8 voxels x 8 channels
// (128 bytes); SBO (the high word) = next 8 channels, LBO = next 8 voxels.
// The low word holds the address in 16-byte units, so an operand further on
// in shared memory is the same descriptor plus a constant.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) {
  return (saddr >> 4) | ((128u >> 4) << 16);
}
__device__ __forceinline__ uint64_t desc(uint32_t hi, uint32_t lo) {
  return ((uint64_t)hi << 32) | lo;
}

// MT: M tiles; KS: K steps of 16 voxels in a row.  Both are compile-time so
// that a row's MMAs are one unrolled run: with loops around single MMAs the
// issuing thread took 170 cycles for each (322 us for 16 -> 16 channels on
// two 128^3 volumes, 115 us unrolled).
template <int MT, int KS>
__global__ void __launch_bounds__(WG_THREADS, 1)
    k_wgrad_tma(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tg,
                WgGeom g, double* __restrict__ dw, int* err, int* bad) {
  extern __shared__ uint8_t dsm[];
  __shared__ __align__(8) uint64_t full[WG_MAX_STAGES], empty[WG_MAX_STAGES], done;
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  uint8_t* base = dsm + ((1024u - (umma::smem_u32(dsm) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.stages;
  const int p0 = blockIdx.y * g.P, q0 = blockIdx.z * g.Q;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    umma::mbar_init(&done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    umma::tmem_alloc(&tslot, g.ncols);
    umma::tmem_relinquish();
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  const uint32_t tbase = tslot;
  const int my_tiles =
      (int)blockIdx.x < g.ntiles ? (g.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const uint32_t row = 256u * KS;  // bytes of a row of BX = 16 KS voxels
  bool ok = true;
  if (warp == 0) {
    // ---- loads: a lane per box of g (y, shift), lane 31 the box of x
    const int ly = lane / g.ndx, lj = lane - ly * g.ndx;
    const bool mine = lane < g.BY * g.ndx;
    const int shift = g.ndx == 3 ? 1 - lj : 0;  // copy j holds g[u - (j - 1)]
    // the tile's place, stepped by gridDim.x tiles with carries
    int tix = (int)blockIdx.x, tiy, tiz, tib;
    int sx_ = (int)gridDim.x, sy_, sz_, sb_;
    tiy = tix / g.tiles_x, tix -= tiy * g.tiles_x;
    tiz = tiy / g.tiles_y, tiy -= tiz * g.tiles_y;
    tib = tiz / g.nz, tiz -= tib * g.nz;
    sy_ = sx_ / g.tiles_x, sx_ -= sy_ * g.tiles_x;
    sz_ = sy_ / g.tiles_y, sy_ -= sz_ * g.tiles_y;
    sb_ = sz_ / g.nz, sz_ -= sb_ * g.nz;
    int s = 0, issued = 0;
    uint32_t phase = 1u;
    for (int i = 0; i < my_tiles; i++) {
      if (abort_flag) break;
      if (i >= S && !umma::mbar_wait_warp(&empty[s], phase)) {
        ok = false;
        break;
      }
      uint8_t* sx = base + (size_t)s * g.stage_bytes;
      if (lane == 0) umma::mbar_expect_tx(&full[s], g.stage_bytes);
      __syncwarp();
      const int x0 = tix * (16 * KS), y0 = tiy * g.BY;
      if (lane == 31)
        umma::tma_load_5d(sx, &tx, x0 * 4, p0, tiz - 1, y0 - 1, tib, &full[s]);
      else if (mine)
        umma::tma_load_5d(sx + g.xbytes + (uint32_t)(lane * g.Q) * row, &tg, (x0 + shift) * 4, q0,
                          tiz, y0 + ly, tib, &full[s]);
      issued = i + 1;
      if (++s == S) s = 0, phase ^= 1u;
      tix += sx_, tiy += sy_, tiz += sz_, tib += sb_;
      if (tix >= g.tiles_x) tix -= g.tiles_x, tiy++;
      if (tiy >= g.tiles_y) tiy -= g.tiles_y, tiz++;
      if (tiz >= g.nz) tiz -= g.nz, tib++;
    }
    if (!ok) abort_flag = 1;
    // every issued copy lands before the CTA may exit
    for (int q = issued > S ? issued - S : 0; q < issued; q++)
      if (!umma::mbar_wait_warp(&full[q % S], (q / S) & 1)) ok = false;
  } else if (warp == 1) {
    // ---- MMAs
    const uint32_t idesc = umma::idesc_bf16(128, g.N) | (1u << 15) | (1u << 16);
    const uint32_t hi = (row >> 4) | (1u << 14);
    const uint32_t xrow = 3u * (uint32_t)g.P * row >> 4;       // x rows per y
    const uint32_t grow = (uint32_t)(g.ndx * g.Q) * row >> 4;  // g rows per y
    constexpr uint32_t MSTEP = 16u * KS * 16u;                 // 16 rows of x
    const uint32_t ncol = (uint32_t)g.N;
    const uint32_t sums = (uint32_t)(MT * g.N);  // columns of an accumulator
    uint32_t phase = 0u;
    int s = 0, a = 0;
    for (int i = 0; i < my_tiles; i++) {
      if (abort_flag) break;
      if (!umma::mbar_wait_warp(&full[s], phase)) {
        ok = false;
        break;
      }
      umma::fence_after();
      const uint32_t sx = umma::smem_u32(base) + (uint32_t)s * g.stage_bytes;
      uint32_t ax = desc_lo(sx), bg = desc_lo(sx + g.xbytes);
      uint32_t acc = i < g.nacc ? 0u : 1u;
      const uint32_t dt = tbase + (uint32_t)a * sums;
#pragma unroll 1
      for (int y = 0; y < g.BY; y++) {
        if (umma::elect_one()) {
#pragma unroll
          for (int k = 0; k < KS; k++)
#pragma unroll
            for (int m = 0; m < MT; m++)
              umma::mma_bf16(dt + m * ncol, desc(hi, ax + k * 16u + m * MSTEP),
                             desc(hi, bg + k * 16u), idesc, k ? 1u : acc);
        }
        acc = 1u;
        ax += xrow;
        bg += grow;
      }
      if (umma::elect_one()) umma::mma_commit(&empty[s]);
      if (++s == S) s = 0, phase ^= 1u;
      if (++a == g.nacc) a = 0;
    }
    if (!ok) abort_flag = 1;
    // every MMA issued has finished before the sums are read
    if (umma::elect_one()) umma::mma_commit(&done);
    if (!umma::mbar_wait_warp(&done, 0)) ok = false;
  }
  const bool all_ok = __syncthreads_and(ok) != 0;
  umma::fence_after();
  if (!all_ok && threadIdx.x == 0) atomicExch(err, 1);
  if (all_ok && my_tiles > 0) {
    float top = 0.0f;  // the largest |sum|; NaN stays
    for (int m = 0; m < MT; m++) {
      // row of D: core matrix r >> 3 = (dy * 3 + dz) * P + plane, channel r & 7
      const int r = m * 128 + warp * 32 + lane;
      const int i = r >> 3, q = i / g.P, pl = i - q * g.P;
      const bool own = q < 9;
      const int dy = q / 3, dz = q - 3 * dy;
      const int c8 = (p0 + pl) * 8 + (r & 7);
      for (int col = 0; col < g.N; col += 16) {
        const uint32_t tv = tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(m * g.N + col);
        float v[16];
        umma::tmem_ld16(tv, v);
        for (int a = 1; a < min(g.nacc, my_tiles); a++) {
          float t[16];
          umma::tmem_ld16(tv + (uint32_t)(a * MT * g.N), t);
#pragma unroll
          for (int e = 0; e < 16; e++) v[e] += t[e];
        }
        if (!own) continue;
#pragma unroll
        for (int e = 0; e < 16; e++)
          asm("max.NaN.f32 %0, %0, %1;" : "+f"(top) : "f"(fabsf(v[e])));
#pragma unroll
        for (int e = 0; e < 16; e++) {
          const int n = col + e;
          int dx, co, ci;
          if (g.pack == 1) {  // g's channels are the shifts of its one channel
            dx = n;
            co = 0;
            ci = c8;
            if (n >= 3) continue;
          } else if (g.pack == 2) {  // x's channels are (shift, channel)
            dx = c8 / g.Cin;
            ci = c8 - dx * g.Cin;
            co = q0 * 8 + n;
            if (dx >= 3) continue;
          } else {
            dx = n / (8 * g.Q);
            co = q0 * 8 + n - dx * 8 * g.Q;
            ci = c8;
          }
          if (co < g.Cout && ci < g.Cin)
            atomicAdd(dw + ((size_t)co * 27 + (dz * 3 + dy) * 3 + dx) * g.Cin + ci, (double)v[e]);
        }
      }
    }
    if (!(top <= FLT_MAX)) *bad = 1;
  }
  umma::fence_before();
  __syncthreads();
  if (warp == 1) umma::tmem_dealloc(tbase, g.ncols);
}

// Planes of 8 channels [planes][nb][nz][ny][nx][8] as (x, plane, z, y, b),
// the order in which a box's rows follow one another in shared memory.
bool encode_planes(CUtensorMap* m, const bf16* p, int planes, int nx, int ny, int nz, int nb,
                   int bx, int bp, int bz, int by) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = (PFN_cuTensorMapEncodeTiled_v12000)tensor_map_encoder();
  if (!enc) return false;
  // as 32-bit elements, four per voxel: a box row may hold 256 elements
  const cuuint64_t plane = (cuuint64_t)nx * 16, vol = plane * ny * nz;
  const cuuint64_t dim[5] = {(cuuint64_t)nx * 4, (cuuint64_t)planes, (cuuint64_t)nz,
                             (cuuint64_t)ny, (cuuint64_t)nb};
  const cuuint64_t str[4] = {vol * nb, plane * ny, plane, vol};
  const cuuint32_t box[5] = {(cuuint32_t)(4 * bx), (cuuint32_t)bp, (cuuint32_t)bz,
                             (cuuint32_t)by, 1};
  const cuuint32_t es[5] = {1, 1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 5, const_cast<bf16*>(p), dim, str, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// conv3_pack_grad and conv3_pack_input: T is a voxel, one or two channels.
template <typename T>
__global__ void __launch_bounds__(256) k_pack_dx(const T* __restrict__ src, size_t V, int nx,
                                                 uint4* __restrict__ dst) {
  const size_t u = blockIdx.x * (size_t)256 + threadIdx.x;
  if (u >= V) return;
  const int x = (int)((uint32_t)u % (uint32_t)nx);
  const uint32_t left = x > 0 ? src[u - 1] : 0u, mid = src[u],
                 right = x + 1 < nx ? src[u + 1] : 0u;
  dst[u] = sizeof(T) == 2 ? make_uint4(right | mid << 16, left, 0u, 0u)
                          : make_uint4(left, mid, right, 0u);
}

}  // namespace

// Channel counts of the TMA form: planes of 8 input channels and pairs of
// planes of output channels (N a multiple of 16).
bool conv3_wgrad_fits(int Cin, int Cout) { return Cin % 8 == 0 && Cout % 16 == 0; }

cudaError_t conv3_pack_grad(const bf16* src, int nx, int ny, int nz, int nb, bf16* dst,
                            cudaStream_t st) {
  const size_t V = (size_t)nx * ny * nz * nb;
  k_pack_dx<<<(unsigned)((V + 255) / 256), 256, 0, st>>>((const uint16_t*)src, V, nx, (uint4*)dst);
  return cudaGetLastError();
}
cudaError_t conv3_pack_input(const bf16* src, int nx, int ny, int nz, int nb, bf16* dst,
                             cudaStream_t st) {
  const size_t V = (size_t)nx * ny * nz * nb;
  k_pack_dx<<<(unsigned)((V + 255) / 256), 256, 0, st>>>((const uint32_t*)src, V, nx, (uint4*)dst);
  return cudaGetLastError();
}

cudaError_t conv3_wgrad_tma(const bf16* x, int Cin, const bf16* gr, int Cout, int pack, int nx,
                            int ny, int nz, int nb, double* dw, int* err, int* bad,
                            cudaStream_t st) {
  WgGeom g{};
  g.nz = nz;
  g.Cin = Cin;
  g.Cout = Cout;
  g.pack = pack;
  g.ndx = pack ? 1 : 3;
  const int planes_x = pack == 2 ? 1 : Cin / 8, planes_g = pack == 1 ? 1 : Cout / 8;
  // one channel of g (pack 1) is a box of two planes, the second past the
  // tensor's end and so zero: N has to be a multiple of 16
  g.Q = planes_g % 4 == 0 && !pack ? 4 : 2;
  g.N = g.ndx * g.Q * 8;
  // The most planes of x per CTA whose sums fit the TMEM and of which three
  // stages (or two) fit the shared memory; then, of the widths that pad the
  // rows least, 64 voxels where that leaves four rows (a tile of BY rows
  // loads (BY + 2) / BY of x, and a box of g costs the same for any width:
  // 16 -> 16 channels 107 us against 140 with 32), else the tallest tile of
  // the widest (48 -> 16: 243 us with 32 x 4, 294 with 64 x 1).
  // MMAs that an accumulator takes at most: the gather GEMM's, or 8, whose error
  // is below that of its additions of more CTAs' sums in FP32
  const long V = (long)nx * ny * nz * nb;
  const int most = std::max(conv3_gather_steps(Cin, V), 8);
  bool found = false;
  for (int P = std::min(planes_x, 8); P >= 1 && !found; P--) {
    if (planes_x % P) continue;
    const int mt = (9 * P + 15) / 16;
    if (mt * g.N > 512) continue;
    for (int want : {3, 2}) {
      int best = 0;
      for (int BX : {64, 32, 16}) {
        if ((nx + BX - 1) / BX * BX > (nx + 15) / 16 * 16) continue;
        const uint32_t row = (uint32_t)BX * 16u;
        // the last M tile reads (16 mt - 9 P) rows past a tile's last row of
        // x: into the stage's g and the slack after the last stage
        const uint32_t slack = (uint32_t)(16 * mt - 9 * P) * row;
        for (int BY : {8, 4, 2, 1}) {
          if (BY > 1 && (BY / 2 >= ny || BY * (BX / 16) > most)) continue;
          const uint32_t xb = (uint32_t)((BY + 2) * 3 * P) * row;
          const uint32_t sb = xb + (uint32_t)(BY * g.ndx * g.Q) * row;
          if (slack >= WG_SMEM || (WG_SMEM - slack) / sb < (uint32_t)want) continue;
          if (std::min(BY, 4) > best) {
            best = std::min(BY, 4);
            g.P = P;
            g.mt = mt;
            g.BX = BX;
            g.BY = BY;
            g.xbytes = xb;
            g.stage_bytes = sb;
            g.stages = (int)std::min<uint32_t>(WG_MAX_STAGES, (WG_SMEM - slack) / sb);
          }
          break;
        }
      }
      if (best) {
        found = true;
        break;
      }
    }
  }
  if (!found) return cudaErrorInvalidValue;
  g.nacc = std::min(512 / (g.mt * g.N), 16);
  g.ncols = 32;
  while ((int)g.ncols < g.nacc * g.mt * g.N) g.ncols *= 2;
  g.tiles_x = (nx + g.BX - 1) / g.BX;
  g.tiles_y = (ny + g.BY - 1) / g.BY;
  const long nt = (long)g.tiles_x * g.tiles_y * nz * nb;
  if (nt >= (1l << 31)) return cudaErrorInvalidValue;
  g.ntiles = (int)nt;
  CUtensorMap mx, mg;
  if (!encode_planes(&mx, x, planes_x, nx, ny, nz, nb, g.BX, g.P, 3, g.BY + 2) ||
      !encode_planes(&mg, gr, planes_g, nx, ny, nz, nb, g.BX, g.Q, 1, 1))
    return cudaErrorInvalidValue;
  const size_t smem = WG_SMEM + 1024;
  using Kern = void (*)(CUtensorMap, CUtensorMap, WgGeom, double*, int*, int*);
  static constexpr Kern kerns[5][3] = {
      {k_wgrad_tma<1, 1>, k_wgrad_tma<1, 2>, k_wgrad_tma<1, 4>},
      {k_wgrad_tma<2, 1>, k_wgrad_tma<2, 2>, k_wgrad_tma<2, 4>},
      {k_wgrad_tma<3, 1>, k_wgrad_tma<3, 2>, k_wgrad_tma<3, 4>},
      {k_wgrad_tma<4, 1>, k_wgrad_tma<4, 2>, k_wgrad_tma<4, 4>},
      {k_wgrad_tma<5, 1>, k_wgrad_tma<5, 2>, k_wgrad_tma<5, 4>}};
  if (g.mt > 5) return cudaErrorInvalidValue;
  const Kern kern = kerns[g.mt - 1][g.BX / 32];
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int gy = planes_x / g.P, gz = std::max(planes_g / g.Q, 1);
  const int per = g.nacc * std::max(1, most / (g.BY * (g.BX / 16)));  // tiles of a CTA at most
  const int ctas = std::max({1, std::min(g.ntiles, nsm / (gy * gz)), (g.ntiles + per - 1) / per});
  kern<<<dim3((unsigned)ctas, (unsigned)gy, (unsigned)gz), WG_THREADS, smem, st>>>(
      mx, mg, g, dw, err, bad);
  return cudaGetLastError();
}

}  // namespace pyro
