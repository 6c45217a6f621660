// k_conv3.cu — 3x3x3 convolutions (padding 1, stride 1) on the tcgen05 tensor
// cores with TMA-staged inputs: the forward pass and, on flipped and
// transposed weights, the data gradient.
//
//   D[voxel][(zo, co)] = sum over (zi, dy, dx, ci) of
//       x[voxel + (zi - 1, dy - 1, dx - 1)][ci] * w[zi - zo][dy][dx][co][ci]
//
// A tile is 8 x 16 voxels of x and y (M = 128) by ZO planes of z.  Its ZO
// output planes are columns of the product (N = ZO co): an input plane zi
// feeds the output planes zi - 2 .. zi at once, with the tap zi - zo as the
// weight of plane zo and zero where that is no tap.  That costs (ZO + 2) / 3
// ZO of the products a dense form would need, and pays because a narrow MMA
// does not run faster: with both operands in shared memory 128 x N x 16 takes
// max(45, 32 + N / 4, N / 2) cycles (measured: 45 for N = 16 and 32, 48 for
// 64, 64 for 128), so 16 channels need 27 x 45 cycles per 128 voxels plane by
// plane and 54 x 48 per 512 with ZO = 4.
//
// A zero weight times an input that is not finite is NaN, which such an input
// would spread over all of the tile's planes.  So a tile whose sums are not
// all finite is done again at the end, plane by plane with the 27 taps alone
// (N = co): the sums of the same products in the same order, and so the bits
// of a volume without it outside the 27 neighbours of such a voxel.  (Windows
// of three planes' columns would need no zeros, but MMAs on overlapping
// columns are ordered only where accumulator and shape are the same.)
//
//  * x: a stage holds 16 input channels: [2 chunks of 8 channels][ZO + 2
//    planes][18 rows][10 voxels], a box per chunk and plane, zero-filled
//    outside the volume.  Rows of A are (y, x): core matrices of 8 voxels,
//    160 bytes (a row of the box) apart, so that every tap is the same descriptor at another start:
//    no gather and no copy per tap.
//  * w: resident in shared memory for the whole kernel, per tap (dy, dx) as
//    the rows [zero planes][tap 2][tap 1][tap 0][zero planes] of co channels:
//    the N rows for input plane zi are the window that starts at plane
//    ZO + 1 - zi.  co is padded to 16 with zero rows.  The block writes it once
//    from the tap-major weights.
//  * a packed input (one plane of 8 channels that holds the three x-shifts of
//    a 1-channel tensor): the taps along x are channels,
//    the box has no x halo, and a K step of 16 is two rows y (the tap pairs
//    (0, 1) and (-, 2), the missing one with zero weights).
//
// Persistent and warp-specialised: warp 0 loads, warp 1 issues the MMAs into
// one of two accumulators, warps 2-9 drain the other (a lane is a voxel, so
// 8 channels are one 16-byte store beside its neighbours').  Loops that issue
// run warp-wide around elect_one (see umma.cuh).  Every wait is bounded; one
// that runs out stops the CTA's roles, sets *err, lets the copies in flight
// land and frees the TMEM.
//
// Measured on 160 x 320 x 160 voxels against the form this replaces (output
// channels as the MMA's 128 rows, of which 16 to 64 were used, and three
// shifted copies of x), in us: 16 -> 16 773 -> 255, 48 -> 16 1990 -> 612; on
// 80 x 160 x 80, 96 -> 32 522 -> 382 with the up-sampled store; the data
// gradient 16 -> 48 on two 128^3 volumes 1411 -> 404 (the test for sums that
// are not finite costs 2 to 8 % of it).  What bounds it now: the boxes' rows
// (16 cycles for 160 bytes: 48 -> 16 0.59 ms at 1.9 GHz) ahead of the MMAs'
// issue (54 of 48 cycles per 512 voxels and group, 0.44 ms); copying the input
// with cp.async from four warps was slower (684 us against 598).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "conv.cuh"
#include "net.h"
#include "umma.cuh"

namespace pyro {

namespace {

constexpr int C3_EPI = 8;  // epilogue warps
constexpr int C3_THREADS = 64 + 32 * C3_EPI;
constexpr int C3_MAX_STAGES = 8;
constexpr int C3_MAX_CO = 128;
constexpr uint32_t C3_SMEM = 224u * 1024u;
constexpr int C3_REDO = 256;  // words of the bit field of tiles to do again
constexpr int TX = 8, TY = 16;  // voxels of a tile along x and y

struct C3Geom {
  int nx, ny, nz, nb, tiles_x, tiles_y, tiles_z, ntiles;
  int groups, stages;    // groups of 16 input channels
  int K, CO, N, rb;      // input channels of w, channels per CTA (a multiple of 16), columns,
                         // rows of a weight tap
  int late_w;            // the kernel before may have written the weights
  uint32_t wbytes, ncols;
};

// max of `top` and |v|, NaN if one is NaN
__device__ __forceinline__ float max_abs(const float (&v)[16], float top) {
#pragma unroll
  for (int e = 0; e < 16; e += 2)
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(fabsf(v[e])), "f"(fabsf(v[e + 1])));
  return top;
}

template <int ZO, bool PACK>
__global__ void __launch_bounds__(C3_THREADS, 1)
    k_conv3(const __grid_constant__ CUtensorMap tx, const bf16* __restrict__ w_tap, C3Geom g,
            ConvEpi ep, int* err) {
  constexpr int ZI = ZO + 2;
  constexpr int PX = PACK ? TX : TX + 2;               // voxels per row of the box
  constexpr uint32_t ROW = PX * 16u, BOX = ROW * (TY + 2),
                     PLANE = (BOX + 127u) & ~127u, CHUNK = PLANE * ZI;
  constexpr int TAPS = PACK ? 2 : 9;                   // K steps per input plane
  constexpr int CHUNKS = PACK ? 1 : 2;
  constexpr uint32_t STAGE = CHUNK * CHUNKS;
  extern __shared__ uint8_t dsm[];
  __shared__ __align__(8) uint64_t full[C3_MAX_STAGES], empty[C3_MAX_STAGES], accf[2], acce[2],
      done;
  __shared__ __align__(16) float sbias[C3_MAX_CO];
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  __shared__ uint32_t redo[C3_REDO], redo_any;
  uint8_t* base = dsm + ((128u - (umma::smem_u32(dsm) & 127u)) & 127u);
  uint8_t* stages = base + g.wbytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.stages, G = g.groups;
  const int co0 = blockIdx.y * g.CO;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      umma::mbar_init(&accf[a], 1);
      umma::mbar_init(&acce[a], C3_EPI);
    }
    umma::mbar_init(&done, 1);
    abort_flag = 0;
    redo_any = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    umma::tmem_alloc(&tslot, g.ncols);
    umma::tmem_relinquish();
    // Only now: a CTA of the next launch on this SM allocates TMEM before it
    // waits for this launch, so this one must hold its own already.
    pdl_trigger();
  }
  if (g.late_w) pdl_wait();
  // ---- weights: [group][K step][chunk][row of rb][8 channels]; row = plane
  // * CO + co, plane p holding tap z = ZO + 1 - p where that is 0, 1 or 2
  for (int c = threadIdx.x; c < C3_REDO; c += C3_THREADS) redo[c] = 0u;
  for (int c = threadIdx.x; c < C3_MAX_CO; c += C3_THREADS)
    sbias[c] = (ep.bias && c < g.CO && co0 + c < ep.Nout) ? ep.bias[co0 + c] : 0.0f;
  const int rows = G * TAPS * 2 * g.rb;
  for (int i = threadIdx.x; i < rows; i += C3_THREADS) {
    int r = i / g.rb;
    const int row = i - r * g.rb;
    const int j = r & 1;
    r >>= 1;
    const int grp = r / TAPS, t = r - grp * TAPS;
    const int p = row / g.CO, c = row - p * g.CO, tz = ZO + 1 - p, co = co0 + c;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (tz >= 0 && tz < 3 && co < ep.Nout) {
      if constexpr (PACK) {
        // K step t, chunk j: row y = t + j; step 1's first chunk has no tap
        const int dy = t + j;
        if (t == 0 || j == 1) {
          bf16* e = reinterpret_cast<bf16*>(&v);
          for (int s = 0; s < 3; s++)  // channel s holds voxel u - (s - 1)
            e[s] = w_tap[(size_t)(tz * 9 + dy * 3 + 2 - s) * ep.Nout + co];
        }
      } else {
        v = *reinterpret_cast<const uint4*>(
            w_tap + ((size_t)(tz * 9 + t) * ep.Nout + co) * g.K + grp * 16 + j * 8);
      }
    }
    *reinterpret_cast<uint4*>(base + (size_t)i * 16) = v;
  }
  umma::fence_proxy_async();
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  // Up to here nothing that the kernel before may still write: the weights are
  // laid out while it ends (unless late_w).  The whole network on 32 x 80 x 32
  // voxels: 172 -> 132 us.
  pdl_wait();
  const uint32_t tbase = tslot;
  const int my_tiles =
      (int)blockIdx.x < g.ntiles ? (g.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  // a bit of `redo` stands for 2^rsh tiles
  int rsh = 0;
  while (((my_tiles - 1) >> rsh) >= 32 * C3_REDO) rsh++;
  bool timed_out = false;
  // a tile's place, stepped by gridDim.x tiles with carries
  int tix, tiy, tiz, tib;
  auto first_tile = [&] {
    tix = (int)blockIdx.x;
    tiy = tix / g.tiles_x, tix -= tiy * g.tiles_x;
    tiz = tiy / g.tiles_y, tiy -= tiz * g.tiles_y;
    tib = tiz / g.tiles_z, tiz -= tib * g.tiles_z;
  };
  int sx_ = (int)gridDim.x;
  int sy_ = sx_ / g.tiles_x;
  sx_ -= sy_ * g.tiles_x;
  int sz_ = sy_ / g.tiles_y;
  sy_ -= sz_ * g.tiles_y;
  const int sb_ = sz_ / g.tiles_z;
  sz_ -= sb_ * g.tiles_z;
  auto next_tile = [&] {
    tix += sx_, tiy += sy_, tiz += sz_, tib += sb_;
    if (tix >= g.tiles_x) tix -= g.tiles_x, tiy++;
    if (tiy >= g.tiles_y) tiy -= g.tiles_y, tiz++;
    if (tiz >= g.tiles_z) tiz -= g.tiles_z, tib++;
  };
  // what each role carries from tile to tile: the tiles it has taken, the loads
  // issued, the stage and its phase
  int it = 0, issued = 0, s = 0;
  uint32_t phase = warp == 0 ? 1u : 0u;
  // pass 0: every tile; pass 1: those with sums that are not finite, again
  for (int pass = 0; pass < (ZO > 1 ? 2 : 1); pass++) {
    if (pass == 1 && (__syncthreads_or(timed_out) || !redo_any)) break;
    first_tile();
    auto skip = [&](int jt) {
      return pass == 1 && !((redo[jt >> rsh >> 5] >> ((jt >> rsh) & 31)) & 1u);
    };
    if (warp == 0) {
      // ---- loads
      for (int jt = 0; jt < my_tiles && !timed_out; jt++, next_tile()) {
        if (skip(jt)) continue;
        for (int grp = 0; grp < G; grp++) {
          if (abort_flag) break;
          if (issued >= S && !umma::mbar_wait_warp(&empty[s], phase)) {
            timed_out = true;
            break;
          }
          // a box per plane and chunk, each from its own lane
          if (lane == 0) umma::mbar_expect_tx(&full[s], CHUNKS * ZI * BOX);
          __syncwarp();
          if (lane < CHUNKS * ZI) {
            const int ch = lane / ZI, zi = lane - ch * ZI;
            umma::tma_load_5d(stages + (size_t)s * STAGE + (uint32_t)lane * PLANE, &tx,
                              (tix * TX - (PACK ? 0 : 1)) * 8, tiy * TY - 1, tiz * ZO - 1 + zi,
                              PACK ? 0 : grp * 2 + ch, tib, &full[s]);
          }
          issued++;
          if (++s == S) s = 0, phase ^= 1u;
        }
        if (abort_flag) break;
      }
      if (timed_out) abort_flag = 1;
    } else if (warp == 1) {
      // ---- MMAs.  Descriptors: the high word holds the stride between core
      // matrices of 8 rows, the low word the K halves' distance and the address
      // in 16-byte units.
      const uint32_t idesc = umma::idesc_bf16(128, g.N);
      const uint32_t hi_a = (ROW >> 4) | (1u << 14), hi_b = (128u >> 4) | (1u << 14);
      const uint32_t lo_a = ((PACK ? ROW : CHUNK) >> 4) << 16;
      const uint32_t step = 2u * (uint32_t)g.rb;  // one K step of weights
      const uint32_t co16 = (uint32_t)g.CO;       // one plane of weight rows
      const uint32_t wb = (umma::smem_u32(base) >> 4) | ((uint32_t)g.rb << 16);
      for (int jt = 0; jt < my_tiles && !timed_out; jt++) {
        if (skip(jt)) continue;
        const int a = it & 1;
        if (abort_flag) break;
        if (it >= 2 && !umma::mbar_wait_warp(&acce[a], ((it >> 1) - 1) & 1)) {
          timed_out = true;
          break;
        }
        const uint32_t dt = tbase + (uint32_t)(a * g.N);
        for (int grp = 0; grp < G; grp++) {
          if (abort_flag) break;
          if (!umma::mbar_wait_warp(&full[s], phase)) {
            timed_out = true;
            break;
          }
          umma::fence_after();
          uint32_t da = ((umma::smem_u32(stages) + (uint32_t)s * STAGE) >> 4) | lo_a;
          uint32_t db = wb + (uint32_t)(grp * TAPS) * step + (uint32_t)(ZO + 1) * co16;
          // the MMAs of one input plane at d_, into the columns at c_
          auto plane = [&](uint32_t c_, uint32_t d_, uint32_t w_, uint32_t id, uint32_t acc) {
            if (umma::elect_one()) {
#pragma unroll
              for (int t = 0; t < TAPS; t++) {
                const uint32_t off = PACK ? (uint32_t)t * (ROW >> 4)
                                          : (uint32_t)(t / 3) * (ROW >> 4) + (uint32_t)(t % 3);
                umma::mma_bf16(c_, ((uint64_t)hi_a << 32) | (d_ + off),
                               ((uint64_t)hi_b << 32) | (w_ + t * step), id, t ? 1u : acc);
              }
            }
          };
          if (pass == 0) {
#pragma unroll 1
            for (int zi = 0; zi < ZI; zi++) {
              plane(dt, da, db, idesc, grp > 0 || zi > 0 ? 1u : 0u);
              da += PLANE >> 4;
              db -= co16;
            }
          } else {
#pragma unroll 1
            for (int zo = 0; zo < ZO; zo++)
#pragma unroll 1
              for (int tz = 0; tz < 3; tz++)
                plane(dt + (uint32_t)zo * co16, da + (uint32_t)(zo + tz) * (PLANE >> 4),
                      db - (uint32_t)tz * co16, umma::idesc_bf16(128, g.CO),
                      grp > 0 || tz > 0 ? 1u : 0u);
          }
          if (umma::elect_one()) umma::mma_commit(&empty[s]);
          if (++s == S) s = 0, phase ^= 1u;
        }
        if (timed_out || abort_flag) break;
        if (umma::elect_one()) umma::mma_commit(&accf[a]);
        it++;
      }
      if (timed_out) abort_flag = 1;
    } else {
      // ---- epilogue: lane = row of D = voxel (x = m % 8, y = m / 8); a column
      // is (zo, channel).  Two warps share the lanes of a quarter of D and take
      // its pairs of 16-column groups in turn.
      const int q = warp & 3, m = q * 32 + lane, half = (warp - 2) >> 2;
      // whole 8-channel chunks, 16-byte accesses of the output and the mask
      const bool planes = ep.out_bf16 && !(ep.Nout & 7) &&
                          !((reinterpret_cast<uintptr_t>(ep.out_bf16) |
                             reinterpret_cast<uintptr_t>(ep.mask)) & 15);
      const int gpz = g.CO >> 4;  // 16-column groups per output plane
      for (int jt = 0; jt < my_tiles; jt++, next_tile()) {
        if (skip(jt)) continue;
        const int a = it & 1;
        if (!umma::mbar_wait_warp(&accf[a], (it >> 1) & 1)) {
          timed_out = true;
          abort_flag = 1;
          break;
        }
        umma::fence_after();
        const int x = tix * TX + (m & 7), y = tiy * TY + (m >> 3), z0 = tiz * ZO;
        const bool in = x < g.nx && y < g.ny;
        const size_t v0 = (((size_t)tib * g.nz + z0) * g.ny + y) * g.nx + x;
        const size_t zs = (size_t)g.ny * g.nx;
        const uint32_t ta = tbase + (uint32_t)(a * g.N) + ((uint32_t)(q * 32) << 16);
        float top = 0.0f;  // the largest |sum|; NaN stays
        if (planes) {
          const int ng = g.N >> 4;
          for (int k0 = 2 * half; k0 < ng; k0 += 4) {
            // a pair of groups, their four masks loaded ahead
            size_t o[2];
            int c[2];
            bool own[2][2];
            uint4 mk[2][2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
              int zo, cg;
              if constexpr (ZO == 1) {
                zo = k0 + k < gpz ? 0 : ZO;
                cg = k0 + k;
              } else {
                zo = gpz == 1 ? k0 + k : (k0 + k) / gpz;
                cg = k0 + k - zo * gpz;
              }
              c[k] = cg * 16;
              o[k] = (size_t)((co0 + c[k]) >> 3) * ep.V + v0 + (size_t)zo * zs;
#pragma unroll
              for (int h = 0; h < 2; h++) {
                own[k][h] = in && k0 + k < ng && zo < ZO && z0 + zo < g.nz &&
                            co0 + c[k] + 8 * h < ep.Nout;
                if (ep.mask && own[k][h])
                  mk[k][h] = __ldg(reinterpret_cast<const uint4*>(ep.mask) + o[k] +
                                   (size_t)h * ep.V);
              }
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
              if (k0 + k >= ng) break;
              float v[16];
              umma::tmem_ld16(ta + (uint32_t)((k0 + k) * 16), v);
              if (ZO > 1) top = max_abs(v, top);
#pragma unroll
              for (int h = 0; h < 2; h++) {
                if (!own[k][h]) continue;
                const float4 b0 = *reinterpret_cast<const float4*>(sbias + c[k] + 8 * h),
                             b1 = *reinterpret_cast<const float4*>(sbias + c[k] + 8 * h + 4);
                float r[8] = {v[8 * h] + b0.x,     v[8 * h + 1] + b0.y, v[8 * h + 2] + b0.z,
                              v[8 * h + 3] + b0.w, v[8 * h + 4] + b1.x, v[8 * h + 5] + b1.y,
                              v[8 * h + 6] + b1.z, v[8 * h + 7] + b1.w};
                if (ep.relu) {
#pragma unroll
                  for (int e = 0; e < 8; e++) r[e] = fmaxf(r[e], 0.0f);
                }
                uint4 u;
                __nv_bfloat162* ub = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
                for (int e = 0; e < 4; e++) ub[e] = __floats2bfloat162_rn(r[2 * e], r[2 * e + 1]);
                if (ep.mask) {
                  // keep a BF16 half only where the mask half is > 0
                  const uint32_t* mw = reinterpret_cast<const uint32_t*>(&mk[k][h]);
                  uint32_t* uw = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
                  for (int e = 0; e < 4; e++) {
                    const float lo = __uint_as_float(mw[e] << 16),
                                hi = __uint_as_float(mw[e] & 0xFFFF0000u);
                    uw[e] &= (lo > 0.0f ? 0x0000FFFFu : 0u) | (hi > 0.0f ? 0xFFFF0000u : 0u);
                  }
                }
                if (ep.up) {
                  const int z = 2 * (z0 + (ZO == 1 ? 0 : (k0 + k) / gpz));
                  uint4* q8 = reinterpret_cast<uint4*>(ep.out_bf16) +
                              (size_t)(((co0 + c[k]) >> 3) + h) * ep.fV;
#pragma unroll
                  for (int j = 0; j < 4; j++) {
                    const int fz = z + (j >> 1), fy = 2 * y + (j & 1);
                    if (fz >= ep.fz || fy >= ep.fy) continue;
                    uint4* row = q8 + (((size_t)tib * ep.fz + fz) * ep.fy + fy) * ep.fx + 2 * x;
                    row[0] = u;
                    if (2 * x + 1 < ep.fx) row[1] = u;
                  }
                } else {
                  reinterpret_cast<uint4*>(ep.out_bf16)[o[k] + (size_t)h * ep.V] = u;
                }
              }
            }
          }
        } else {
          for (int col = 16 * half; col < g.N; col += 32) {
            float v[16];
            umma::tmem_ld16(ta + (uint32_t)col, v);
            if (ZO > 1) top = max_abs(v, top);
            const int zo = col / g.CO, c0 = col - zo * g.CO;
            if (!in || z0 + zo >= g.nz) continue;
            const size_t vox = v0 + (size_t)zo * zs;
#pragma unroll
            for (int k = 0; k < 16; k++) {
              const int c = c0 + k, co = co0 + c;
              if (co >= ep.Nout) break;
              float val = v[k] + sbias[c];
              if (ep.relu) val = fmaxf(val, 0.0f);
              if (ep.mask && !(__bfloat162float(ep.mask[act_off(vox, co, ep.Nout, ep.V)]) > 0.0f))
                val = 0.0f;
              if (ep.out_f32) ep.out_f32[vox * ep.Nout + co] = val;
              else ep.out_bf16[act_off(vox, co, ep.Nout, ep.V)] = __float2bfloat16_rn(val);
            }
          }
        }
        if (ZO > 1 && pass == 0 && __any_sync(0xffffffffu, !(top <= FLT_MAX)) && lane == 0) {
          atomicOr(&redo[jt >> rsh >> 5], 1u << ((jt >> rsh) & 31));
          redo_any = 1u;
        }
        umma::fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&acce[a]))
                       : "memory");
        it++;
      }
    }
  }
  if (warp == 0) {
    // every issued copy lands before the CTA may exit
    for (int q = issued > S ? issued - S : 0; q < issued; q++)
      if (!umma::mbar_wait_warp(&full[q % S], (q / S) & 1)) timed_out = true;
  } else if (warp == 1) {
    // every MMA issued has finished before the TMEM is freed
    if (umma::elect_one()) umma::mma_commit(&done);
    if (!umma::mbar_wait_warp(&done, 0)) timed_out = true;
  }
  if (timed_out && lane == 0) atomicExch(err, 1);
  umma::fence_before();
  __syncthreads();
  if (warp == 1) umma::tmem_dealloc(tbase, g.ncols);
}

using Kern3 = void (*)(CUtensorMap, const bf16*, C3Geom, ConvEpi, int*);

// Cycles of an MMA of 128 x N x 16 from shared memory (measured).
double mma_cycles(int N) { return std::max({45.5, 32.0 + N / 4.0, N / 2.0}); }

// Bytes of a stage (the kernel's STAGE).
long c3_stage(int zo, bool pack) {
  const long plane = (TY + 2) * (pack ? TX : TX + 2) * 16;
  return (plane + 127) / 128 * 128 * (zo + 2) * (pack ? 1 : 2);
}

struct C3Plan {
  int zo = 0, co = 0, split = 0, stages = 0;
  double cost = 0.0;
};

// The planes per tile and the channels per CTA with the shortest time: waves
// of tiles times a tile's MMAs, plus the weights each CTA writes first (about
// 1 cycle per 16-byte row and thread).  Tall tiles pay while there are waves
// of them; a small volume takes flat ones so that every SM has a tile.
// flat: one plane per tile, for an output that overwrites its mask (a tile that
// is done again reads the mask again).
C3Plan c3_plan(int nx, int ny, int nz, int nb, int groups, int N_out, bool pack, bool flat,
               int nsm) {
  C3Plan best;
  const int taps = pack ? 2 : 9;
  for (int zo : {1, 2, 4, 8}) {
    if (zo > 1 && (flat || zo / 2 >= nz)) continue;
    for (int split = 1; split <= (N_out + 15) / 16; split++) {
      const int co = ((N_out + split - 1) / split + 15) / 16 * 16;
      if (split > 1 && (co * (split - 1) >= N_out)) continue;
      if (co > C3_MAX_CO) continue;
      const int N = zo * co;
      if (N > 256) continue;
      const long rb = (long)(zo + 1) * co + N;
      const long wbytes = ((long)groups * taps * 2 * rb * 16 + 127) / 128 * 128;
      const long box = c3_stage(zo, pack);
      if (rb >= 16384 || wbytes + 2 * box > (long)C3_SMEM) continue;
      const long tiles = (long)((nx + TX - 1) / TX) * ((ny + TY - 1) / TY) *
                         ((nz + zo - 1) / zo) * nb;
      const long per = std::max<long>(1, nsm / split);
      const double cost = (double)((tiles + per - 1) / per) *
                              ((zo + 2) * taps * groups * mma_cycles(N) + 150.0) +
                          (double)groups * taps * 2 * rb * 30.0 / C3_THREADS;
      if (!best.zo || cost < best.cost) {
        best.zo = zo;
        best.co = co;
        best.split = split;
        best.stages = (int)std::min<long>(C3_MAX_STAGES, ((long)C3_SMEM - wbytes) / box);
        best.cost = cost;
      }
    }
  }
  return best;
}

}  // namespace

// y[v][n] = sum_{t, k} w_tap[t][n][k] x[v + tap(t)][k] (+ bias, ReLU, or
// zeroed where mask[v][n] <= 0); K (channels of x) a multiple of 16, or with
// pack K = 1 and the x-shifts of a one-channel tensor in one plane of 8
// channels (conv3_pack_grad); N <= 128 output channels.  x must be 16-byte aligned.
cudaError_t conv3_tma(const bf16* x, int K, bool pack, int nx, int ny, int nz, int nb,
                      const bf16* w_tap, int N, const float* bias, int relu, const bf16* mask,
                      bf16* y_bf16, float* y_f32, int* err, cudaStream_t st, const NetVol* fine,
                      bool old_weights) {
  if (fine && (!y_bf16 || N % 16)) return cudaErrorInvalidValue;
  if ((pack ? K != 1 : K % 16 != 0) || N < 1 || N > C3_MAX_CO)
    return cudaErrorInvalidValue;
  PFN_cuTensorMapEncodeTiled_v12000 enc = (PFN_cuTensorMapEncodeTiled_v12000)tensor_map_encoder();
  if (!enc) return cudaErrorNotSupported;
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  C3Geom g{};
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.nb = nb;
  g.K = K;
  g.late_w = old_weights ? 0 : 1;
  g.groups = pack ? 1 : K / 16;
  // the bytes of a BF16 or FP32 output and of its mask
  const size_t elems = (size_t)nx * ny * nz * nb * N;
  const char *y0 = y_f32 ? (const char*)y_f32 : (const char*)y_bf16, *m0 = (const char*)mask;
  const bool flat = mask && y0 < m0 + elems * 2 && m0 < y0 + elems * (y_f32 ? 4 : 2);
  const C3Plan pl = c3_plan(nx, ny, nz, nb, g.groups, N, pack, flat, nsm);
  if (!pl.zo) return cudaErrorInvalidValue;
  const int taps = pack ? 2 : 9, px = pack ? TX : TX + 2;
  g.CO = pl.co;
  g.N = pl.zo * pl.co;
  g.rb = (pl.zo + 1) * pl.co + g.N;
  g.stages = pl.stages;
  g.wbytes = ((uint32_t)(g.groups * taps * 2 * g.rb) * 16u + 127u) & ~127u;
  g.ncols = 32;
  while ((int)g.ncols < 2 * g.N) g.ncols *= 2;
  g.tiles_x = (nx + TX - 1) / TX;
  g.tiles_y = (ny + TY - 1) / TY;
  g.tiles_z = (nz + pl.zo - 1) / pl.zo;
  g.ntiles = g.tiles_x * g.tiles_y * g.tiles_z * nb;
  // planes of 8 channels as (x, y, z, plane, volume)
  const cuuint64_t row = (cuuint64_t)nx * 16, vol = row * ny * nz;
  const cuuint64_t dim[5] = {(cuuint64_t)nx * 8, (cuuint64_t)ny, (cuuint64_t)nz,
                             (cuuint64_t)(pack ? 1 : K / 8), (cuuint64_t)nb};
  const cuuint64_t str[4] = {row, row * ny, vol * nb, vol};
  const cuuint32_t box[5] = {(cuuint32_t)(8 * px), TY + 2, 1, 1, 1};
  const cuuint32_t es[5] = {1, 1, 1, 1, 1};
  CUtensorMap tx;
  if (enc(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(x), dim, str, box, es,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  static constexpr Kern3 kerns[4][2] = {{k_conv3<1, false>, k_conv3<1, true>},
                                        {k_conv3<2, false>, k_conv3<2, true>},
                                        {k_conv3<4, false>, k_conv3<4, true>},
                                        {k_conv3<8, false>, k_conv3<8, true>}};
  const Kern3 kern = kerns[pl.zo == 1 ? 0 : pl.zo == 2 ? 1 : pl.zo == 4 ? 2 : 3][pack ? 1 : 0];
  const size_t smem = (size_t)g.wbytes + (size_t)g.stages * c3_stage(pl.zo, pack) + 128;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  ConvEpi ep{y_bf16, y_f32, bias, mask, nx * ny * nz * nb, N, relu,
             fine ? 1 : 0, fine ? fine->nx : 0, fine ? fine->ny : 0, fine ? fine->nz : 0,
             fine ? (int)fine->voxels() : 0};
  const int ctas = std::max(1, std::min(g.ntiles, nsm / pl.split));
  return launch_pdl(kern, dim3((unsigned)ctas, (unsigned)pl.split), dim3(C3_THREADS), smem, st, tx,
                    w_tap, g, ep, err);
}

}  // namespace pyro
