// k_conv.cu — 3x3x3 convolutions (padding 1, stride 1) as implicit GEMMs on
// the tcgen05 tensor cores, for the learned pressure warm start.
//
// One kernel, k_gemm<N, Load, Epi>, computes a 128 x N tile of
// D = A * B^T with BF16 operands staged in shared memory (two-stage
// pipeline, K in steps of 16) and the FP32 accumulator in TMEM:
//
//   forward          A[m = voxel][k = (tap, ci)] = x[voxel + tap][ci]
//                    B[n = co][k]                = W[co][tap][ci]
//   backward (data)  A[m = voxel][k = (tap, co)] = dy[voxel - tap][co]
//                    B[n = ci][k]                = W[co][tap][ci]
//   backward (weight) A[m = (tap, ci)][k = voxel] = x[voxel + tap][ci]
//                    B[n = co][k = voxel]        = dy[voxel][co]   (split over K;
//                    channel counts and alignments that k_wgrad.cu does not
//                    take, and gradients with sums that are not finite)
//
// Activations are BF16 in planes of 8 channels, [C / 8][volume][z][y][x][8]
// (C a multiple of 8; [volume][z][y][x][C] otherwise); a tap
// outside its volume reads zero.  One thread issues the MMA, tcgen05.commit
// signals an mbarrier per stage, and every wait is bounded: a wait that runs
// out sets *err and the CTA still frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "conv.cuh"
#include "net.h"
#include "umma.cuh"

namespace pyro {

namespace {

using bf16 = __nv_bfloat16;
constexpr int GEMM_THREADS = 128;

struct Vol {
  int nx, ny, nz, nb;  // volume dims and count
  __device__ __forceinline__ int voxels() const { return nx * ny * nz * nb; }
};

// Voxel v shifted by tap (dx, dy, dz) within its volume, or -1.
__device__ __forceinline__ int shifted(const Vol& g, int v, int dx, int dy, int dz) {
  int x = v % g.nx;
  int r = v / g.nx;
  int y = r % g.ny;
  r /= g.ny;
  int z = r % g.nz;
  int b = r / g.nz;
  x += dx;
  y += dy;
  z += dz;
  if ((unsigned)x >= (unsigned)g.nx || (unsigned)y >= (unsigned)g.ny ||
      (unsigned)z >= (unsigned)g.nz)
    return -1;
  return ((b * g.nz + z) * g.ny + y) * g.nx + x;
}
__device__ __forceinline__ void tap_offset(int t, int& dx, int& dy, int& dz) {
  dx = t % 3 - 1;
  dy = (t / 3) % 3 - 1;
  dz = t / 9 - 1;
}

__device__ __forceinline__ void st16(uint8_t* s, uint32_t off, uint4 v) {
  *reinterpret_cast<uint4*>(s + off) = v;
}
__device__ __forceinline__ void st_bf(uint8_t* s, uint32_t off, bf16 v) {
  *reinterpret_cast<bf16*>(s + off) = v;
}

// TMEM of a block that computes tiles one after another (allocated once: a
// block that has given up its permit may not allocate again).
constexpr int gemm_cols(int N) { return N <= 32 ? 32 : (N <= 64 ? 64 : 128); }
template <int N>
__device__ uint32_t gemm_alloc() {
  __shared__ uint32_t tslot;
  if (threadIdx.x < 32) {
    umma::tmem_alloc(&tslot, gemm_cols(N));
    umma::tmem_relinquish();
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  return tslot;
}
template <int N>
__device__ void gemm_free(uint32_t tbase) {
  umma::fence_before();
  __syncthreads();
  if (threadIdx.x < 32) umma::tmem_dealloc(tbase, gemm_cols(N));
}

// One tile: rows m0 .. m0 + 127, K steps k0 .. k1 - 1; the whole block calls.
// False when a wait ran out: the block computes no further tile.
template <int N, class Load, class Epi>
__device__ bool gemm_tile(const Load& ld, const Epi& ep, uint32_t tbase, int m0, int k0, int k1,
                          int* err) {
  __shared__ __align__(1024) uint8_t sA[2][128 * 32];
  __shared__ __align__(1024) uint8_t sB[2][N * 32];
  __shared__ __align__(8) uint64_t mbar[2];
  const int nks = max(k1 - k0, 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    umma::mbar_init(&mbar[0], 1);
    umma::mbar_init(&mbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  constexpr uint32_t IDESC = umma::idesc_bf16(128, N);
  bool ok = true;
  for (int i = 0; i < nks; i++) {
    const int s = i & 1;
    if (i >= 2 && !umma::mbar_wait_bounded(&mbar[s], ((i - 2) >> 1) & 1)) ok = false;
    ld(sA[s], sB[s], m0, k0 + i);
    umma::fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      umma::fence_after();
      umma::mma_bf16(tbase, umma::smem_desc(sA[s], 128), umma::smem_desc(sB[s], N), IDESC,
                     i > 0 ? 1u : 0u);
      umma::mma_commit(&mbar[s]);
    }
  }
  // both barriers' last phases: nothing arrives on them any more
  for (int i = max(nks - 2, 0); i < nks; i++)
    if (!umma::mbar_wait_bounded(&mbar[i & 1], (i >> 1) & 1)) ok = false;
  umma::fence_after();
  const bool all_ok = __syncthreads_and(ok) != 0;
  if (all_ok && nks > 0) {
#pragma unroll
    for (int col = 0; col < N; col += 16) {
      float v[16];
      umma::tmem_ld16(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)col, v);
      ep(m0 + warp * 32 + lane, col, v);
    }
  }
  if (!all_ok && threadIdx.x == 0) atomicExch(err, 1);
  // the sums are read and the barriers done with before the next tile
  umma::fence_before();
  __syncthreads();
  if (all_ok && threadIdx.x == 0) {
    umma::mbar_inval(&mbar[0]);
    umma::mbar_inval(&mbar[1]);
  }
  __syncthreads();
  return all_ok;
}

template <int N, class Load, class Epi>
__global__ void __launch_bounds__(GEMM_THREADS) k_gemm(Load ld, Epi ep, int ksteps_total,
                                                       int ksteps_per_cta, int* err,
                                                       const int* only_if) {
  pdl_wait();  // no early trigger: the next launch's CTAs may allocate TMEM before they wait
  if (only_if && *only_if == 0) return;
  const int k0 = blockIdx.y * ksteps_per_cta;
  const uint32_t tbase = gemm_alloc<N>();
  gemm_tile<N>(ld, ep, tbase, blockIdx.x * 128, k0, min(k0 + ksteps_per_cta, ksteps_total), err);
  gemm_free<N>(tbase);
}

// ---------------------------------------------------------------- loaders
// A = shifted activations (voxel rows, K = (tap, channel)); B = weight rows.
// `flip` negates the tap (backward data); `wt` selects the transposed
// weight gather for backward data: B[n = ci][k = (tap, co)] = W[co][tap][ci].
struct ConvLoad {
  const bf16* x;      // [V][C]
  const bf16* w;      // [Cw_out][27][Cw_in]
  Vol g;
  int C;              // channels of x (K = 27 C)
  int Nrows;          // rows of B that exist (co, or ci for backward data)
  int cw_in, cw_out;  // weight dims
  int flip, wt;
  __device__ void operator()(uint8_t* sA, uint8_t* sB, int m0, int ks) const {
    const int t0 = threadIdx.x;
    const int V = g.voxels();
    const int K = 27 * C;
    // A: row r = voxel m0 + r
    {
      int r = t0;
      int v = m0 + r;
      if ((C & 15) == 0) {
        int t = ks / (C >> 4), cc = ks % (C >> 4);
        int dx, dy, dz;
        tap_offset(t, dx, dy, dz);
        if (flip) { dx = -dx; dy = -dy; dz = -dz; }
        uint4 a0 = make_uint4(0, 0, 0, 0), a1 = a0;
        if (v < V) {
          int vs = shifted(g, v, dx, dy, dz);
          if (vs >= 0) {
            const uint4* p = reinterpret_cast<const uint4*>(x + act_off(vs, cc * 16, C, V));
            a0 = __ldg(p);
            a1 = __ldg(p + V);  // the next 8-channel plane
          }
        }
        st16(sA, umma::core_offset(r, 0, 128), a0);
        st16(sA, umma::core_offset(r, 8, 128), a1);
      } else {
        for (int e = 0; e < 16; e++) {
          int k = ks * 16 + e;
          bf16 val = __float2bfloat16(0.0f);
          if (v < V && k < K) {
            int t = k / C, ci = k % C;
            int dx, dy, dz;
            tap_offset(t, dx, dy, dz);
            if (flip) { dx = -dx; dy = -dy; dz = -dz; }
            int vs = shifted(g, v, dx, dy, dz);
            if (vs >= 0) val = x[act_off(vs, ci, C, V)];
          }
          st_bf(sA, umma::core_offset(r, e, 128), val);
        }
      }
    }
    // B: row n (co for forward, ci for backward data)
    if (t0 < Nrows_pad()) {
      int n = t0;
      for (int e = 0; e < 16; e++) {
        int k = ks * 16 + e;
        bf16 val = __float2bfloat16(0.0f);
        if (n < Nrows && k < K) {
          if (!wt) {
            val = w[(size_t)n * K + k];  // W[co][tap][ci], K index tap * C + ci
          } else {
            int t = k / C, co = k % C;   // K index tap * Cout + co
            val = w[((size_t)co * 27 + t) * cw_in + n];
          }
        }
        st_bf(sB, umma::core_offset(n, e, npad), val);
      }
    }
  }
  int npad;
  __device__ __forceinline__ int Nrows_pad() const { return npad; }
};

// Weight gradient: A[m = (tap, ci)][k = voxel] = x[voxel + tap][ci],
// B[n = co][k = voxel] = dy[voxel][co].
struct WgradLoad {
  const bf16* x;   // [V][Cin]
  const bf16* dy;  // [V][Cout]
  Vol g;
  int Cin, Cout, npad;
  __device__ void operator()(uint8_t* sA, uint8_t* sB, int m0, int ks) const {
    const int V = g.voxels();
    const int M = 27 * Cin;
    {
      int r = threadIdx.x;
      int m = m0 + r;
      int t = m / Cin, ci = m % Cin;
      int dx, dy_, dz;
      tap_offset(t < 27 ? t : 0, dx, dy_, dz);
      for (int e = 0; e < 16; e++) {
        int v = ks * 16 + e;
        bf16 val = __float2bfloat16(0.0f);
        if (m < M && v < V) {
          int vs = shifted(g, v, dx, dy_, dz);
          if (vs >= 0) val = x[act_off(vs, ci, Cin, V)];
        }
        st_bf(sA, umma::core_offset(r, e, 128), val);
      }
    }
    if ((int)threadIdx.x < npad) {
      int n = threadIdx.x;
      for (int e = 0; e < 16; e++) {
        int v = ks * 16 + e;
        bf16 val = __float2bfloat16(0.0f);
        if (n < Cout && v < V) val = dy[act_off(v, n, Cout, V)];
        st_bf(sB, umma::core_offset(n, e, npad), val);
      }
    }
  }
};

// -------------------------------------------------------------- epilogues
// Weight gradient: row m = (tap, ci), column n = co; FP32 atomics into
// dw[co][tap][ci] (split-K partial sums).
struct WgradEpi {
  float* dw;
  int M, Cout;
  __device__ void operator()(int m, int col, const float (&v)[16]) const {
    if (m >= M) return;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      int n = col + j;
      if (n >= Cout) break;
      atomicAdd(dw + (size_t)n * M + m, v[j]);
    }
  }
};

// The weight gradients of a network's layers that have bad[l] set, one launch
// for all: the blocks share a layer's tiles, layer after layer (a launch per
// layer that ends at once took 7 us each).
constexpr int WG_N = 64;  // output channels at most
struct WgradJobs {
  WgradLoad ld[NET_LAYERS];
  WgradEpi ep[NET_LAYERS];
  int ksteps[NET_LAYERS], per[NET_LAYERS];
};
__global__ void __launch_bounds__(GEMM_THREADS)
    k_wgrad_gathers(const __grid_constant__ WgradJobs J, const int* __restrict__ bad, int* err) {
  pdl_wait();
  int any = 0;
  for (int l = 0; l < NET_LAYERS; l++) any |= bad[l];
  if (!any) return;
  const uint32_t tbase = gemm_alloc<WG_N>();
  bool ok = true;
  for (int l = 0; l < NET_LAYERS; l++) {
    if (!bad[l]) continue;
    const int mt = (J.ep[l].M + 127) / 128, splits = (J.ksteps[l] + J.per[l] - 1) / J.per[l];
    for (int t = blockIdx.x; ok && t < mt * splits; t += gridDim.x) {
      const int k0 = t / mt * J.per[l];
      ok = gemm_tile<WG_N>(J.ld[l], J.ep[l], tbase, t % mt * 128, k0,
                           min(k0 + J.per[l], J.ksteps[l]), err);
    }
  }
  gemm_free<WG_N>(tbase);
}

template <int N, class Load, class Epi>
cudaError_t gemm_launch(dim3 grid, const Load& ld, const Epi& ep, int ksteps_total,
                        int ksteps_per_cta, int* err, cudaStream_t st, const int* only_if) {
  return launch_pdl(k_gemm<N, Load, Epi>, grid, dim3(GEMM_THREADS), 0, st, ld, ep, ksteps_total,
                    ksteps_per_cta, err, only_if);
}

template <class Load, class Epi>
cudaError_t gemm_dispatch(int npad, dim3 grid, const Load& ld, const Epi& ep, int kt, int kpc,
                          int* err, cudaStream_t st, const int* only_if = nullptr) {
  switch (npad) {
    case 16: return gemm_launch<16>(grid, ld, ep, kt, kpc, err, st, only_if);
    case 32: return gemm_launch<32>(grid, ld, ep, kt, kpc, err, st, only_if);
    case 48: return gemm_launch<48>(grid, ld, ep, kt, kpc, err, st, only_if);
    case 64: return gemm_launch<64>(grid, ld, ep, kt, kpc, err, st, only_if);
    case 96: return gemm_launch<96>(grid, ld, ep, kt, kpc, err, st, only_if);
    case 128: return gemm_launch<128>(grid, ld, ep, kt, kpc, err, st, only_if);
    default: return cudaErrorInvalidValue;
  }
}


// --------------------------------------------------------- direct (CUDA cores)
// The two narrow layers, 2 -> 16 channels on [voxel][2] inputs and 16 -> 1,
// whose sums stay FP32 fused multiply-adds in one fixed order: the tensor
// cores' sums are faster (160 x 320 x 160 voxels: 2 -> 16 101 us instead of
// 420, 16 -> 1 159 instead of 491) but further from 64 bits (normal inputs:
// 16 -> 1 4.1e-7 against 1.5e-7, 2 -> 16 7.0e-8 against 5.2e-8), and the first
// layer's rounding travels through all that follow.
// A thread computes DV consecutive voxels of an x-row.  For every (dz, dy)
// input row it loads the DV + 2 voxels x0-1 .. x0+DV once (zero outside
// the volume), and the three dx taps of all DV outputs read them from
// registers; every weight read from shared memory (FP32, [tap][ci][co])
// feeds DV fused multiply-adds.  FP32 accumulation.
template <int CIN, int COUT>
struct DirectShape {
  static constexpr int DV = 4;                  // voxels per thread
  static constexpr int CC = CIN == 2 ? 2 : 8;   // input channels per chunk
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(256, 2) k_conv_direct(const bf16* __restrict__ x, Vol g,
                                                     const bf16* __restrict__ w,
                                                     const float* __restrict__ bias, int relu,
                                                     bf16* __restrict__ y_bf16,
                                                     float* __restrict__ y_f32) {
  pdl_trigger();
  pdl_wait();
  static_assert(CIN == 2 || CIN % 8 == 0, "input rows are loaded as 4- or 16-byte chunks");
  constexpr int DV = DirectShape<CIN, COUT>::DV, CC = DirectShape<CIN, COUT>::CC;
  __shared__ __align__(16) float ws[27 * CIN * COUT];
  for (int i = threadIdx.x; i < 27 * CIN * COUT; i += blockDim.x) {
    const int co = i / (27 * CIN), t = (i / CIN) % 27, ci = i % CIN;  // w[co][t][ci]
    ws[(t * CIN + ci) * COUT + co] = __bfloat162float(w[i]);
  }
  __syncthreads();
  const long V = (long)g.nx * g.ny * g.nz * g.nb;
  const int cpr = (g.nx + DV - 1) / DV;  // chunks per x-row
  const long nchunks = (long)cpr * g.ny * g.nz * g.nb;
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nchunks) return;
  const long row = c / cpr;  // (b, z, y) row index
  const int x0 = (int)(c - row * cpr) * DV;
  const int yy = (int)(row % g.ny);
  const int zz = (int)((row / g.ny) % g.nz);
  const long v0 = row * g.nx + x0;
  float acc[DV][COUT];
#pragma unroll
  for (int i = 0; i < DV; i++)
#pragma unroll
    for (int co = 0; co < COUT; co++) acc[i][co] = bias ? bias[co] : 0.0f;
  const long sy = g.nx, sz = (long)g.nx * g.ny;
#pragma unroll 1
  for (int dz = -1; dz <= 1; dz++) {
    if ((unsigned)(zz + dz) >= (unsigned)g.nz) continue;
#pragma unroll 1
    for (int dy = -1; dy <= 1; dy++) {
      if ((unsigned)(yy + dy) >= (unsigned)g.ny) continue;
      const long vr = v0 + sy * dy + sz * dz;  // voxel x0 of the input row
#pragma unroll
      for (int c0 = 0; c0 < CIN; c0 += CC) {
        float xin[DV + 2][CC];
#pragma unroll
        for (int i = 0; i < DV + 2; i++) {
          const int xs = x0 - 1 + i;
          const bool in = (unsigned)xs < (unsigned)g.nx;
          const long vs = vr - 1 + i;
          if constexpr (CIN == 2) {
            float2 f = make_float2(0.0f, 0.0f);
            if (in) f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + vs * 2));
            xin[i][0] = f.x;
            xin[i][1] = f.y;
          } else {
            uint4 u = make_uint4(0, 0, 0, 0);
            if (in) u = __ldg(reinterpret_cast<const uint4*>(x + act_off(vs, c0, CIN, V)));
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const float2 f = __bfloat1622float2(h[j]);
              xin[i][2 * j] = f.x;
              xin[i][2 * j + 1] = f.y;
            }
          }
        }
#pragma unroll
        for (int dx = 0; dx < 3; dx++) {
          const float* wt = ws + ((dx + 3 * (dy + 1) + 9 * (dz + 1)) * CIN + c0) * COUT;
#pragma unroll
          for (int ci = 0; ci < CC; ci++)
#pragma unroll
            for (int co = 0; co < COUT; co++) {
              const float wv = wt[ci * COUT + co];
#pragma unroll
              for (int i = 0; i < DV; i++)
                acc[i][co] = __fmaf_rn(xin[i + dx][ci], wv, acc[i][co]);
            }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < DV; i++) {
    if (x0 + i >= g.nx) break;
    const long v = v0 + i;
    if (relu) {
#pragma unroll
      for (int co = 0; co < COUT; co++) acc[i][co] = fmaxf(acc[i][co], 0.0f);
    }
    if (y_f32) {
#pragma unroll
      for (int co = 0; co < COUT; co++) y_f32[v * COUT + co] = acc[i][co];
    } else if constexpr (COUT % 8 == 0) {
#pragma unroll
      for (int c8 = 0; c8 < COUT; c8 += 8) {
        uint4 o;
        __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; j++)
          ob[j] = __floats2bfloat162_rn(acc[i][c8 + 2 * j], acc[i][c8 + 2 * j + 1]);
        *reinterpret_cast<uint4*>(y_bf16 + act_off(v, c8, COUT, V)) = o;
      }
    } else {
#pragma unroll
      for (int co = 0; co < COUT; co++)
        y_bf16[act_off(v, co, COUT, V)] = __float2bfloat16_rn(acc[i][co]);
    }
  }
}

__global__ void k_wprep(const bf16* __restrict__ w, int Cout, int Cin, int backward,
                        bf16* __restrict__ out) {
  const int n = Cout * 27 * Cin;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int co = i / (27 * Cin), t = (i / Cin) % 27, ci = i % Cin;
    if (!backward)
      out[((size_t)t * Cout + co) * Cin + ci] = w[i];
    else
      out[((size_t)(26 - t) * Cin + ci) * Cout + co] = w[i];
  }
}

// dw += s, nothing when *bad is set
__global__ void __launch_bounds__(256) k_add_unless(const double* __restrict__ s, int n,
                                                    const int* __restrict__ bad,
                                                    float* __restrict__ dw) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n && !*bad) dw[i] = (float)((double)dw[i] + s[i]);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

inline int pad16(int n) { return (n + 15) / 16 * 16; }

}  // namespace

void* tensor_map_encoder() { return (void*)encode_fn(); }

// y = conv(x, W) (+ bias, ReLU), or its transpose for backward data.
cudaError_t conv3_forward(const bf16* x, int C, int nx, int ny, int nz, int nb, const bf16* w,
                          int Cout, const float* bias, int relu, bf16* y_bf16, float* y_f32,
                          int* err, cudaStream_t st) {
  Vol g{nx, ny, nz, nb};
  int V = nx * ny * nz * nb;
  int npad = pad16(Cout);
  int ksteps = (27 * C + 15) / 16;
  ConvLoad ld{x, w, g, C, Cout, C, Cout, 0, 0, npad};
  ConvEpi ep{y_bf16, y_f32, bias, nullptr, V, Cout, relu};
  dim3 grid((V + 127) / 128, 1, 1);
  return gemm_dispatch(npad, grid, ld, ep, ksteps, ksteps, err, st);
}

// dx = conv^T(dy, W), masked by (act > 0) when act is given.
cudaError_t conv3_backward_data(const bf16* dy, int Cout, int nx, int ny, int nz, int nb,
                                const bf16* w, int Cin, const bf16* act, bf16* dx_bf16,
                                float* dx_f32, int* err, cudaStream_t st) {
  Vol g{nx, ny, nz, nb};
  int V = nx * ny * nz * nb;
  int npad = pad16(Cin);
  int ksteps = (27 * Cout + 15) / 16;
  ConvLoad ld{dy, w, g, Cout, Cin, Cin, Cout, 1, 1, npad};
  ConvEpi ep{dx_bf16, dx_f32, nullptr, act, V, Cin, 0};
  dim3 grid((V + 127) / 128, 1, 1);
  return gemm_dispatch(npad, grid, ld, ep, ksteps, ksteps, err, st);
}

int conv3_gather_steps(int Cin, long V) {
  const long ksteps = (V + 15) / 16, mt = (27 * Cin + 127) / 128;
  // split K so that the grid covers the GPU a few times over
  const long splits = std::max(1l, std::min(ksteps, (148 * 8) / std::max(mt, 1l)));
  return (int)((ksteps + splits - 1) / splits);
}

cudaError_t conv3_wgrad_gathers(const WgradJob (&jobs)[NET_LAYERS], const int* bad, int* err,
                                cudaStream_t st) {
  WgradJobs J;
  for (int l = 0; l < NET_LAYERS; l++) {
    const WgradJob& j = jobs[l];
    const NetLayer& L = NET_SPEC[l];
    const long V = (long)j.v.voxels();
    static_assert(NET_SPEC[5].cout == WG_N, "");
    J.ld[l] = WgradLoad{j.x, j.g, Vol{j.v.nx, j.v.ny, j.v.nz, j.v.nb}, L.cin, L.cout, WG_N};
    J.ep[l] = WgradEpi{j.dw, 27 * L.cin, L.cout};
    J.ksteps[l] = (int)((V + 15) / 16);
    J.per[l] = conv3_gather_steps(L.cin, V);
  }
  return launch_pdl(k_wgrad_gathers, dim3(148 * 8), dim3(GEMM_THREADS), 0, st, J, bad, err);
}

// dw[co][tap][ci] += sum_voxels dy[v][co] x[v + tap][ci]  (dw FP32).
cudaError_t conv3_wgrad_gather(const bf16* x, int Cin, const bf16* dy, int Cout, int nx, int ny,
                               int nz, int nb, float* dw, int* err, const int* only_if,
                               cudaStream_t st) {
  Vol g{nx, ny, nz, nb};
  int V = nx * ny * nz * nb;
  int M = 27 * Cin;
  int npad = pad16(Cout);
  if (only_if && npad > 64) npad = npad > 96 ? 128 : 96;  // behind the boxes, which take 80 and 112
  const int ksteps = (V + 15) / 16, mt = (M + 127) / 128, kpc = conv3_gather_steps(Cin, V);
  const int splits = (ksteps + kpc - 1) / kpc;
  WgradLoad ld{x, dy, g, Cin, Cout, npad};
  WgradEpi ep{dw, M, Cout};
  dim3 grid(mt, splits, 1);
  return gemm_dispatch(npad, grid, ld, ep, ksteps, kpc, err, st, only_if);
}

// Direct convolution for the shapes k_conv_direct covers (2 -> 16 and
// 16 -> 1 channels); cudaErrorInvalidValue for others and for tensors off the
// boundary of its accesses (x: a voxel's 4 bytes, a plane's 16; BF16 output of
// 16 channels: 16).
bool conv3_direct_fits(int C, int Cout) { return (C == 2 && Cout == 16) || (C == 16 && Cout == 1); }

cudaError_t conv3_direct(const bf16* x, int C, int nx, int ny, int nz, int nb, const bf16* w,
                         int Cout, const float* bias, int relu, bf16* y_bf16, float* y_f32,
                         cudaStream_t st) {
  if (reinterpret_cast<uintptr_t>(x) % (C == 2 ? 4 : 16) ||
      (!y_f32 && Cout % 8 == 0 && reinterpret_cast<uintptr_t>(y_bf16) % 16))
    return cudaErrorInvalidValue;
  Vol g{nx, ny, nz, nb};
  auto blocks = [&](int dv) {
    return (unsigned)(((long)((nx + dv - 1) / dv) * ny * nz * nb + 255) / 256);
  };
  if (C == 2 && Cout == 16)
    return launch_pdl(k_conv_direct<2, 16>, dim3(blocks(DirectShape<2, 16>::DV)), dim3(256), 0, st,
                      x, g, w, bias, relu, y_bf16, y_f32);
  if (C == 16 && Cout == 1)
    return launch_pdl(k_conv_direct<16, 1>, dim3(blocks(DirectShape<16, 1>::DV)), dim3(256), 0, st,
                      x, g, w, bias, relu, y_bf16, y_f32);
  return cudaErrorInvalidValue;
}

// Weight layouts for conv3_tma: forward w_tap[t][co][ci] = w[co][t][ci];
// backward (data) w_tap[t][ci][co] = w[co][26 - t][ci] (flipped taps,
// transposed channels).
cudaError_t conv3_prep_weights(const bf16* w, int Cout, int Cin, int backward, bf16* w_tap,
                               cudaStream_t st) {
  const int n = Cout * 27 * Cin;
  k_wprep<<<std::min((n + 255) / 256, 1024), 256, 0, st>>>(w, Cout, Cin, backward, w_tap);
  return cudaGetLastError();
}

}  // namespace pyro

// ------------------------------------------------------------------ C ABI
using namespace pyro;
using bf16 = __nv_bfloat16;

namespace {
int finish(cudaError_t e, DevBuf& err, cudaStream_t st, const char* what) {
  if (e != cudaSuccess) {
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return PYRO_E_CUDA;
  }
  int h = 0;
  PYRO_CU(cudaMemcpyAsync(&h, err.p, 4, cudaMemcpyDeviceToHost, st));
  PYRO_CU(cudaStreamSynchronize(st));
  if (h) {
    set_error(std::string(what) + ": a tensor-core wait ran out");
    return PYRO_E_TIMEOUT;
  }
  return PYRO_OK;
}
bool conv_dims_ok(int nx, int ny, int nz, int nb) {
  return nx >= 1 && ny >= 1 && nz >= 1 && nb >= 1 && (int64_t)nx * ny * nz * nb < (1ll << 31);
}
bool chan_ok(int c) { return c >= 1 && c <= 128; }
}  // namespace

extern "C" {

int pyro_conv3_forward(const void* x, int C, int nx, int ny, int nz, int nb, const void* w,
                       int Cout, const float* bias, int relu, void* y, int y_f32, void* stream) {
  clear_error();
  PYRO_REQUIRE(x && w && y, "pyro_conv3_forward: null buffer");
  PYRO_REQUIRE(conv_dims_ok(nx, ny, nz, nb) && chan_ok(C) && chan_ok(Cout),
               "pyro_conv3_forward: invalid sizes");
  DevBuf err;
  int rc = err.alloc(4);
  if (rc != PYRO_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (conv3_direct_fits(C, Cout)) {  // narrow layers on the CUDA cores
    e = conv3_direct((const bf16*)x, C, nx, ny, nz, nb, (const bf16*)w, Cout, bias, relu,
                     y_f32 ? nullptr : (bf16*)y, y_f32 ? (float*)y : nullptr, st);
    return finish(e, err, st, "pyro_conv3_forward");
  }
  if (C % 16 == 0) {  // TMA-staged kernel on tap-major weights
    DevBuf wt;
    if ((rc = wt.alloc((size_t)Cout * 27 * C * 2)) != PYRO_OK) return rc;
    e = conv3_prep_weights((const bf16*)w, Cout, C, 0, wt.as<bf16>(), st);
    if (e == cudaSuccess)
      e = conv3_tma((const bf16*)x, C, false, nx, ny, nz, nb, wt.as<bf16>(), Cout, bias, relu,
                    nullptr, y_f32 ? nullptr : (bf16*)y, y_f32 ? (float*)y : nullptr,
                    err.as<int>(), st);
    return finish(e, err, st, "pyro_conv3_forward");
  }
  e = conv3_forward((const bf16*)x, C, nx, ny, nz, nb, (const bf16*)w, Cout, bias, relu,
                    y_f32 ? nullptr : (bf16*)y, y_f32 ? (float*)y : nullptr, err.as<int>(), st);
  return finish(e, err, st, "pyro_conv3_forward");
}

int pyro_conv3_backward_data(const void* dy, int Cout, int nx, int ny, int nz, int nb,
                             const void* w, int Cin, const void* act, void* dx, int dx_f32,
                             void* stream) {
  clear_error();
  PYRO_REQUIRE(dy && w && dx, "pyro_conv3_backward_data: null buffer");
  PYRO_REQUIRE(conv_dims_ok(nx, ny, nz, nb) && chan_ok(Cin) && chan_ok(Cout),
               "pyro_conv3_backward_data: invalid sizes");
  DevBuf err;
  int rc = err.alloc(4);
  if (rc != PYRO_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (Cout % 16 == 0) {  // TMA-staged kernel on flipped, transposed weights
    DevBuf wt;
    if ((rc = wt.alloc((size_t)Cout * 27 * Cin * 2)) != PYRO_OK) return rc;
    e = conv3_prep_weights((const bf16*)w, Cout, Cin, 1, wt.as<bf16>(), st);
    if (e == cudaSuccess)
      e = conv3_tma((const bf16*)dy, Cout, false, nx, ny, nz, nb, wt.as<bf16>(), Cin, nullptr, 0,
                    (const bf16*)act, dx_f32 ? nullptr : (bf16*)dx, dx_f32 ? (float*)dx : nullptr,
                    err.as<int>(), st);
    return finish(e, err, st, "pyro_conv3_backward_data");
  }
  e = conv3_backward_data((const bf16*)dy, Cout, nx, ny, nz, nb, (const bf16*)w, Cin,
                          (const bf16*)act, dx_f32 ? nullptr : (bf16*)dx,
                          dx_f32 ? (float*)dx : nullptr, err.as<int>(), st);
  return finish(e, err, st, "pyro_conv3_backward_data");
}

int pyro_conv3_backward_weight(const void* x, int Cin, const void* dy, int Cout, int nx, int ny,
                               int nz, int nb, float* dw, void* stream) {
  clear_error();
  PYRO_REQUIRE(x && dy && dw, "pyro_conv3_backward_weight: null buffer");
  PYRO_REQUIRE(conv_dims_ok(nx, ny, nz, nb) && chan_ok(Cin) && chan_ok(Cout),
               "pyro_conv3_backward_weight: invalid sizes");
  // the boxes need 16-byte aligned tensors; others are gathered, and so is a
  // gradient with sums that are not finite
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy);
  const bool boxes = conv3_wgrad_fits(Cin, Cout) && at % 16 == 0;
  const int n = Cout * 27 * Cin;
  DevBuf err;  // the error and bad flags, then the boxes' sums
  int rc = err.alloc(16 + (boxes ? (size_t)n * 8 : 0));
  if (rc != PYRO_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int *E = err.as<int>(), *bad = boxes ? E + 1 : nullptr;
  cudaError_t e = cudaSuccess;
  if (boxes) {
    double* sums = err.as<double>() + 2;
    e = conv3_wgrad_tma((const bf16*)x, Cin, (const bf16*)dy, Cout, 0, nx, ny, nz, nb, sums, E,
                        bad, st);
    if (e == cudaSuccess) {
      k_add_unless<<<(n + 255) / 256, 256, 0, st>>>(sums, n, bad, dw);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess)
    e = conv3_wgrad_gather((const bf16*)x, Cin, (const bf16*)dy, Cout, nx, ny, nz, nb, dw, E, bad,
                           st);
  return finish(e, err, st, "pyro_conv3_backward_weight");
}

}  // extern "C"
