// k_mg.cu — geometric multigrid kernels for the pressure Poisson system.
//
// Operator on every level (src/shaders/mg.wgsl:2,25-35):
//   (sum over fluid neighbours of phi_n - cnt * phi) / h^2 = b
// A neighbour below the floor (y < 0) is skipped (Neumann floor), one outside
// the other faces counts in cnt with phi = 0 (Dirichlet sides and top), a
// solid neighbour is skipped (Neumann at solids).  bc_mode 1 keeps only the
// top face Dirichlet.  Neighbours are visited in the reference's order
// (+x, -x, +y, -y, +z, -z) so sums round identically.
//
//   mg_resid     mg.wgsl:122-158 sums of r^2 and b^2
//   mg_coarse    the whole coarsest-level solve (src/sim.rs:473: 80 SOR
//                sweeps at omega 1.6) in one thread-block cluster with the
//                level in distributed shared memory, replacing 160 dispatches.
// The per-colour smoother, the restriction and the prolongation of every
// other level run on per-cell neighbour masks (k_mgf.cu).
#include <cooperative_groups.h>
#include <cstdlib>
#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.h"

namespace pyro {

namespace {

// Storage of phi and b: FP32 (the reference) or BF16 (the low-precision
// preconditioner); arithmetic is FP32 either way.
__device__ __forceinline__ float ldv(const float* p) { return *p; }
__device__ __forceinline__ float ldv(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void stv(float* p, float v) { *p = v; }
__device__ __forceinline__ void stv(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

constexpr int BX = 32, BY = 4, BZ = 2;

inline dim3 grid_for(int x, int y, int z) {
  return dim3((unsigned)((x + BX - 1) / BX), (unsigned)((y + BY - 1) / BY),
              (unsigned)((z + BZ - 1) / BZ));
}

struct Lvl {
  int nx, ny, nz;
  __device__ __forceinline__ bool inb(int x, int y, int z) const {
    return (unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny && (unsigned)z < (unsigned)nz;
  }
  __device__ __forceinline__ int idx(int x, int y, int z) const { return x + nx * (y + ny * z); }
};

// Accumulate the 6-neighbour sum and count of cell (x,y,z).
template <typename PhiAt, typename SolidAt>
__device__ __forceinline__ void neigh_sum(const Lvl& d, int x, int y, int z, int bc_mode,
                                          PhiAt phi_at, SolidAt solid_at, float& sum,
                                          float& cnt) {
  sum = 0.0f;
  cnt = 0.0f;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    int nx_ = x + (k == 0) - (k == 1);
    int ny_ = y + (k == 2) - (k == 3);
    int nz_ = z + (k == 4) - (k == 5);
    if (ny_ < 0) continue;
    if (!d.inb(nx_, ny_, nz_)) {
      if (bc_mode == 0 || ny_ >= d.ny) cnt += 1.0f;
      continue;
    }
    int j = d.idx(nx_, ny_, nz_);
    if (solid_at(j)) continue;
    sum += phi_at(j);
    cnt += 1.0f;
  }
}

template <typename TS>
__device__ __forceinline__ float resid_cell(const Lvl& d, float h2, const TS* __restrict__ p,
                                            const TS* __restrict__ b,
                                            const uint32_t* __restrict__ f, int x, int y, int z,
                                            int bc_mode) {
  int i = d.idx(x, y, z);
  if (__ldg(f + i) == 1u) return 0.0f;
  float pcen = ldv(p + i);
  float sum, cnt;
  neigh_sum(
      d, x, y, z, bc_mode, [&](int j) { return ldv(p + j); },
      [&](int j) { return __ldg(f + j) == 1u; }, sum, cnt);
  return ldv(b + i) - (sum - cnt * pcen) / h2;
}

__global__ void __launch_bounds__(256) k_mg_resid(Lvl d, float h2, const float* __restrict__ p,
                                                  const float* __restrict__ b,
                                                  const uint32_t* __restrict__ f, int bc_mode,
                                                  float* __restrict__ stats) {
  __shared__ float sh[2 * 32];
  int x = blockIdx.x * BX + threadIdx.x;
  int y = blockIdx.y * BY + threadIdx.y;
  int z = blockIdx.z * BZ + threadIdx.z;
  float vals[2] = {0.0f, 0.0f};  // r^2, b^2
  if (d.inb(x, y, z)) {
    int i = d.idx(x, y, z);
    if (__ldg(f + i) != 1u) {
      float r = resid_cell(d, h2, p, b, f, x, y, z, bc_mode);
      float bi = __ldg(b + i);
      vals[0] = r * r;
      vals[1] = bi * bi;
    }
  }
  block_stats<2>(sh, vals, stats, {10, 11}, 0u);
}

// ------------------------------------------------------------ coarse solve
// The coarsest level is swept 80 times per V-cycle (src/sim.rs:473), 160
// dependent red-black passes over ~1-30 k cells.  One thread-block cluster
// runs them all in a single launch: CTA r of the C that own planes (one plane
// each at least; a cluster's further CTAs only join its barriers) owns z-planes
// [r nz / C, (r + 1) nz / C) of phi in its shared memory, with a ghost plane on
// either side.
//
// What bounds it is the latency of a pass, so a pass costs one block barrier
// and one message to each neighbour: a thread that has updated a cell of the
// slab's first or last plane stores it straight into the neighbour's ghost
// plane with st.async, which also counts its bytes on the neighbour's
// mbarrier, and the neighbour's threads wait for that count before they start
// the next pass.  (Reading the neighbour's planes remotely between two
// barriers of the whole cluster took 0.88 us a pass: a cluster barrier is
// 0.24-0.32 us and a remote read 0.24.)
// A ghost plane is not overwritten while it is read: a neighbour sends in
// pass p + 1 only after it has all of this CTA's cells of pass p, and a thread
// here sends a cell after it has loaded that cell's ghost neighbour; in pass
// p + 1 itself this CTA reads the other colour of the ghosts.  The last pass
// sends nothing, so no store is in flight to a CTA that ends.
//
// The two colours live in separate arrays, indexed by the reference
// smoother's own numbering q = hx + hxn (y + ny z), x = 2 hx + ((y + z + c) &
// 1) (mg.wgsl:17-19): the y and z neighbours of cell q are q +- hxn and
// q +- hxn ny of the other colour, the x neighbours q and q - 1 or q + 1, so
// loads and messages of a warp are contiguous.  Thread t holds cells t + T k
// (k < K) of each colour, with the neighbours' addresses, the count and h^2 b
// in registers.  The
// arithmetic per cell is the reference's, in the same order, so the result
// equals 160 separate passes bit for bit.
// Measured, 80 sweeps: 20 x 40 x 20 144 -> 82 us, 16 x 30 x 16 113 -> 53 us,
// 8 x 20 x 8 101 -> 43 us (0.16 us of a pass is one warp's chain of loads,
// additions, division and barrier, 0.09 us the message).
constexpr int COARSE_MAX_CLUSTER = 16;
constexpr int COARSE_SMEM = 200 * 1024;
// Threads per CTA at most with K cells per thread and colour (each keeps
// ~22 K registers of cell state).
constexpr int coarse_threads(int K) { return K == 1 ? 1024 : K == 2 ? 640 : 512; }
constexpr uint32_t COARSE_SPINS = 1u << 22;

// A cell of a thread: shared-memory addresses of its six neighbours (a place
// that holds 0 where there is none to add: the sum starts at +0 and never
// becomes -0, so adding +0 leaves its bits) and of itself.
struct CoarseCell {
  uint32_t nb[6], self;
  float cnt, rcp, hb;
  uint32_t to;  // bit 0: updated, bits 1 / 2: sent to the CTA below / above
};

__device__ __forceinline__ float lds(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// x / c for c = 1 .. 6 and rcp = 1 / c rounded: Markstein's correction of
// x rcp (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990, theorem on division from a correctly rounded
// reciprocal).  Equal to x / c bit for bit for 2^-100 <= |x| < 2^100 and for
// x = +0 (every FP32 value checked against the division); other values take
// the division.
__device__ __forceinline__ float div_count(float x, float c, float rcp) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  if (u - 0x0d800000u < 0x64000000u || u == 0u) {
    const float q = x * rcp;
    return __fmaf_rn(__fmaf_rn(-q, c, x), rcp, q);
  }
  return x / c;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// The shared::cluster address of this CTA's address `a` in CTA `rank`.
__device__ __forceinline__ uint32_t map_rank(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void send_async(uint32_t addr, float v, uint32_t mbar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
      "r"(__float_as_uint(v)), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ bool wait_cluster(uint32_t mbar, uint32_t parity) {
  for (uint32_t i = 0; i < COARSE_SPINS; i++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// ORDER of an iteration's colours: red-black, black-red, or the two in turn.
// SMOOTH: the sweeps of a smoother: neighbours from the level's masks (`meta`
// instead of the flags), and a cell's value is rounded to the storage type
// after every pass, as separate pass launches store it.
enum SweepOrder { RED_BLACK, BLACK_RED, ALTERNATE };

template <typename TS, int K, int ORDER, bool SMOOTH>
__global__ void __launch_bounds__(coarse_threads(K), 1)
    k_mg_coarse_rb(Lvl d, float h2, const TS* __restrict__ b, const uint32_t* __restrict__ f,
                   const uint8_t* __restrict__ meta, TS* __restrict__ p, int iters, float omega,
                   int bc_mode) {
  namespace cg = cooperative_groups;
  pdl_trigger();
  pdl_wait();
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ float sp[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ float zero;
  const int T = (int)blockDim.x;
  const int C = min((int)cl.num_blocks(), d.nz);
  const int rank = (int)cl.block_rank();
  if (rank >= C) {  // no planes
    cl.sync();
    cl.sync();
    return;
  }
  const int z0 = rank * d.nz / C, z1 = (rank + 1) * d.nz / C, planes = z1 - z0;
  const int hxn = (d.nx + 1) / 2, pl = hxn * d.ny;
  const int cap = ((d.nz + C - 1) / C + 2) * pl;  // floats of one colour, the same in every CTA
  // sp[c cap + q]: colour c, plane 0 and plane planes + 1 are the ghosts
  const int total = (planes + 2) * pl;
  for (int q = threadIdx.x; q < total; q += T) {
    const int hx = q % hxn, r = q / hxn, y = r % d.ny, z = z0 - 1 + r / d.ny;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int x = 2 * hx + ((y + z + c) & 1);
      sp[c * cap + q] = d.inb(x, y, z) ? ldv(p + d.idx(x, y, z)) : 0.0f;
    }
  }
  const uint32_t bar0 = smem_addr(&bar[0]), sp0 = smem_addr(sp);
  const uint32_t expect = 4u * (uint32_t)pl * (uint32_t)((rank > 0) + (rank + 1 < C));
  if (threadIdx.x == 0) {
    zero = 0.0f;
    for (int i = 0; i < 2; i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // what turns a cell's own address into its place at a neighbour: the ghost
  // plane above the last plane of the CTA below, or the one below the first
  // plane of the CTA above
  uint32_t lo_off = 0, hi_off = 0, lo_bar = 0, hi_bar = 0;
  if (rank > 0) {
    const int below = z0 - (rank - 1) * d.nz / C;  // its planes
    lo_off = map_rank(sp0, rank - 1) + 4u * (uint32_t)(below * pl) - sp0;
    lo_bar = map_rank(bar0, rank - 1);
  }
  if (rank + 1 < C) {
    hi_off = map_rank(sp0, rank + 1) - 4u * (uint32_t)(planes * pl) - sp0;
    hi_bar = map_rank(bar0, rank + 1);
  }
  CoarseCell cell[2][K];
#pragma unroll
  for (int c = 0; c < 2; c++)
#pragma unroll
    for (int k = 0; k < K; k++) {
      CoarseCell& e = cell[c][k];
      const uint32_t za = smem_addr(&zero);
      e.self = za;
#pragma unroll
      for (int n = 0; n < 6; n++) e.nb[n] = za;
      e.cnt = e.rcp = 1.0f;
      e.hb = 0.0f;
      e.to = 0u;
      const int v = threadIdx.x + T * k;
      if (v >= planes * pl) continue;
      const int hx = v % hxn, r = v / hxn;
      const int y = r % d.ny, zl = r / d.ny, z = z0 + zl;
      const int par = (y + z + c) & 1, x = 2 * hx + par;
      const uint32_t own = sp0 + 4u * (uint32_t)(c * cap + v + pl);
      const uint32_t oth = sp0 + 4u * (uint32_t)((1 - c) * cap + v + pl);
      e.self = own;
      // every cell of a boundary plane is sent, updated or not: the number of
      // bytes a CTA waits for does not depend on the flags
      if (zl == 0 && rank > 0) e.to |= 2u;
      if (zl == planes - 1 && rank + 1 < C) e.to |= 4u;
      if (x >= d.nx) continue;
      const int gi = d.idx(x, y, z);
      const int step[6] = {par, par - 1, hxn, -hxn, pl, -pl};
      float cnt = 0.0f;
      const uint32_t m = SMOOTH ? meta[gi] : 0u;  // bits 0-5: fluid neighbours, 6: solid
#pragma unroll
      for (int n = 0; n < 6; n++) {
        const int ax = x + (n == 0) - (n == 1), ay = y + (n == 2) - (n == 3),
                  az = z + (n == 4) - (n == 5);
        if (ay < 0) continue;
        if (!d.inb(ax, ay, az)) {
          if (bc_mode == 0 || ay >= d.ny) cnt += 1.0f;
          continue;
        }
        if (SMOOTH ? !((m >> n) & 1u) : f[d.idx(ax, ay, az)] == 1u) continue;
        e.nb[n] = oth + 4u * (uint32_t)step[n];
        cnt += 1.0f;
      }
      if (!(SMOOTH ? (m & 0x40u) != 0u : f[gi] == 1u) && cnt >= 0.5f) {
        e.to |= 1u;
        e.cnt = cnt;
        e.rcp = 1.0f / cnt;
      }
      e.hb = h2 * ldv(b + gi);
    }
  cl.sync();  // the ghosts are loaded and every mbarrier is initialised
  bool ok = true;
  const int npass = 2 * iters;
  // pass number `n` on colour c
  auto pass = [&](const CoarseCell (&cells)[K], int n) {
    const bool send = C > 1 && n + 1 < npass;
    const uint32_t bo = 8u * (uint32_t)(n & 1);
    // this pass's messages to this CTA are counted on bar[n & 1]
    if (send && threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar0 + bo),
                   "r"(expect)
                   : "memory");
    // after a wait that ran out the passes go on without waiting
    if (C > 1 && n > 0 && ok) ok = wait_cluster(bar0 + 8u - bo, (uint32_t)((n - 1) >> 1) & 1u);
    float nbv[K][6], ownv[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
#pragma unroll
      for (int j = 0; j < 6; j++) nbv[k][j] = lds(cells[k].nb[j]);
      ownv[k] = lds(cells[k].self);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const CoarseCell& e = cells[k];
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 6; j++) sum += nbv[k][j];
      float v = wmix(ownv[k], div_count(sum - e.hb, e.cnt, e.rcp), omega);
      if (SMOOTH && sizeof(TS) == 2) v = __bfloat162float(__float2bfloat16_rn(v));
      if (e.to & 1u) sts(e.self, v);
      else v = ownv[k];
      if (send) {
        if (e.to & 2u) send_async(e.self + lo_off, v, lo_bar + bo);
        if (e.to & 4u) send_async(e.self + hi_off, v, hi_bar + bo);
      }
    }
    __syncthreads();
  };
#pragma unroll 1
  for (int it = 0; it < iters; it++) {
    if (ORDER == BLACK_RED || (ORDER == ALTERNATE && (it & 1))) {
      pass(cell[1], 2 * it);
      pass(cell[0], 2 * it + 1);
    } else {
      pass(cell[0], 2 * it);
      pass(cell[1], 2 * it + 1);
    }
  }
  // A wait that ran out: the level becomes NaN, which the residual statistics
  // and the solvers' convergence test report.
  const bool all_ok = __syncthreads_and(ok) != 0;
  for (int v = threadIdx.x; v < planes * pl; v += T) {
    const int hx = v % hxn, r = v / hxn, y = r % d.ny, z = z0 + r / d.ny;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int x = 2 * hx + ((y + z + c) & 1);
      if (x < d.nx)
        stv(p + d.idx(x, y, z), all_ok ? sp[c * cap + v + pl] : __int_as_float(0x7fc00000));
    }
  }
  cl.sync();  // no CTA ends while another may still send to it
}

__global__ void k_f32_to_bf16(const float* __restrict__ a, __nv_bfloat16* __restrict__ b,
                              size_t n) {
  pdl_trigger();
  pdl_wait();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = __float2bfloat16_rn(a[i]);
}
__global__ void k_bf16_to_f32(const __nv_bfloat16* __restrict__ a, float* __restrict__ b,
                              size_t n) {
  pdl_trigger();
  pdl_wait();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = __bfloat162float(a[i]);
}

// Shared memory of a CTA: two colours of its planes and two ghost planes.
size_t coarse_smem(Dims3 d, int C) {
  C = std::min(C, d.nz);
  return (size_t)((d.nz + C - 1) / C + 2) * ((d.nx + 1) / 2) * d.ny * 2 * 4;
}

// Cluster size, cells per thread and colour and threads per CTA for a level;
// C = 0 when it does not fit.  A CTA per plane, up to the largest cluster: a
// message to a neighbour costs less than the warps that more planes per CTA
// would add (20 x 30 x 20: 67 us on 16 CTAs, 89 on 8; 20 x 40 x 12: 63 us on
// 16 of which 12 have a plane, 84 on 8; 16 x 32 x 6: 51 us on 8, 62 on 4).  As
// few cells per thread as fit: the same cells in fewer warps wait longer (two
// per thread instead of one: 20 x 40 x 20 88 us against 82, 16 x 30 x 16 65
// against 53).
struct CoarsePlan {
  int C = 0, K = 0, T = 0;
};
CoarsePlan coarse_plan(Dims3 d, int max_cluster) {
  CoarsePlan pl;
  int C = 2;
  while (C < max_cluster && C < d.nz) C *= 2;
  const int planes = (d.nz + C - 1) / C;
  const long vpc = (long)((d.nx + 1) / 2) * d.ny * planes;
  if (coarse_smem(d, C) > (size_t)COARSE_SMEM) return pl;
  for (int K : {1, 2, 4}) {
    const long T = ((vpc + K - 1) / K + 31) / 32 * 32;
    if (T > coarse_threads(K)) continue;
    pl.C = C;
    pl.K = K;
    pl.T = (int)T;
    return pl;
  }
  return pl;
}

template <typename TS, int K, int ORDER, bool SMOOTH>
cudaError_t coarse_launch(const CoarsePlan& pl, Dims3 d, float h, const TS* b, const uint32_t* f,
                          const uint8_t* meta, TS* p, int iters, float omega, int bc_mode,
                          cudaStream_t st) {
  auto kern = k_mg_coarse_rb<TS, K, ORDER, SMOOTH>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       COARSE_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)pl.C, 1, 1);
  cfg.blockDim = dim3((unsigned)pl.T, 1, 1);
  cfg.dynamicSmemBytes = coarse_smem(d, pl.C);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)pl.C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_pdl
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, Lvl{d.nx, d.ny, d.nz}, h * h, b, f, meta, p, iters,
                            omega, bc_mode);
}

// The largest cluster this device co-schedules for the coarse kernel (16
// where non-portable cluster sizes are allowed, else 8), found once.
int coarse_max_cluster() {
  static int mc = 0;
  if (mc) return mc;
  auto kern = k_mg_coarse_rb<float, 2, RED_BLACK, false>;
  int q = 8;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
          cudaSuccess &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, COARSE_SMEM) ==
          cudaSuccess) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(COARSE_MAX_CLUSTER, 1, 1);
    c.blockDim = dim3(coarse_threads(2), 1, 1);
    c.dynamicSmemBytes = 64 * 1024;
    if (cudaOccupancyMaxPotentialClusterSize(&q, kern, &c) != cudaSuccess) q = 8;
  }
  mc = q >= COARSE_MAX_CLUSTER ? COARSE_MAX_CLUSTER : 8;
  return mc;
}

int coarse_cluster_size(Dims3 d) { return coarse_plan(d, COARSE_MAX_CLUSTER).C; }

template <typename TS>
cudaError_t mg_coarse_t(Dims3 d, float h, const TS* b, const uint32_t* f, TS* p, int iters,
                        float omega, int bc_mode, cudaStream_t st, int symmetric = 0) {
  const CoarsePlan pl = coarse_plan(d, coarse_max_cluster());
  if (pl.C == 0) return cudaErrorInvalidValue;
#define PYRO_COARSE(K)                                                                       \
  case K:                                                                                   \
    return symmetric ? coarse_launch<TS, K, ALTERNATE, false>(pl, d, h, b, f, nullptr, p,   \
                                                              iters, omega, bc_mode, st)    \
                     : coarse_launch<TS, K, RED_BLACK, false>(pl, d, h, b, f, nullptr, p,   \
                                                              iters, omega, bc_mode, st)
  switch (pl.K) {
    PYRO_COARSE(1);
    PYRO_COARSE(2);
    PYRO_COARSE(4);
    default: return cudaErrorInvalidValue;
  }
#undef PYRO_COARSE
}

template <typename TS>
cudaError_t mg_sweeps_t(Dims3 d, float h, const TS* b, const uint8_t* meta, TS* p, int iters,
                        float omega, int black_first, int bc_mode, cudaStream_t st) {
  const CoarsePlan pl = coarse_plan(d, coarse_max_cluster());
  if (pl.C == 0 || pl.K != 1) return cudaErrorInvalidValue;
  return black_first ? coarse_launch<TS, 1, BLACK_RED, true>(pl, d, h, b, nullptr, meta, p, iters,
                                                             omega, bc_mode, st)
                     : coarse_launch<TS, 1, RED_BLACK, true>(pl, d, h, b, nullptr, meta, p, iters,
                                                             omega, bc_mode, st);
}

}  // namespace

bool mg_coarse_fits(Dims3 d) { return coarse_cluster_size(d) != 0; }

// Levels with one cell of a colour per thread: four cells per thread make a
// pass longer than a launch (32 x 60 x 32 in the V-cycles on 128 x 240 x 128:
// 1043 us against 968 with a launch per pass).
bool mg_sweeps_fit(Dims3 d) {
  const CoarsePlan pl = coarse_plan(d, coarse_max_cluster());
  return pl.C != 0 && pl.K == 1;
}

// A launch sets its cells up once for all passes, which pays for the eight of
// MGPCG's smoother on every level that fits (us, cluster against passes: 16 x 40
// x 16 7.7 / 12.6, 19 x 46 x 19 11.1 / 12.1, 40 x 50 x 16 12.2 / 13.7, BF16 11.1
// / 14.0 and 12.4 / 12.5) and for the four of the V-cycles up to 320 cells of a
// colour per CTA (16 x 32 x 16 6.2 / 6.3, 16 x 40 x 16 6.4 / 6.4; beyond, 16 x
// 48 x 16 6.7 / 6.3, 19 x 46 x 19 9.0 / 5.8).
bool mg_sweeps_pay(Dims3 d, int passes) {
  const CoarsePlan pl = coarse_plan(d, coarse_max_cluster());
  return pl.C != 0 && pl.K == 1 && (passes >= 8 || pl.T <= 320);
}

cudaError_t launch_mg_sweeps(Dims3 d, float h, const void* b, const uint8_t* meta, void* p,
                             int iters, float omega, int black_first, int bc_mode, bool bf16,
                             cudaStream_t st) {
  if (bf16)
    return mg_sweeps_t<__nv_bfloat16>(d, h, (const __nv_bfloat16*)b, meta, (__nv_bfloat16*)p,
                                      iters, omega, black_first, bc_mode, st);
  return mg_sweeps_t<float>(d, h, (const float*)b, meta, (float*)p, iters, omega, black_first,
                            bc_mode, st);
}

cudaError_t launch_mg_resid(Dims3 d, float h, const float* p, const float* b, const uint32_t* f,
                            int bc_mode, float* stats, cudaStream_t st) {
  k_mg_resid<<<grid_for(d.nx, d.ny, d.nz), dim3(BX, BY, BZ), 0, st>>>(
      Lvl{d.nx, d.ny, d.nz}, h * h, p, b, f, bc_mode, stats);
  return cudaGetLastError();
}

cudaError_t launch_mg_coarse(Dims3 d, float h, const float* b, const uint32_t* f, float* p,
                             int iters, float omega, int bc_mode, cudaStream_t st) {
  return mg_coarse_t<float>(d, h, b, f, p, iters, omega, bc_mode, st);
}

// ---- BF16-storage hierarchy (MGPCG preconditioner) -----------------------
cudaError_t launch_f32_to_bf16(const float* a, void* b, size_t n, cudaStream_t st) {
  return launch_pdl(k_f32_to_bf16, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, a,
                    (__nv_bfloat16*)b, n);
}
cudaError_t launch_bf16_to_f32(const void* a, float* b, size_t n, cudaStream_t st) {
  return launch_pdl(k_bf16_to_f32, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st,
                    (const __nv_bfloat16*)a, b, n);
}
cudaError_t launch_mg_coarse_sym(Dims3 d, float h, const float* b, const uint32_t* f, float* p,
                                 int iters, float omega, int bc_mode, cudaStream_t st) {
  return mg_coarse_t<float>(d, h, b, f, p, iters, omega, bc_mode, st, 1);
}
cudaError_t launch_mg_coarse_sym_bf16(Dims3 d, float h, const void* b, const uint32_t* f,
                                      void* p, int iters, float omega, int bc_mode,
                                      cudaStream_t st) {
  return mg_coarse_t<__nv_bfloat16>(d, h, (const __nv_bfloat16*)b, f, (__nv_bfloat16*)p, iters,
                                    omega, bc_mode, st, 1);
}

}  // namespace pyro
