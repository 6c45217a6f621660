// net.h — the learned pressure stage: a 3-level 3D convolutional
// encoder-decoder (16/32/64 channels, 3x3x3 convolutions, BF16 weights and
// activations, FP32 accumulation in TMEM) that maps a right-hand side and the
// solid mask to a pressure estimate, with its training (MSE loss, backward
// pass, Adam on FP32 master weights).
//
//   in0 = [b / s, solid]                      level 0, 2 channels
//   e0a = relu(conv1(in0))   e0 = relu(conv2(e0a))          16
//   p1  = avgpool2(e0)       e1a = relu(conv3(p1)), e1 = relu(conv4(e1a))  32
//   p2  = avgpool2(e1)       e2a = relu(conv5(p2)), e2 = relu(conv6(e2a))  64
//   c1  = [up2(e2), e1]      d1  = relu(conv7(c1))          96 -> 32
//   c0  = [up2(d1), e0]      d0  = relu(conv8(c0))          48 -> 16
//   out = conv9(d0)                                         16 -> 1 (FP32)
//   phi = out * out_scale * s * h^2 on fluid cells, 0 in solids
//
// s is the root mean square of b over the fluid cells of each volume, so
// the map is linear in the scale of b, as the Poisson solution is.  Pooling
// halves with ceil (a coarse cell averages its children inside the volume);
// up2 copies a coarse cell to its children.  Activations of C channels are
// stored as C / 8 planes of [volume][z][y][x][8 channels] (C a multiple of
// 8), the 2-channel input as [volume][z][y][x][2].
#pragma once

#include <cuda_bf16.h>

#include "runtime.h"

namespace pyro {

constexpr int NET_LAYERS = 9;
struct NetLayer {
  int cin, cout, level, relu;
};
// conv1 .. conv9 in order
constexpr NetLayer NET_SPEC[NET_LAYERS] = {{2, 16, 0, 1},  {16, 16, 0, 1}, {16, 32, 1, 1},
                                           {32, 32, 1, 1}, {32, 64, 2, 1}, {64, 64, 2, 1},
                                           {96, 32, 1, 1}, {48, 16, 0, 1}, {16, 1, 0, 0}};

struct NetVol {
  int nx, ny, nz, nb;
  size_t voxels() const { return (size_t)nx * ny * nz * nb; }
  NetVol half() const { return NetVol{(nx + 1) / 2, (ny + 1) / 2, (nz + 1) / 2, nb}; }
  bool operator==(const NetVol& o) const {
    return nx == o.nx && ny == o.ny && nz == o.nz && nb == o.nb;
  }
};

cudaError_t conv3_forward(const __nv_bfloat16* x, int C, int nx, int ny, int nz, int nb,
                          const __nv_bfloat16* w, int Cout, const float* bias, int relu,
                          __nv_bfloat16* y_bf16, float* y_f32, int* err, cudaStream_t st);
cudaError_t conv3_backward_data(const __nv_bfloat16* dy, int Cout, int nx, int ny, int nz,
                                int nb, const __nv_bfloat16* w, int Cin,
                                const __nv_bfloat16* act, __nv_bfloat16* dx_bf16, float* dx_f32,
                                int* err, cudaStream_t st);
// Weight gradient by the gather GEMM, accumulated into dw (FP32); nothing when
// only_if is given and *only_if is 0.
cudaError_t conv3_wgrad_gather(const __nv_bfloat16* x, int Cin, const __nv_bfloat16* dy, int Cout,
                               int nx, int ny, int nz, int nb, float* dw, int* err,
                               const int* only_if, cudaStream_t st);

// Direct convolution on the CUDA cores for 2 -> 16 channels on [V][2] inputs
// and 16 -> 1, FP32 sums in a fixed order.
bool conv3_direct_fits(int C, int Cout);
cudaError_t conv3_direct(const __nv_bfloat16* x, int C, int nx, int ny, int nz, int nb,
                         const __nv_bfloat16* w, int Cout, const float* bias, int relu,
                         __nv_bfloat16* y_bf16, float* y_f32, cudaStream_t st);

// K steps of 16 voxels that one of its sums takes, for V voxels.
int conv3_gather_steps(int Cin, long V);

// TMA-staged convolution (k_conv3.cu) on tap-major weights prepared by
// conv3_prep_weights: input channels K a multiple of 16, or (pack) the one
// channel of a tensor packed by conv3_pack_grad.  fine (BF16
// output of a multiple of 16 channels): every voxel's result is written to its
// children in the first planes of a tensor over that volume, y_bf16.
// old_weights: weights and bias were complete before the launch that precedes
// this one on the stream started, so they may be read while it ends.
cudaError_t conv3_prep_weights(const __nv_bfloat16* w, int Cout, int Cin, int backward,
                               __nv_bfloat16* w_tap, cudaStream_t st);
cudaError_t conv3_tma(const __nv_bfloat16* x, int K, bool pack, int nx, int ny, int nz, int nb,
                      const __nv_bfloat16* w_tap, int N, const float* bias, int relu,
                      const __nv_bfloat16* mask, __nv_bfloat16* y_bf16, float* y_f32, int* err,
                      cudaStream_t st, const NetVol* fine = nullptr, bool old_weights = false);

// The driver's cuTensorMapEncodeTiled (PFN_cuTensorMapEncodeTiled_v12000), or
// null.
void* tensor_map_encoder();

// Weight gradient with TMA-staged operands (k_wgrad.cu), accumulated into dw
// (FP64): input channels in planes of 8 and output channels a multiple of 16;
// pack 1: one output channel, gr packed by conv3_pack_grad; pack 2: two input
// channels, x packed by conv3_pack_input.  *bad is set when a sum is not
// finite: dw then holds NaN also where conv3_wgrad_gather does not.
bool conv3_wgrad_fits(int Cin, int Cout);
cudaError_t conv3_wgrad_tma(const __nv_bfloat16* x, int Cin, const __nv_bfloat16* gr, int Cout,
                            int pack, int nx, int ny, int nz, int nb, double* dw, int* err,
                            int* bad, cudaStream_t st);
// The three x-shifts of a gradient of one channel ([V]) or of an input of two
// ([V][2]) as one plane of 8 channels, 0 outside the row and past the shifts:
// dst[u][j] = src[u - (j - 1)], dst[u][2 j + c] = src[u + j - 1][c].
cudaError_t conv3_pack_grad(const __nv_bfloat16* src, int nx, int ny, int nz, int nb,
                            __nv_bfloat16* dst, cudaStream_t st);
cudaError_t conv3_pack_input(const __nv_bfloat16* src, int nx, int ny, int nz, int nb,
                             __nv_bfloat16* dst, cudaStream_t st);

// The same of the network's layers with bad[l] set (device), in one launch.
struct WgradJob {
  const __nv_bfloat16 *x, *g;
  NetVol v;
  float* dw;
};
cudaError_t conv3_wgrad_gathers(const WgradJob (&jobs)[NET_LAYERS], const int* bad, int* err,
                                cudaStream_t st);

}  // namespace pyro

// Parameters: all weights first ([Cout][27][Cin] per layer, layers in
// order), then all biases; the BF16 weight copy mirrors the weight part.
struct PyroNet {
  size_t w_off[pyro::NET_LAYERS + 1] = {};  // into the weight part
  size_t b_off[pyro::NET_LAYERS + 1] = {};  // into the bias part (after weights)
  size_t n_w = 0, n_params = 0;
  float out_scale = 1.0f;
  float w_phi = 1.0f, w_res = 0.0f;  // loss weights (pyro_net_set_loss)
  pyro::DevBuf master, grad, adam_m, adam_v, wbf;  // FP32 x n_params; BF16 x n_w
  pyro::DevBuf wtf, wtb;  // tap-major BF16 weights for the forward / backward-data TMA path
  pyro::DevBuf scal;   // FP64 device scalars: [0] loss, [1] grad sum of squares, then 2 per volume
  pyro::DevBuf err;    // tensor-core wait error flag
  double* host_scal = nullptr;
  long adam_t = 0;
  // activation buffers for the current volume shape
  pyro::NetVol vol{0, 0, 0, 0};
  bool has_bwd = false;
  pyro::DevBuf in0, e0a, p1, e1a, p2, e2a, c1, c0, d0, out, res;
  // skip activations e0 (16 channels, level 0) and e1 (32, level 1): the
  // last 2 / 4 planes of the concatenations c0 / c1
  __nv_bfloat16* skip0() const { return c0.as<__nv_bfloat16>() + (size_t)4 * vol.voxels() * 8; }
  __nv_bfloat16* skip1() const {
    return c1.as<__nv_bfloat16>() + (size_t)8 * vol.half().voxels() * 8;
  }
  pyro::DevBuf wsum;  // weight gradients' sums in FP64 (backward)
  pyro::DevBuf pk;  // packed x-shifts of the output gradient, then of the input (backward)
  pyro::DevBuf g9, g8, gc0, g7, gc1, g6, g5, gp2, g4, g3, gp1, g2, g1;
  cudaStream_t stream = nullptr;

  int init();
  ~PyroNet();
  int ensure(pyro::NetVol v, bool bwd);
  const float* bias(int l) const { return master.as<float>() + n_w + b_off[l]; }
  const __nv_bfloat16* w(int l) const { return wbf.as<__nv_bfloat16>() + w_off[l]; }
  const __nv_bfloat16* wf(int l) const { return wtf.as<__nv_bfloat16>() + w_off[l]; }
  const __nv_bfloat16* wb(int l) const { return wtb.as<__nv_bfloat16>() + w_off[l]; }
  // rebuild wtf / wtb from the BF16 weights
  int refresh_taps(cudaStream_t st);
  // Forward pass; out holds the network output (FP32, per voxel).
  int forward(const float* b, const uint32_t* flags, pyro::NetVol v, cudaStream_t st);
  // Loss (weights w_phi, w_res; see pyro_net_set_loss) and the full
  // backward pass; gradients are accumulated into `grad` (zeroed here).
  int loss_backward(const float* b, const uint32_t* flags, const float* phi_t, float h,
                    pyro::NetVol v, cudaStream_t st);
  int adam(float lr, float clip, cudaStream_t st);
  // phi = out * out_scale * s * h^2 (fluid), 0 (solid)
  int output(const uint32_t* flags, float h, float* phi, pyro::NetVol v, cudaStream_t st);
  int check_err(cudaStream_t st);
  // loss of the last loss_backward from the device scalars (synchronises)
  int read_loss(cudaStream_t st, double* loss);
};
