// conv.cuh — activation layout of the learned stage (net.cu) and the epilogue
// shared by its convolution kernels (k_conv.cu, k_conv3.cu).
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace pyro {
namespace {

using bf16 = __nv_bfloat16;

// Activation layout: a tensor of C channels over V voxels with C a multiple of
// 8 is stored as C / 8 planes of [V][8 channels] (a plane is one 16-byte chunk
// per voxel, so a TMA box along x reads long contiguous rows); other channel
// counts (the 2-channel input, 1-channel gradients) as [V][C].  Element offset
// of channel c of voxel v:
__device__ __forceinline__ size_t act_off(size_t v, int c, int C, size_t V) {
  return (C & 7) ? v * C + c : ((size_t)(c >> 3) * V + v) * 8 + (c & 7);
}

// Forward / backward data: row = voxel.  out_bf16 [V][Nout] with optional
// bias and ReLU, or out_f32 [V][Nout]; `mask` (BF16 activations of the layer
// input, [V][Nout]) zeroes the gradient where the input was <= 0 (ReLU).
struct ConvEpi {
  bf16* out_bf16;
  float* out_f32;
  const float* bias;
  const bf16* mask;
  int V, Nout, relu;
  // up != 0: out_bf16 is over a volume of twice the size (fx, fy, fz; fV voxels
  // in all), and a voxel's result goes to its children there (k_conv3.cu)
  int up, fx, fy, fz, fV;
  __device__ void operator()(int m, int col, const float (&v)[16]) const {
    if (m < 0 || m >= V) return;
    const uintptr_t at = reinterpret_cast<uintptr_t>(out_bf16) |
                         reinterpret_cast<uintptr_t>(mask) | reinterpret_cast<uintptr_t>(bias);
    if (out_bf16 && (Nout & 15) == 0 && (at & 15) == 0) {
      // 16 channels of one row: 32 contiguous bytes, two 16-byte stores
      float a[16];
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        float4 bb = bias ? __ldg(reinterpret_cast<const float4*>(bias + col + j))
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        a[j] = v[j] + bb.x;
        a[j + 1] = v[j + 1] + bb.y;
        a[j + 2] = v[j + 2] + bb.z;
        a[j + 3] = v[j + 3] + bb.w;
      }
      if (!bias) {
#pragma unroll
        for (int j = 0; j < 16; j++) a[j] = v[j];
      }
      if (relu) {
#pragma unroll
        for (int j = 0; j < 16; j++) a[j] = fmaxf(a[j], 0.0f);
      }
      if (mask) {
        const uint4* mp = reinterpret_cast<const uint4*>(mask + act_off(m, col, Nout, V));
        uint4 mk[2] = {__ldg(mp), __ldg(mp + V)};
        const bf16* mb = reinterpret_cast<const bf16*>(mk);
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (!(__bfloat162float(mb[j]) > 0.0f)) a[j] = 0.0f;
      }
      uint4 o[2];
      __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
      for (int j = 0; j < 8; j++) ob[j] = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
      uint4* op = reinterpret_cast<uint4*>(out_bf16 + act_off(m, col, Nout, V));
      op[0] = o[0];
      op[V] = o[1];  // the next 8-channel plane
      return;
    }
#pragma unroll
    for (int j = 0; j < 16; j++) {
      int n = col + j;
      if (n >= Nout) break;
      float a = v[j];
      if (bias) a += bias[n];
      if (relu) a = fmaxf(a, 0.0f);
      if (mask && !(__bfloat162float(mask[act_off(m, n, Nout, V)]) > 0.0f)) a = 0.0f;
      if (out_f32) out_f32[(size_t)m * Nout + n] = a;
      else out_bf16[act_off(m, n, Nout, V)] = __float2bfloat16(a);
    }
  }
};

}  // namespace
}  // namespace pyro
