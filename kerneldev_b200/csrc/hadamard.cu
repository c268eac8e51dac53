// Incoherent-processing pre-pass: per-head sign flip and normalised Walsh-Hadamard transform
// over the head dimension. HBM-bound: reads and writes each element once; the butterflies run
// in registers (in-thread stages for the low index bits, warp shuffles for the high ones).
#include <algorithm>

#include "common.cuh"
#include "sm100_prims.cuh"

namespace kd {

// Unnormalised transform of rows of 8 CH TPR elements, in place. Element index = 8 * (sub + TPR * i) + k of v[i][k]: the bits of k and of i are
// butterflied in registers, the bits of `sub` with warp shuffles (all lanes call it).
template <int CH, int TPR>
__device__ __forceinline__ void walsh_hadamard(float (&v)[CH][8], int sub) {
  // inside a chunk
#pragma unroll
  for (int i = 0; i < CH; ++i) {
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if ((k & s) == 0) {
          const float a0 = v[i][k], a1 = v[i][k | s];
          v[i][k] = a0 + a1;
          v[i][k | s] = a0 - a1;
        }
      }
    }
  }
  // across the threads of the row
#pragma unroll
  for (int s = 1; s < TPR; s <<= 1) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float other = __shfl_xor_sync(0xffffffffu, v[i][k], s);
        v[i][k] = (sub & s) ? (other - v[i][k]) : (v[i][k] + other);
      }
    }
  }
  // between this thread's chunks
#pragma unroll
  for (int s = 1; s < CH; s <<= 1) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      if ((i & s) == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float a0 = v[i][k], a1 = v[i | s][k];
          v[i][k] = a0 + a1;
          v[i | s][k] = a0 - a1;
        }
      }
    }
  }
}

// TPR = min(4, HD/8) threads share a token row; thread `sub` holds the 16-byte chunks sub, sub + TPR, ... of the
// row (CH = HD/8/TPR chunks of 8 elements), so that a warp-wide load covers 64 contiguous bytes per row.
// Element index = 8 * (sub + TPR * i) + k: index bits 0-2 (k) and the bits of i are butterflied in registers,
// the bits of `sub` with warp shuffles (two stages at most). Rows are walked with a grid-stride loop; bound by
// HBM bandwidth (2 * rows * HD * 2 bytes per call).
template <int HD, bool kBf16>
__global__ void __launch_bounds__(256) hadamard_kernel(const uint16_t* x, int64_t x_sb, int64_t x_sh, int64_t x_st,
                                                       uint16_t* y, int64_t y_sb, int64_t y_sh, int64_t y_st,
                                                       int B, int H, int T, const float* signs, int inverse) {
  constexpr int TPR = (HD / 8 < 4) ? HD / 8 : 4;   // threads per row
  constexpr int CH = HD / 8 / TPR;                 // chunks per thread
  constexpr int RPB = 256 / TPR;                   // rows per block and iteration
  const int sub = threadIdx.x % TPR;
  const long long rows = (long long)B * H * T;
  const float norm = rsqrtf(static_cast<float>(HD));
  pdl_wait();
  pdl_launch_dependents();
  // the loop bound is the same for every thread of a warp: the shuffles below need all lanes
  for (long long base = (long long)blockIdx.x * RPB; base < rows; base += (long long)gridDim.x * RPB) {
    const long long row = base + threadIdx.x / TPR;
    const bool live = row < rows;
    const long long rr = live ? row : rows - 1;
    const int t = static_cast<int>(rr % T);
    const int h = static_cast<int>((rr / T) % H);
    const int b = static_cast<int>(rr / ((long long)T * H));
    const uint16_t* src = x + (size_t)b * x_sb + (size_t)h * x_sh + (size_t)t * x_st;
    uint16_t* dst = y + (size_t)b * y_sb + (size_t)h * y_sh + (size_t)t * y_st;
    const float* sg = signs ? signs + h * HD : nullptr;
    uint4 in[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) in[i] = *reinterpret_cast<const uint4*>(src + (sub + TPR * i) * 8);
    float v[CH][8];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const uint32_t w[4] = {in[i].x, in[i].y, in[i].z, in[i].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack2<kBf16>(w[k]);
        v[i][2 * k] = f.x; v[i][2 * k + 1] = f.y;
      }
      if (sg != nullptr && !inverse) {
        const float4 s0 = *reinterpret_cast<const float4*>(sg + (sub + TPR * i) * 8);
        const float4 s1 = *reinterpret_cast<const float4*>(sg + (sub + TPR * i) * 8 + 4);
        v[i][0] *= s0.x; v[i][1] *= s0.y; v[i][2] *= s0.z; v[i][3] *= s0.w;
        v[i][4] *= s1.x; v[i][5] *= s1.y; v[i][6] *= s1.z; v[i][7] *= s1.w;
      }
    }
    walsh_hadamard<CH, TPR>(v, sub);
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float f[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] = v[i][k] * norm;
      if (sg != nullptr && inverse) {
        const float4 s0 = *reinterpret_cast<const float4*>(sg + (sub + TPR * i) * 8);
        const float4 s1 = *reinterpret_cast<const float4*>(sg + (sub + TPR * i) * 8 + 4);
        f[0] *= s0.x; f[1] *= s0.y; f[2] *= s0.z; f[3] *= s0.w; f[4] *= s1.x; f[5] *= s1.y; f[6] *= s1.z; f[7] *= s1.w;
      }
      if (live) {
        uint4 out;
        out.x = pack2<kBf16>(f[0], f[1]);
        out.y = pack2<kBf16>(f[2], f[3]);
        out.z = pack2<kBf16>(f[4], f[5]);
        out.w = pack2<kBf16>(f[6], f[7]);
        *reinterpret_cast<uint4*>(dst + (sub + TPR * i) * 8) = out;
      }
    }
  }
}

// The last pass of a fused backward on transformed Q and K: dQ from the fp32 scratch, scaled, and dK, both times the transform's transpose. One
// launch in the place of the conversion to 16 bits and two transforms (fp16 4 x 32 x 8192 x 128 with a fifth of padding 172 + 2 x 128 us -> 307, bf16
// 8 x 16 x 2048 x 64 18 + 2 x 20 -> 32), which write and read dQ once more, and dQ is rounded once. Rows of padding: dQ is 0 and its scratch not
// read; dK is 0 already. By the bytes it would take 175 us (hadamard_kernel: 82 of 128): the pipe that loads, stores and shuffles share is busy for 81 % of the
// cycles (73 %), issue slots for 61 % (74 %). Pieces of 4 floats, so that a load takes whole sectors: 317; five or six blocks to an SM 325 and 394 (registers).
// blockIdx.x: 2 * (block of rows) + (0: dQ, 1: dK).
struct GradTransformArgs {
  const float* acc;
  const int32_t* len;
  const float* signs;
  kd_tensor dq, dk;
  int H, T, width;   // width: of the scratch's rows
  float scale;
};
template <int HD, bool kBf16>
__global__ void __launch_bounds__(256) grad_transform_kernel(const GradTransformArgs a) {
  constexpr int TPR = (HD / 8 < 4) ? HD / 8 : 4, CH = HD / 8 / TPR, RPB = 256 / TPR;
  const int sub = threadIdx.x % TPR, b = blockIdx.z, h = blockIdx.y, t = static_cast<int>(blockIdx.x >> 1) * RPB + threadIdx.x / TPR;
  const bool is_k = (blockIdx.x & 1) != 0;
  const int len = __ldcg(a.len + b);   // (the plan was complete before the fused kernel let this one start)
  pdl_wait();
  pdl_launch_dependents();
  const kd_tensor& out = is_k ? a.dk : a.dq;
  uint16_t* row = static_cast<uint16_t*>(out.ptr) + (size_t)b * out.stride_b + (size_t)h * out.stride_h + (size_t)t * out.stride_t;
  float v[CH][8];
#pragma unroll
  for (int i = 0; i < CH; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k) v[i][k] = 0.f;
  const float norm = rsqrtf(static_cast<float>(HD)) * (is_k ? 1.0f : a.scale);
  if (t < len) {
    if (is_k) {
      uint4 in[CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) in[i] = *reinterpret_cast<const uint4*>(row + (sub + TPR * i) * 8);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const uint32_t w[4] = {in[i].x, in[i].y, in[i].z, in[i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = unpack2<kBf16>(w[k]);
          v[i][2 * k] = f.x; v[i][2 * k + 1] = f.y;
        }
      }
    } else {
      const float* src = a.acc + (((size_t)b * a.H + h) * a.T + t) * a.width;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(src + (sub + TPR * i) * 8), y = *reinterpret_cast<const float4*>(src + (sub + TPR * i) * 8 + 4);
        v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
        v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
      }
    }
  }
  walsh_hadamard<CH, TPR>(v, sub);
  if (t >= (is_k ? len : a.T)) return;
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const float* sg = a.signs + h * HD + (sub + TPR * i) * 8;
    const float4 s0 = *reinterpret_cast<const float4*>(sg), s1 = *reinterpret_cast<const float4*>(sg + 4);
    uint4 w;
    w.x = pack2<kBf16>(v[i][0] * norm * s0.x, v[i][1] * norm * s0.y);
    w.y = pack2<kBf16>(v[i][2] * norm * s0.z, v[i][3] * norm * s0.w);
    w.z = pack2<kBf16>(v[i][4] * norm * s1.x, v[i][5] * norm * s1.y);
    w.w = pack2<kBf16>(v[i][6] * norm * s1.z, v[i][7] * norm * s1.w);
    *reinterpret_cast<uint4*>(row + (sub + TPR * i) * 8) = w;
  }
}

int launch_grad_transform(const float* acc, int width, float scale, const int32_t* len, const float* signs, const kd_tensor& dq, const kd_tensor& dk,
                          int B, int H, int T, int D, int dtype, cudaStream_t stream) {
  const GradTransformArgs a = {acc, len, signs, dq, dk, H, T, width, scale};
  const int rows_per_block = 256 / (D / 8 < 4 ? D / 8 : 4);
  const dim3 grid(2 * ((T + rows_per_block - 1) / rows_per_block), H, B);
  auto run = [&](auto kernel) { return launch(kernel, grid, 256, 0, stream, a); };
  const bool bf16 = dtype == KD_BF16;
  cudaError_t e;
  if (D == 16) e = bf16 ? run(grad_transform_kernel<16, true>) : run(grad_transform_kernel<16, false>);
  else if (D == 32) e = bf16 ? run(grad_transform_kernel<32, true>) : run(grad_transform_kernel<32, false>);
  else if (D == 64) e = bf16 ? run(grad_transform_kernel<64, true>) : run(grad_transform_kernel<64, false>);
  else e = bf16 ? run(grad_transform_kernel<128, true>) : run(grad_transform_kernel<128, false>);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "grad_transform_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

int launch_hadamard(const kd_tensor& x, const kd_tensor& y, int B, int H, int T, int D, int dtype,
                    const float* signs, int inverse, cudaStream_t stream) {
  const long long rows = (long long)B * H * T;
  const int rows_per_block = 256 / (D / 8 < 4 ? D / 8 : 4);
  const unsigned blocks = static_cast<unsigned>(std::min<long long>((rows + rows_per_block - 1) / rows_per_block, 148LL * 32));
  const uint16_t* xp = static_cast<const uint16_t*>(x.ptr);
  uint16_t* yp = static_cast<uint16_t*>(y.ptr);
  cudaError_t e;
#define KD_LAUNCH_H(HD, BF)                                                                             \
  e = launch(hadamard_kernel<HD, BF>, blocks, 256, 0, stream, xp, x.stride_b, x.stride_h, x.stride_t, yp, y.stride_b,           \
             y.stride_h, y.stride_t, B, H, T, signs, inverse)
  if (D == 16 && dtype == KD_BF16) KD_LAUNCH_H(16, true);
  else if (D == 16) KD_LAUNCH_H(16, false);
  else if (D == 32 && dtype == KD_BF16) KD_LAUNCH_H(32, true);
  else if (D == 32) KD_LAUNCH_H(32, false);
  else if (D == 64 && dtype == KD_BF16) KD_LAUNCH_H(64, true);
  else if (D == 64) KD_LAUNCH_H(64, false);
  else if (D == 128 && dtype == KD_BF16) KD_LAUNCH_H(128, true);
  else KD_LAUNCH_H(128, false);
#undef KD_LAUNCH_H
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "hadamard_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace kd
