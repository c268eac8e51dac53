// Conversion between float32 tensors and the 16-bit operands of the kernels: all tensors of a call in one launch.
// float32 Q, K, V take part as float16 operands (the mantissa of tf32). O, dO and the gradients need no pass of their own (kd_attn_f32),
// but with incoherent processing, whose transform of dQ and dK works on 16-bit tensors, dO and the gradients come here as well.
// Bound by HBM traffic (6 bytes per element), for small calls by launches.
#include <algorithm>

#include "common.cuh"
#include "sm100_prims.cuh"

namespace kd {

struct CastArgs {
  kd_tensor src[KD_CAST_MAX], dst[KD_CAST_MAX];
  int B, H, T, D8;   // D8: groups of 8 elements in a row
};

// eight elements per thread and step; blockIdx.y = tensor
template <bool kWiden>
__global__ void __launch_bounds__(256) cast_kernel(const __grid_constant__ CastArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const kd_tensor src = a.src[blockIdx.y], dst = a.dst[blockIdx.y];
  const size_t n = (size_t)a.B * a.H * a.T * a.D8;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    const size_t r = i / a.D8, bh = r / a.T;
    const int c = static_cast<int>(i - r * a.D8) * 8, t = static_cast<int>(r - bh * a.T);
    const int b = static_cast<int>(bh / a.H), h = static_cast<int>(bh - (size_t)b * a.H);
    const size_t from = (size_t)b * src.stride_b + (size_t)h * src.stride_h + (size_t)t * src.stride_t + c;
    const size_t to = (size_t)b * dst.stride_b + (size_t)h * dst.stride_h + (size_t)t * dst.stride_t + c;
    if constexpr (kWiden) {
      const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(src.ptr) + from);
      const float2 x0 = unpack2<false>(v.x), x1 = unpack2<false>(v.y), x2 = unpack2<false>(v.z), x3 = unpack2<false>(v.w);
      float4* out = reinterpret_cast<float4*>(static_cast<float*>(dst.ptr) + to);
      out[0] = make_float4(x0.x, x0.y, x1.x, x1.y);
      out[1] = make_float4(x2.x, x2.y, x3.x, x3.y);
    } else {
      const float4* in = reinterpret_cast<const float4*>(static_cast<const float*>(src.ptr) + from);
      const float4 x = in[0], y = in[1];
      uint4 v;
      v.x = pack2<false>(x.x, x.y);
      v.y = pack2<false>(x.z, x.w);
      v.z = pack2<false>(y.x, y.y);
      v.w = pack2<false>(y.z, y.w);
      *reinterpret_cast<uint4*>(static_cast<uint16_t*>(dst.ptr) + to) = v;
    }
  }
}

int launch_cast(const kd_tensor* src, const kd_tensor* dst, int n, int B, int H, int T, int D, bool widen, cudaStream_t stream) {
  CastArgs a;
  for (int i = 0; i < n; ++i) {
    a.src[i] = src[i];
    a.dst[i] = dst[i];
  }
  a.B = B; a.H = H; a.T = T; a.D8 = D / 8;
  const size_t steps = (size_t)B * H * T * a.D8;
  const unsigned blocks = static_cast<unsigned>(std::min<size_t>((steps + 255) / 256, size_t(148) * 16));
  const cudaError_t e = launch(widen ? cast_kernel<true> : cast_kernel<false>, dim3(blocks, n), 256, 0, stream, a);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "cast_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace kd
