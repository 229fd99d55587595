// The elementwise steps of a Conformer block, most of them around the convolution module's three convolutions (which stay the
// vendor library's), in the layouts these read and write:
//
//   bias_glu          (B, 2C, T) -> (B, C, T): bias, then a * sigmoid(g) of the channel halves;
//   bias_affine_silu  (B, C, T): bias, * scale, + shift (the folded batch norm), SiLU;
//   half_step         x + 0.5 * y, the product rounded (it is exact but for subnormals): a half-step feed-forward's residual;
//   bias_add_transposed   x (B, T, C) + (conv (B, C, T) + bias) -> (B, T, C): the residual, across the layouts.
//
// Bound, at 64 utterances of 250 steps and 1024 channels: half_step memory (98 MB in 15 us); the two around the convolutions
// instruction issue (74% of the slots, 27-29 us for 98 MB); bias_add_transposed the latency of its two-byte loads (51 us for 98 MB,
// DRAM 18% busy).  As steps of their own (a broadcast bias addition after every convolution among them, at 50 us for 33 MB) they
// took 10 of the 69 ms of 64 utterances' encoder.  Every step rounds to 16 bits where the sequence of modules rounds, with the
// same expressions, so that the results are its bits: behind 4-bit activations a last-place difference moves a code.
#include <algorithm>

#include "common.cuh"

namespace asrq {
namespace {

template <bool bf16>
__device__ __forceinline__ float r16(float v) { return out16_to_float(float_to_out16(v, bf16), bf16); }

// Eight consecutive elements of a (channels, T) plane per thread when VEC (plane and pointers aligned to them), else one.
// The channel of the first by one division, of the others by counting.
template <bool bf16, bool VEC, bool GLU>
__global__ void __launch_bounds__(256)
conv_elementwise_kernel(const uint16_t* __restrict__ in, const uint16_t* __restrict__ bias, const uint16_t* __restrict__ scale,
                        const uint16_t* __restrict__ shift, uint16_t* __restrict__ out, int C, int T) {
  constexpr int E = VEC ? 8 : 1;
  const unsigned plane = unsigned(C) * unsigned(T), i = (blockIdx.x * 256u + threadIdx.x) * E;
  if (i >= plane) return;
  const uint16_t* src = in + size_t(blockIdx.y) * plane * (GLU ? 2 : 1) + i;
  uint32_t a[4] = {0, 0, 0, 0}, g[4] = {0, 0, 0, 0}, o[4] = {0, 0, 0, 0};
  if (VEC) {
    const uint4 u = *reinterpret_cast<const uint4*>(src);
    a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w;
    if (GLU) {
      const uint4 w = *reinterpret_cast<const uint4*>(src + plane);
      g[0] = w.x, g[1] = w.y, g[2] = w.z, g[3] = w.w;
    }
  } else {
    a[0] = src[0];
    if (GLU) g[0] = src[plane];
  }
  unsigned c = i / unsigned(T), left = T - (i - c * unsigned(T));  // elements left of this channel
  auto value = [&](const uint16_t* p, unsigned k) { return out16_to_float(__ldg(p + k), bf16); };
  float b0 = value(bias, c), b1 = GLU ? value(bias, c + C) : value(scale, c), b2 = GLU ? 0.f : value(shift, c);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float v = out16_to_float(uint16_t(a[e >> 1] >> (16 * (e & 1))), bf16);
    float y;
    if (GLU) {
      const float gate = out16_to_float(uint16_t(g[e >> 1] >> (16 * (e & 1))), bf16);
      y = r16<bf16>(v + b0) * (1.f / (1.f + expf(-r16<bf16>(gate + b1))));
    } else {
      const float s = r16<bf16>(r16<bf16>(r16<bf16>(v + b0) * b1) + b2);
      y = s / (1.f + expf(-s));
    }
    o[e >> 1] |= uint32_t(float_to_out16(y, bf16)) << (16 * (e & 1));
    if (VEC && --left == 0 && e + 1 < E) {
      ++c;
      left = T;
      if (c < unsigned(C)) {
        b0 = value(bias, c);
        b1 = GLU ? value(bias, c + C) : value(scale, c);
        b2 = GLU ? 0.f : value(shift, c);
      }
    }
  }
  uint16_t* dst = out + size_t(blockIdx.y) * plane + i;
  if (VEC) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
    dst[0] = uint16_t(o[0]);
  }
}

template <bool bf16>
__global__ void __launch_bounds__(256)
half_step_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ y, uint16_t* __restrict__ out, size_t n) {
  const size_t i = (size_t(blockIdx.x) * 256 + threadIdx.x) * 8;
  if (i >= n) return;  // n is a multiple of 8
  const uint4 a = *reinterpret_cast<const uint4*>(x + i), b = *reinterpret_cast<const uint4*>(y + i);
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float lo = out16_to_float(uint16_t(aw[j] & 0xffffu), bf16) + r16<bf16>(0.5f * out16_to_float(uint16_t(bw[j] & 0xffffu), bf16));
    const float hi = out16_to_float(uint16_t(aw[j] >> 16), bf16) + r16<bf16>(0.5f * out16_to_float(uint16_t(bw[j] >> 16), bf16));
    o[j] = uint32_t(float_to_out16(lo, bf16)) | (uint32_t(float_to_out16(hi, bf16)) << 16);
  }
  *reinterpret_cast<uint4*>(out + i) = make_uint4(o[0], o[1], o[2], o[3]);
}

// 64 time steps x 64 channels through shared memory; rows of T are read two bytes a lane (T may be odd), rows of C written four.
template <bool bf16>
__global__ void __launch_bounds__(256)
bias_add_transposed_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ conv, const uint16_t* __restrict__ bias,
                           uint16_t* __restrict__ out, int C, int T) {
  __shared__ uint16_t tile[64][66];
  const int t0 = blockIdx.x * 64, c0 = blockIdx.y * 64, tid = threadIdx.x;
  const uint16_t* src = conv + (size_t(blockIdx.z) * C + c0) * T + t0;
  const int t = tid & 63;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int c = (tid >> 6) + 4 * k;
    if (c0 + c < C && t0 + t < T) tile[t][c] = src[size_t(c) * T + t];
  }
  __syncthreads();
  const int cp = (tid & 31) * 2;
  if (c0 + cp >= C) return;  // C is even
  const uint32_t bw = *reinterpret_cast<const uint32_t*>(bias + c0 + cp);
  const float b0 = out16_to_float(uint16_t(bw & 0xffffu), bf16), b1 = out16_to_float(uint16_t(bw >> 16), bf16);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int tt = (tid >> 5) + 8 * k;
    if (t0 + tt >= T) break;
    const size_t at = (size_t(blockIdx.z) * T + t0 + tt) * C + c0 + cp;
    const uint32_t xv = *reinterpret_cast<const uint32_t*>(x + at), v = *reinterpret_cast<const uint32_t*>(&tile[tt][cp]);
    const float y0 = out16_to_float(uint16_t(xv & 0xffffu), bf16) + r16<bf16>(out16_to_float(uint16_t(v & 0xffffu), bf16) + b0);
    const float y1 = out16_to_float(uint16_t(xv >> 16), bf16) + r16<bf16>(out16_to_float(uint16_t(v >> 16), bf16) + b1);
    *reinterpret_cast<uint32_t*>(out + at) = uint32_t(float_to_out16(y0, bf16)) | (uint32_t(float_to_out16(y1, bf16)) << 16);
  }
}

}  // namespace

// scale and shift NULL: bias and gate over 2 C channels, else bias, affine and SiLU over C
int conv_elementwise(const void* in, const void* bias, const void* scale, const void* shift, void* out, int64_t B, int64_t C, int64_t T, int dtype,
                     cudaStream_t stream) {
  const bool glu = scale == nullptr, vec = C * T % 8 == 0 && aligned16(in) && aligned16(out), bf16 = dtype == ASRQ_BF16;
  const dim3 grid(unsigned((C * T + (vec ? 2047 : 255)) / (vec ? 2048 : 256)), unsigned(B));
  auto q = [](const void* p) { return static_cast<const uint16_t*>(p); };
  auto run = [&](auto kern) {
    kern<<<grid, 256, 0, stream>>>(q(in), q(bias), q(scale), q(shift), static_cast<uint16_t*>(out), int(C), int(T));
    ASRQ_CUDA_TRY(cudaGetLastError());
    return int(ASRQ_OK);
  };
  if (bf16) {
    if (glu) return vec ? run(conv_elementwise_kernel<true, true, true>) : run(conv_elementwise_kernel<true, false, true>);
    return vec ? run(conv_elementwise_kernel<true, true, false>) : run(conv_elementwise_kernel<true, false, false>);
  }
  if (glu) return vec ? run(conv_elementwise_kernel<false, true, true>) : run(conv_elementwise_kernel<false, false, true>);
  return vec ? run(conv_elementwise_kernel<false, true, false>) : run(conv_elementwise_kernel<false, false, false>);
}

int half_step(const void* x, const void* y, void* out, int64_t n, int dtype, cudaStream_t stream) {
  auto kern = dtype == ASRQ_BF16 ? half_step_kernel<true> : half_step_kernel<false>;
  kern<<<unsigned((n / 8 + 255) / 256), 256, 0, stream>>>(static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(y), static_cast<uint16_t*>(out), size_t(n));
  ASRQ_CUDA_TRY(cudaGetLastError());
  return ASRQ_OK;
}

int bias_add_transposed(const void* x, const void* conv, const void* bias, void* out, int64_t B, int64_t T, int64_t C, int dtype, cudaStream_t stream) {
  const dim3 grid(unsigned((T + 63) / 64), unsigned((C + 63) / 64), unsigned(B));
  auto q = [](const void* p) { return static_cast<const uint16_t*>(p); };
  auto kern = dtype == ASRQ_BF16 ? bias_add_transposed_kernel<true> : bias_add_transposed_kernel<false>;
  kern<<<grid, 256, 0, stream>>>(q(x), q(conv), q(bias), static_cast<uint16_t*>(out), int(C), int(T));
  ASRQ_CUDA_TRY(cudaGetLastError());
  return ASRQ_OK;
}

}  // namespace asrq
