// What stands between the layers of a Conformer block, channels last:
//
//   residual_norms   s = x + scale * delta (optional), y = LayerNorm(s); with a second norm also z = LayerNorm(y): the end of
//                    one block and the start of the next.  One warp per row, held in registers;
//   glu_dwconv       the convolution module between its two pointwise projections: a * sigmoid(g) of the first one's halves,
//                    depthwise convolution over time, scale and shift per channel (the folded batch norm), SiLU.
//
// Both are bound by memory (the conv by latency for a few hundred rows).  As separate torch steps in (batch, channel, time)
// order the module took two transposing copies, a gated pass, the convolution and three elementwise passes around it.
// 16-bit in and out, fp32 arithmetic, rounded to 16 bits where the sequence of modules rounds.
#include "common.cuh"

namespace asrq {
namespace {

constexpr int kRowWarps = 4;

__device__ __forceinline__ void words(const uint4& u, uint32_t (&w)[4]) {
  w[0] = u.x;
  w[1] = u.y;
  w[2] = u.z;
  w[3] = u.w;
}
__device__ __forceinline__ float lo16(uint32_t w, bool bf16) { return out16_to_float(uint16_t(w & 0xffffu), bf16); }
__device__ __forceinline__ float hi16(uint32_t w, bool bf16) { return out16_to_float(uint16_t(w >> 16), bf16); }
__device__ __forceinline__ uint32_t pack16(float lo, float hi, bool bf16) {
  return uint32_t(float_to_out16(lo, bf16)) | (uint32_t(float_to_out16(hi, bf16)) << 16);
}

template <int VEC>
__device__ __forceinline__ void norm_row(uint4 (&row)[VEC], const uint16_t* __restrict__ gamma, const uint16_t* __restrict__ beta, float eps, bool bf16, int lane) {
  float mean, rstd;
  ln_row_stats<VEC>(row, 256 * VEC, eps, bf16, mean, rstd);
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const int e = (i * 32 + lane) * 8;
    uint32_t v[4], g[4], b[4];
    words(row[i], v);
    words(__ldg(reinterpret_cast<const uint4*>(gamma + e)), g);
    words(__ldg(reinterpret_cast<const uint4*>(beta + e)), b);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = pack16(ln_apply(lo16(v[j], bf16), mean, rstd, lo16(g[j], bf16), lo16(b[j], bf16)),
                    ln_apply(hi16(v[j], bf16), mean, rstd, hi16(g[j], bf16), hi16(b[j], bf16)), bf16);
    row[i] = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

struct NormsParams {
  const uint16_t *x, *delta, *g1, *b1, *g2, *b2;
  uint16_t *x_out, *h_out;  // x_out: the residual stream that goes on (s, or y when there is a second norm); may be NULL
  float scale, eps1, eps2;
  int rows;
};

template <int VEC, bool bf16>
__global__ void __launch_bounds__(32 * kRowWarps)
residual_norms_kernel(const NormsParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31, r = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (r >= p.rows) return;
  const size_t off = size_t(r) * (256 * VEC) + lane * 8;
  uint4 row[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) row[i] = *reinterpret_cast<const uint4*>(p.x + off + i * 256);
  if (p.delta) {
    uint4 d[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) d[i] = *reinterpret_cast<const uint4*>(p.delta + off + i * 256);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      uint32_t a[4], b[4];
      words(row[i], a);
      words(d[i], b);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = out16_to_float(float_to_out16(p.scale * lo16(b[j], bf16), bf16), bf16);
        const float hi = out16_to_float(float_to_out16(p.scale * hi16(b[j], bf16), bf16), bf16);
        a[j] = pack16(lo16(a[j], bf16) + lo, hi16(a[j], bf16) + hi, bf16);
      }
      row[i] = make_uint4(a[0], a[1], a[2], a[3]);
    }
  }
  if (p.g2) norm_row<VEC>(row, p.g1, p.b1, p.eps1, bf16, lane);
  if (p.x_out) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) *reinterpret_cast<uint4*>(p.x_out + off + i * 256) = row[i];
  }
  if (!p.h_out) return;
  norm_row<VEC>(row, p.g2 ? p.g2 : p.g1, p.g2 ? p.b2 : p.b1, p.g2 ? p.eps2 : p.eps1, bf16, lane);
#pragma unroll
  for (int i = 0; i < VEC; ++i) *reinterpret_cast<uint4*>(p.h_out + off + i * 256) = row[i];
}

// A thread takes two channels (a warp 128 contiguous bytes of a row) and TL positions: all TL + KW - 1 gated inputs go into
// registers first, so every load of the thread is in flight at once and the taps are fully unrolled.  TL = 16: the halo costs
// half as many loads again (from L2); longer runs leave a single sequence with too few threads.
template <int KW, int TL, bool bf16>
__global__ void __launch_bounds__(128)
glu_dwconv_kernel(const uint16_t* __restrict__ in, const uint16_t* __restrict__ w, const uint16_t* __restrict__ bias, const uint16_t* __restrict__ scale,
                  const uint16_t* __restrict__ shift, uint16_t* __restrict__ out, int T, int d) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int c = (blockIdx.x * 128 + threadIdx.x) * 2, t0 = blockIdx.y * TL;
  const bool on = c < d;
  float wt[2][KW], bs[2], sc[2], sh[2];
  if (on) {
    auto two = [&](const uint16_t* q) { return __ldg(reinterpret_cast<const unsigned int*>(q)); };
#pragma unroll
    for (int i = 0; i < KW; ++i) {  // 2 KW consecutive taps
      const uint32_t v = two(w + size_t(c) * KW + 2 * i);
      wt[(2 * i) / KW][(2 * i) % KW] = lo16(v, bf16);
      wt[(2 * i + 1) / KW][(2 * i + 1) % KW] = hi16(v, bf16);
    }
    const uint32_t vb = two(bias + c), vs = two(scale + c), vh = two(shift + c);
    bs[0] = lo16(vb, bf16), bs[1] = hi16(vb, bf16);
    sc[0] = lo16(vs, bf16), sc[1] = hi16(vs, bf16);
    sh[0] = lo16(vh, bf16), sh[1] = hi16(vh, bf16);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!on) return;
  const uint16_t* base = in + size_t(blockIdx.z) * T * 2 * d + c;
  uint32_t a[TL + KW - 1], g[TL + KW - 1];
#pragma unroll
  for (int i = 0; i < TL + KW - 1; ++i) {
    const int t = t0 + i - KW / 2;
    const bool in_range = t >= 0 && t < T;
    a[i] = in_range ? __ldg(reinterpret_cast<const unsigned int*>(base + size_t(t) * 2 * d)) : 0u;
    g[i] = in_range ? __ldg(reinterpret_cast<const unsigned int*>(base + size_t(t) * 2 * d + d)) : 0u;
  }
  auto r16 = [&](float v) { return out16_to_float(float_to_out16(v, bf16), bf16); };
  // a few fp32 ulps (exponential and quotient) under a rounding to 16 bits; a denominator past 2^126 gives 0, its limit
  auto sigmoid_of = [](float v, float g) { return __fdividef(v, 1.f + __expf(-g)); };
  float u[2][TL + KW - 1];
#pragma unroll
  for (int i = 0; i < TL + KW - 1; ++i) {  // outside the sequence a = 0: the padding of the convolution
    u[0][i] = r16(sigmoid_of(lo16(a[i], bf16), lo16(g[i], bf16)));
    u[1][i] = r16(sigmoid_of(hi16(a[i], bf16), hi16(g[i], bf16)));
  }
  uint16_t* o = out + (size_t(blockIdx.z) * T + t0) * d + c;
#pragma unroll
  for (int t = 0; t < TL; ++t) {
    if (t0 + t >= T) break;
    float y[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < KW; ++i) acc = fmaf(u[k][t + i], wt[k][i], acc);
      const float v = r16(r16(r16(acc + bs[k]) * sc[k]) + sh[k]);
      y[k] = sigmoid_of(v, v);
    }
    *reinterpret_cast<unsigned int*>(o + size_t(t) * d) = pack16(y[0], y[1], bf16);
  }
}

template <typename K, typename... Args>
int launch(K kern, dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
  return ASRQ_OK;
}

}  // namespace

int residual_norms(const void* x, const void* delta, float scale, const void* g1, const void* b1, float eps1, const void* g2, const void* b2, float eps2,
                   void* x_out, void* h_out, int64_t rows, int64_t dim, int dtype, cudaStream_t stream) {
  auto in = [](const void* q) { return static_cast<const uint16_t*>(q); };
  const NormsParams p = {in(x), in(delta), in(g1), in(b1), in(g2), in(b2), static_cast<uint16_t*>(x_out), static_cast<uint16_t*>(h_out),
                         scale, eps1, eps2, int(rows)};
  const dim3 grid(unsigned((rows + kRowWarps - 1) / kRowWarps)), block(32 * kRowWarps);
  const bool bf16 = dtype == ASRQ_BF16;
  switch (dim / 256) {
#define ASRQ_NORMS(V) \
  case V: return bf16 ? launch(residual_norms_kernel<V, true>, grid, block, stream, p) : launch(residual_norms_kernel<V, false>, grid, block, stream, p)
    ASRQ_NORMS(1);
    ASRQ_NORMS(2);
    ASRQ_NORMS(3);
    ASRQ_NORMS(4);
    ASRQ_NORMS(5);
    ASRQ_NORMS(6);
    ASRQ_NORMS(7);
    ASRQ_NORMS(8);
#undef ASRQ_NORMS
    default: return fail(ASRQ_ERR_SHAPE, "residual_norms: dim=%lld", (long long)dim);
  }
}

int glu_dwconv(const void* in, const void* w, const void* bias, const void* scale, const void* shift, void* out, int64_t B, int64_t T, int64_t d,
               int dtype, cudaStream_t stream) {
  constexpr int TL = 16;
  auto q = [](const void* v) { return static_cast<const uint16_t*>(v); };
  const dim3 grid(unsigned((d / 2 + 127) / 128), unsigned((T + TL - 1) / TL), unsigned(B));
  return launch(dtype == ASRQ_BF16 ? glu_dwconv_kernel<9, TL, true> : glu_dwconv_kernel<9, TL, false>, grid, dim3(128), stream, q(in), q(w), q(bias), q(scale),
                q(shift), static_cast<uint16_t*>(out), int(T), int(d));
}

}  // namespace asrq
