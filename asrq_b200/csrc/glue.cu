// The steps either side of a quantized layer in a decoder block, as kernels of their own:
//
//   add_layernorm   x' = x + delta (optional), h = LayerNorm(x') * gamma + beta, one warp per row (a block per
//                   row up to 296 rows, as for the RMS norm), fp32 statistics on the 16-bit-rounded x' (what
//                   the unfused sequence "add, then layer_norm" computes), 16-bit in and out;
//   add_rmsnorm     x' = x + delta (optional), h = (x' / rms(x')) rounded to 16 bits, then * gamma: the RMS norm of
//                   the Qwen3 decoder blocks (statistics in fp32, the normalised value rounded before the weight
//                   multiplies it, as the module does);
//   silu_mul        out[m, i] = silu(gu[m, i]) * gu[m, I + i] on the output of a fused gate/up projection, each
//                   factor rounded to 16 bits as the unfused sequence rounds them;
//   qk_norm_rope    what sits between a fused q/k/v projection and the attention of a Qwen3 block, in one launch: the
//                   per-head RMS norm of queries and keys, the rotary embedding, and the write of the new keys and
//                   values into the caches at the sequence position (read from device memory when decoding under a
//                   graph), every step rounded to 16 bits where the module sequence rounds it;
//   epilogue16      y = act(y) or y = residual + y on an already written output: the fall-back for
//                   layers whose kernel does not fuse the epilogue.
//
// All open with griddepcontrol.launch_dependents / .wait and are launched with programmatic stream
// serialisation, so in a chain of this library's kernels (a decoder step replayed as a CUDA graph)
// consecutive launches overlap their ramp-up with the predecessor's tail.  Behind the wait, what is not
// a constant is read by ld_x4 and ld_x1 or through behind_wait (common.cuh).
#include <algorithm>

#include "common.cuh"

namespace asrq {

namespace {

__device__ __forceinline__ float in16(uint16_t b, bool bf16) {
  return bf16 ? bf16_bits_to_float(b) : __half2float(__ushort_as_half(b));
}

constexpr int kLnWarps = 8;

// use(e, x[e] (+ delta[e], rounded)) for a lane's elements of a row of any width, in order, eight loads of each in flight
template <bool bf16, bool DELTA, typename F>
__device__ __forceinline__ void each_of_row(const uint16_t* x, const uint16_t* delta, int dim, int lane, F use) {
  constexpr int kBatch = 8;
  uint16_t a[kBatch], d[kBatch];
  auto value = [&](int k) { return float_to_out16(DELTA ? in16(a[k], bf16) + in16(d[k], bf16) : in16(a[k], bf16), bf16); };
  int e0 = lane;
  for (; e0 + 32 * (kBatch - 1) < dim; e0 += 32 * kBatch) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) a[k] = ld_x1(x + e0 + 32 * k);
    if (DELTA) {
#pragma unroll
      for (int k = 0; k < kBatch; ++k) d[k] = ld_x1(delta + e0 + 32 * k);
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) use(e0 + 32 * k, value(k));
  }
  // the rest: fewer than a batch
#pragma unroll
  for (int k = 0; k < kBatch - 1; ++k) {
    if (e0 + 32 * k < dim) {
      a[k] = ld_x1(x + e0 + 32 * k);
      if (DELTA) d[k] = ld_x1(delta + e0 + 32 * k);
    }
  }
#pragma unroll
  for (int k = 0; k < kBatch - 1; ++k)
    if (e0 + 32 * k < dim) use(e0 + 32 * k, value(k));
}
template <bool bf16, typename F>
__device__ __forceinline__ void each_of_row(const uint16_t* x, const uint16_t* delta, int dim, int lane, F use) {
  if (delta) each_of_row<bf16, true>(x, delta, dim, lane, use);
  else each_of_row<bf16, false>(x, delta, dim, lane, use);
}

// VEC: 16-byte vectors per lane (dim = 256 * VEC); generic dims take the strided loop with VEC = 0
template <int VEC, bool bf16>
__global__ void __launch_bounds__(32 * kLnWarps)
add_layernorm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ delta, const uint16_t* __restrict__ gamma,
                     const uint16_t* __restrict__ beta, float eps, uint16_t* __restrict__ x_out, uint16_t* __restrict__ h_out,
                     int rows, int dim) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kLnWarps + (threadIdx.x >> 5);
  // the norm's weight and bias are constants: fetched ahead of the stream dependency (vector path)
  uint4 gpre[VEC > 0 ? VEC : 1], bpre[VEC > 0 ? VEC : 1];
  if constexpr (VEC > 0) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int e = (i * 32 + lane) * 8;
      gpre[i] = __ldg(reinterpret_cast<const uint4*>(gamma + e));
      bpre[i] = __ldg(reinterpret_cast<const uint4*>(beta + e));
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (row >= rows) return;
  const size_t off = size_t(row) * dim;
  if constexpr (VEC > 0) {
    uint4 xr[VEC > 0 ? VEC : 1];  // the row (after the add, rounded to 16 bits), as the statistics see it
#pragma unroll
    for (int i = 0; i < VEC; ++i) xr[i] = ld_x4(x + off + (i * 32 + lane) * 8);
    if (delta) {
      uint4 d8[VEC > 0 ? VEC : 1];
#pragma unroll
      for (int i = 0; i < VEC; ++i) d8[i] = ld_x4(delta + off + (i * 32 + lane) * 8);
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const uint32_t aw[4] = {xr[i].x, xr[i].y, xr[i].z, xr[i].w}, dw[4] = {d8[i].x, d8[i].y, d8[i].z, d8[i].w};
        uint32_t ow[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = in16(uint16_t(aw[j] & 0xffffu), bf16) + in16(uint16_t(dw[j] & 0xffffu), bf16);
          const float hi = in16(uint16_t(aw[j] >> 16), bf16) + in16(uint16_t(dw[j] >> 16), bf16);
          ow[j] = uint32_t(float_to_out16(lo, bf16)) | (uint32_t(float_to_out16(hi, bf16)) << 16);
        }
        xr[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
    if (x_out) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) *reinterpret_cast<uint4*>(x_out + off + (i * 32 + lane) * 8) = xr[i];
    }
    float mean, rstd;
    ln_row_stats<(VEC > 0 ? VEC : 1)>(xr, dim, eps, bf16, mean, rstd);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int e = (i * 32 + lane) * 8;
      const uint4 g = gpre[i], b = bpre[i];
      const uint32_t xw[4] = {xr[i].x, xr[i].y, xr[i].z, xr[i].w};
      const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, bw[4] = {b.x, b.y, b.z, b.w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = ln_apply(in16(uint16_t(xw[j] & 0xffffu), bf16), mean, rstd, in16(uint16_t(gw[j] & 0xffffu), bf16),
                                  in16(uint16_t(bw[j] & 0xffffu), bf16));
        const float hi = ln_apply(in16(uint16_t(xw[j] >> 16), bf16), mean, rstd, in16(uint16_t(gw[j] >> 16), bf16),
                                  in16(uint16_t(bw[j] >> 16), bf16));
        ow[j] = uint32_t(float_to_out16(lo, bf16)) | (uint32_t(float_to_out16(hi, bf16)) << 16);
      }
      *reinterpret_cast<uint4*>(h_out + off + e) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
  } else {
    // any dimension: three passes over the row (the second and third hit L1/L2)
    float sum = 0.f;
    each_of_row<bf16>(x + off, delta ? delta + off : nullptr, dim, lane, [&](int e, uint16_t a16) {
      if (x_out) x_out[off + e] = a16;
      sum += in16(a16, bf16);
    });
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / float(dim);
    float sq = 0.f;
    each_of_row<bf16>(x + off, delta ? delta + off : nullptr, dim, lane, [&](int, uint16_t a16) {
      const float d = in16(a16, bf16) - mean;
      sq = fmaf(d, d, sq);
    });
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq / float(dim) + eps);
    each_of_row<bf16>(x + off, delta ? delta + off : nullptr, dim, lane, [&](int e, uint16_t a16) {
      h_out[off + e] = float_to_out16((in16(a16, bf16) - mean) * rstd * in16(gamma[e], bf16) + in16(beta[e], bf16), bf16);
    });
  }
}

// One warp per row; VEC 16-byte vectors per lane when dim == 256 * VEC, else (VEC = 0) a strided loop.  All of a row's loads go
// out before the first is used.
template <int VEC, bool bf16>
__global__ void __launch_bounds__(32 * kLnWarps, 2)
add_rmsnorm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ delta, const uint16_t* __restrict__ gamma,
                   float eps, uint16_t* __restrict__ x_out, uint16_t* __restrict__ h_out, int rows, int dim) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31;
  uint4 gpre[VEC > 0 ? VEC : 1];  // the weight is a constant: fetched ahead of the stream dependency
  if constexpr (VEC > 0) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) gpre[i] = __ldg(reinterpret_cast<const uint4*>(gamma + (i * 32 + lane) * 8));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int row = blockIdx.x * kLnWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  const size_t off = size_t(row) * dim;
  if constexpr (VEC > 0) {
    float v[VEC > 0 ? VEC * 8 : 1];
    float sq = 0.f;
    uint4 a8[VEC > 0 ? VEC : 1], d8[VEC > 0 ? VEC : 1];
#pragma unroll
    for (int i = 0; i < VEC; ++i) a8[i] = ld_x4(x + off + (i * 32 + lane) * 8);
    if (delta) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) d8[i] = ld_x4(delta + off + (i * 32 + lane) * 8);
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int e = (i * 32 + lane) * 8;
      const uint32_t aw[4] = {a8[i].x, a8[i].y, a8[i].z, a8[i].w}, dw[4] = {d8[i].x, d8[i].y, d8[i].z, d8[i].w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float lo = in16(uint16_t(aw[j] & 0xffffu), bf16), hi = in16(uint16_t(aw[j] >> 16), bf16);
        if (delta) {
          lo += in16(uint16_t(dw[j] & 0xffffu), bf16);
          hi += in16(uint16_t(dw[j] >> 16), bf16);
        }
        const uint16_t lo16 = float_to_out16(lo, bf16), hi16 = float_to_out16(hi, bf16);
        ow[j] = uint32_t(lo16) | (uint32_t(hi16) << 16);
        const float l = in16(lo16, bf16), h = in16(hi16, bf16);
        v[i * 8 + 2 * j] = l;
        v[i * 8 + 2 * j + 1] = h;
        sq = fmaf(l, l, sq);
        sq = fmaf(h, h, sq);
      }
      if (x_out) *reinterpret_cast<uint4*>(x_out + off + e) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rs = rsqrtf(sq / float(dim) + eps);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int e = (i * 32 + lane) * 8;
      const uint4 g = gpre[i];
      const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = in16(float_to_out16(v[i * 8 + 2 * j] * rs, bf16), bf16) * in16(uint16_t(gw[j] & 0xffffu), bf16);
        const float hi = in16(float_to_out16(v[i * 8 + 2 * j + 1] * rs, bf16), bf16) * in16(uint16_t(gw[j] >> 16), bf16);
        ow[j] = uint32_t(float_to_out16(lo, bf16)) | (uint32_t(float_to_out16(hi, bf16)) << 16);
      }
      *reinterpret_cast<uint4*>(h_out + off + e) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
  } else {
    float sq = 0.f;
    each_of_row<bf16>(x + off, delta ? delta + off : nullptr, dim, lane, [&](int e, uint16_t a16) {
      if (x_out) x_out[off + e] = a16;
      const float c = in16(a16, bf16);
      sq = fmaf(c, c, sq);
    });
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rs = rsqrtf(sq / float(dim) + eps);
    each_of_row<bf16>(x + off, delta ? delta + off : nullptr, dim, lane, [&](int e, uint16_t a16) {
      h_out[off + e] = float_to_out16(in16(float_to_out16(in16(a16, bf16) * rs, bf16), bf16) * in16(gamma[e], bf16), bf16);
    });
  }
}

// A few rows (a decoding step's): one block per row, eight elements per thread, so that a row's loads leave from all of its warps
// at once and the norm's weights are there before the stream dependency resolves.  A warp per row took 3.2 us (RMS, 2048) between
// two kernels of a step of one sequence and 4.8 us for 64, most of it the warp's own chain.
constexpr int kRowBlockMax = 256;  // threads: dim up to 2048
template <bool bf16, bool LAYER>
__global__ void __launch_bounds__(kRowBlockMax)
row_norm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ delta, const uint16_t* __restrict__ gamma, const uint16_t* __restrict__ beta,
                float eps, uint16_t* __restrict__ x_out, uint16_t* __restrict__ h_out, int dim) {
  __shared__ float part[2][kRowBlockMax / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int e = threadIdx.x * 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const uint4 gq = __ldg(reinterpret_cast<const uint4*>(gamma + e)), bq = LAYER ? __ldg(reinterpret_cast<const uint4*>(beta + e)) : make_uint4(0, 0, 0, 0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const size_t off = size_t(blockIdx.x) * dim + e;
  const uint4 a = ld_x4(x + off);
  uint32_t w[4] = {a.x, a.y, a.z, a.w};
  if (delta) {
    const uint4 d = ld_x4(delta + off);
    const uint32_t dw[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = uint32_t(float_to_out16(in16(uint16_t(w[j] & 0xffffu), bf16) + in16(uint16_t(dw[j] & 0xffffu), bf16), bf16)) |
             (uint32_t(float_to_out16(in16(uint16_t(w[j] >> 16), bf16) + in16(uint16_t(dw[j] >> 16), bf16), bf16)) << 16);
  }
  if (x_out) *reinterpret_cast<uint4*>(x_out + off) = make_uint4(w[0], w[1], w[2], w[3]);
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = in16(uint16_t(w[i >> 1] >> (16 * (i & 1))), bf16);
  auto total = [&](float s, int which) {  // over the block, the same in every thread
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) part[which][warp] = s;
    __syncthreads();
    float t = 0.f;
    for (int i = 0; i < nw; ++i) t += part[which][i];
    return t;
  };
  float mean = 0.f;
  if (LAYER) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += v[i];
    mean = total(s, 0) / float(dim);
  }
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) sq = fmaf(v[i] - mean, v[i] - mean, sq);
  const float rs = rsqrtf(total(sq, 1) / float(dim) + eps);
  const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w}, bw[4] = {bq.x, bq.y, bq.z, bq.w};
  uint32_t o[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float g = in16(uint16_t(gw[i >> 1] >> (16 * (i & 1))), bf16);
    const float y = LAYER ? ln_apply(v[i], mean, rs, g, in16(uint16_t(bw[i >> 1] >> (16 * (i & 1))), bf16))
                          : in16(float_to_out16(v[i] * rs, bf16), bf16) * g;
    o[i >> 1] |= uint32_t(float_to_out16(y, bf16)) << (16 * (i & 1));
  }
  *reinterpret_cast<uint4*>(h_out + off) = make_uint4(o[0], o[1], o[2], o[3]);
}

// gu: rows x 2*inter (gate columns first, then up), out: rows x inter; eight elements per thread and row, kSiluRows rows in
// flight.  Bound: issue of the exponential and the IEEE quotient beside the memory (6144 wide, fp16: 64 rows 2.4 us, 16512 rows
// 120 us or 5.07 TB/s; bf16 2.4 and 135).  __expf and __fdividef take 2.0 and 98 (2.1 and 106) but are tens of fp32 ulps off for
// large negative gates, and the quotient is 0 from a divisor of 2^126 on: bf16 gates of -87.5 to -88.5 lost their result.
constexpr int kSiluRows = 2;
template <bool bf16>
__global__ void __launch_bounds__(256)
silu_mul_kernel(const uint16_t* __restrict__ gu, uint16_t* __restrict__ out, int rows, int inter) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  gu = behind_wait(gu);
  const int c = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (c >= inter) return;
  for (int r0 = blockIdx.y * kSiluRows; r0 < rows; r0 += gridDim.y * kSiluRows) {
    uint4 g[kSiluRows], u[kSiluRows];
#pragma unroll
    for (int k = 0; k < kSiluRows; ++k) {
      const uint16_t* src = gu + size_t(min(r0 + k, rows - 1)) * 2 * inter + c;
      g[k] = *reinterpret_cast<const uint4*>(src);
      u[k] = *reinterpret_cast<const uint4*>(src + inter);
    }
#pragma unroll
    for (int k = 0; k < kSiluRows; ++k) {
      const uint32_t gw[4] = {g[k].x, g[k].y, g[k].z, g[k].w}, uw[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint16_t o2[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float gv = in16(uint16_t(gw[j] >> (16 * h)), bf16), uv = in16(uint16_t(uw[j] >> (16 * h)), bf16);
          const float sv = in16(float_to_out16(gv / (1.f + expf(-gv)), bf16), bf16);  // silu, rounded as the module rounds it
          o2[h] = float_to_out16(sv * uv, bf16);
        }
        ow[j] = uint32_t(o2[0]) | (uint32_t(o2[1]) << 16);
      }
      if (r0 + k < rows) *reinterpret_cast<uint4*>(out + size_t(r0 + k) * inter + c) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
  }
}

// qkv: rows x (nq + 2 nkv) x HD, a row = sequence b, step t (rows = B * T).  A warp takes up to kRopeHeads heads of one row, so
// that the row's cosines and sines are read once for them and all its loads are in flight together; HD / 8 lanes share a head,
// 8 elements each; the rotary partner of an element is the same slot of the lane HD / 16 away.  VEC: 16-byte accesses (else 8-byte
// aligned tensors).  q_out: B x nq x T x HD; caches: B x nkv x max_len x HD, written at position pos0 + t.
// Bound: memory.  With a warp per head, 4 elements a lane and the tables read by element it took four times its bytes.
constexpr int kRopeHeads = 8;
template <int HD, bool bf16, bool VEC>
__global__ void __launch_bounds__(256)
qk_norm_rope_kernel(const uint16_t* __restrict__ qkv, const uint16_t* __restrict__ qw, const uint16_t* __restrict__ kw,
                    const uint16_t* __restrict__ cos_t, const uint16_t* __restrict__ sin_t, const long long* __restrict__ pos_dev,
                    long long pos_host, uint16_t* __restrict__ q_out, uint16_t* __restrict__ k_cache, uint16_t* __restrict__ v_cache,
                    int rows, int T, int nq, int nkv, int max_len, float eps) {
  constexpr int LPH = HD / 8, PER = 32 / LPH, PASSES = kRopeHeads / PER;  // lanes per head, heads per pass
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  qkv = behind_wait(qkv);
  pos_dev = behind_wait(pos_dev);
  const int lane = threadIdx.x & 31, sub = lane % LPH, hg = lane / LPH;
  const int heads = nq + 2 * nkv;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), head0 = blockIdx.y * kRopeHeads;
  if (row >= rows) return;  // whole warps
  auto load8 = [&](const uint16_t* p, uint32_t (&w)[4]) {
    if (VEC) {
      const uint4 u = *reinterpret_cast<const uint4*>(p);
      w[0] = u.x, w[1] = u.y, w[2] = u.z, w[3] = u.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = uint32_t(p[2 * i]) | (uint32_t(p[2 * i + 1]) << 16);
    }
  };
  auto value = [&](const uint32_t (&w)[4], int i) { return in16(uint16_t(w[i >> 1] >> (16 * (i & 1))), bf16); };
  const int b = row / T, t = row - b * T;
  const long long pos = (pos_dev ? *pos_dev : pos_host) + t;
  uint32_t v[PASSES][4], cw[4], sw[4], wq[4], wk[4];
#pragma unroll
  for (int i = 0; i < PASSES; ++i) {
    const int head = head0 + i * PER + hg;
    if (head < heads) load8(qkv + (size_t(row) * heads + head) * HD + sub * 8, v[i]);
  }
  load8(cos_t + size_t(pos) * HD + sub * 8, cw);
  load8(sin_t + size_t(pos) * HD + sub * 8, sw);
  load8(qw + sub * 8, wq);
  load8(kw + sub * 8, wk);
#pragma unroll
  for (int i = 0; i < PASSES; ++i) {
    const int head = head0 + i * PER + hg;
    const bool is_q = head < nq, is_k = !is_q && head < nq + nkv, on = head < heads;
    // queries and keys: norm over the head, weight, rotary embedding (every lane takes part in the shuffles)
    float f[8], sq = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      f[e] = on ? value(v[i], e) : 0.f;
      sq = fmaf(f[e], f[e], sq);
    }
#pragma unroll
    for (int o = 1; o < LPH; o *= 2) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rs = rsqrtf(sq / float(HD) + eps);
    uint32_t out[4] = {0, 0, 0, 0};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float n = in16(float_to_out16(f[e] * rs, bf16), bf16);
      const float y = in16(float_to_out16((is_q ? value(wq, e) : value(wk, e)) * n, bf16), bf16);
      const float partner = __shfl_xor_sync(0xffffffffu, y, LPH / 2);
      const float rot = sub < LPH / 2 ? -partner : partner;
      const float a = in16(float_to_out16(y * value(cw, e), bf16), bf16);
      const float c = in16(float_to_out16(rot * value(sw, e), bf16), bf16);
      out[e >> 1] |= uint32_t(float_to_out16(a + c, bf16)) << (16 * (e & 1));
    }
    if (!on) continue;
    uint16_t* dst;
    if (is_q) {
      dst = q_out + ((size_t(b) * nq + head) * T + t) * HD + sub * 8;
    } else if (is_k) {
      dst = k_cache + ((size_t(b) * nkv + (head - nq)) * max_len + size_t(pos)) * HD + sub * 8;
    } else {
      dst = v_cache + ((size_t(b) * nkv + (head - nq - nkv)) * max_len + size_t(pos)) * HD + sub * 8;
    }
    const bool rotated = is_q || is_k;
    const uint4 o = make_uint4(rotated ? out[0] : v[i][0], rotated ? out[1] : v[i][1], rotated ? out[2] : v[i][2], rotated ? out[3] : v[i][3]);
    if (VEC) {
      *reinterpret_cast<uint4*>(dst) = o;
    } else {
      reinterpret_cast<uint2*>(dst)[0] = make_uint2(o.x, o.y);
      reinterpret_cast<uint2*>(dst)[1] = make_uint2(o.z, o.w);
    }
  }
}

// 16-byte vectors per thread in flight: four for the activation, whose arithmetic they hide, in one pass per block; one for the
// residual, whose three streams then move through memory together (12288 x 48000: 730 us a pass against 850 with four).  Bound:
// memory (with the type, the activation and the residual tested per element the activation ran at half of that).
constexpr int kEpiVecsResidual = 1, kEpiVecsActivation = 4;
template <bool bf16, bool GELU, bool RES>
__global__ void __launch_bounds__(256)
epilogue16_kernel(uint16_t* __restrict__ y, const uint16_t* __restrict__ residual, size_t n_vec) {
  constexpr int kEpiVecs = RES ? kEpiVecsResidual : kEpiVecsActivation;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  y = behind_wait(y);
  residual = behind_wait(residual);
  for (size_t i0 = size_t(blockIdx.x) * (256 * kEpiVecs) + threadIdx.x; i0 < n_vec; i0 += size_t(gridDim.x) * (256 * kEpiVecs)) {
    uint4 a[kEpiVecs], r[kEpiVecs];
#pragma unroll
    for (int k = 0; k < kEpiVecs; ++k) {
      const size_t i = i0 + k * 256;
      if (i < n_vec) {
        a[k] = reinterpret_cast<const uint4*>(y)[i];
        if (RES) r[k] = reinterpret_cast<const uint4*>(residual)[i];
      }
    }
#pragma unroll
    for (int k = 0; k < kEpiVecs; ++k) {
      const size_t i = i0 + k * 256;
      if (i >= n_vec) break;
      uint32_t aw[4] = {a[k].x, a[k].y, a[k].z, a[k].w};
      const uint32_t rw[4] = {RES ? r[k].x : 0u, RES ? r[k].y : 0u, RES ? r[k].z : 0u, RES ? r[k].w : 0u};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint16_t lo = epilogue16(uint16_t(aw[j] & 0xffffu), GELU ? kActGelu : kActNone, RES, uint16_t(rw[j] & 0xffffu), bf16);
        const uint16_t hi = epilogue16(uint16_t(aw[j] >> 16), GELU ? kActGelu : kActNone, RES, uint16_t(rw[j] >> 16), bf16);
        aw[j] = uint32_t(lo) | (uint32_t(hi) << 16);
      }
      reinterpret_cast<uint4*>(y)[i] = make_uint4(aw[0], aw[1], aw[2], aw[3]);
    }
  }
}

template <typename K, typename... Args>
int launch_pdl(K kern, dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
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

namespace {
// Rows up to which a block takes one: with more, warps of different rows hide each other's latencies and need no block barrier.
constexpr int kRowBlockRows = 296;
template <bool bf16>
int add_layernorm_as(const uint16_t* x, const uint16_t* delta, const uint16_t* gamma, const uint16_t* beta, float eps, uint16_t* x_out, uint16_t* h_out,
                     int rows, int dim, cudaStream_t stream) {
  const dim3 grid(unsigned((rows + kLnWarps - 1) / kLnWarps)), block(32 * kLnWarps);
  const bool vec_ok = aligned16(x) && aligned16(h_out) && aligned16(gamma) && aligned16(beta) && (!delta || aligned16(delta)) &&
                      (!x_out || aligned16(x_out));
  if (vec_ok && rows <= kRowBlockRows && dim % 256 == 0 && dim <= 8 * kRowBlockMax)
    return launch_pdl(row_norm_kernel<bf16, true>, dim3(unsigned(rows)), dim3(unsigned(dim / 8)), stream, x, delta, gamma, beta, eps, x_out, h_out, dim);
  auto run = [&](auto kern) { return launch_pdl(kern, grid, block, stream, x, delta, gamma, beta, eps, x_out, h_out, rows, dim); };
  if (vec_ok && dim == 1280) return run(add_layernorm_kernel<5, bf16>);
  if (vec_ok && dim == 1024) return run(add_layernorm_kernel<4, bf16>);
  if (vec_ok && dim == 2048) return run(add_layernorm_kernel<8, bf16>);
  if (vec_ok && dim == 256) return run(add_layernorm_kernel<1, bf16>);
  return run(add_layernorm_kernel<0, bf16>);
}
template <bool bf16>
int add_rmsnorm_as(const uint16_t* x, const uint16_t* delta, const uint16_t* gamma, float eps, uint16_t* x_out, uint16_t* h_out, int rows, int dim,
                   cudaStream_t stream) {
  const dim3 grid(unsigned((rows + kLnWarps - 1) / kLnWarps)), block(32 * kLnWarps);
  const bool vec_ok = aligned16(x) && aligned16(h_out) && aligned16(gamma) && (!delta || aligned16(delta)) && (!x_out || aligned16(x_out));
  if (vec_ok && rows <= kRowBlockRows && dim % 256 == 0 && dim <= 8 * kRowBlockMax)
    return launch_pdl(row_norm_kernel<bf16, false>, dim3(unsigned(rows)), dim3(unsigned(dim / 8)), stream, x, delta, gamma,
                      static_cast<const uint16_t*>(nullptr), eps, x_out, h_out, dim);
  auto run = [&](auto kern) { return launch_pdl(kern, grid, block, stream, x, delta, gamma, eps, x_out, h_out, rows, dim); };
  if (vec_ok && dim == 2048) return run(add_rmsnorm_kernel<8, bf16>);
  if (vec_ok && dim == 1024) return run(add_rmsnorm_kernel<4, bf16>);
  if (vec_ok && dim == 256) return run(add_rmsnorm_kernel<1, bf16>);
  return run(add_rmsnorm_kernel<0, bf16>);
}
const uint16_t* in_ptr(const void* v) { return static_cast<const uint16_t*>(v); }
uint16_t* out_ptr(void* v) { return static_cast<uint16_t*>(v); }
}  // namespace

int add_layernorm(const void* x, const void* delta, const void* gamma, const void* beta, float eps, void* x_out, void* h_out,
                  int64_t rows, int64_t dim, int dtype, cudaStream_t stream) {
  auto run = dtype == ASRQ_BF16 ? add_layernorm_as<true> : add_layernorm_as<false>;
  return run(in_ptr(x), in_ptr(delta), in_ptr(gamma), in_ptr(beta), eps, out_ptr(x_out), out_ptr(h_out), int(rows), int(dim), stream);
}

int add_rmsnorm(const void* x, const void* delta, const void* gamma, float eps, void* x_out, void* h_out, int64_t rows,
                int64_t dim, int dtype, cudaStream_t stream) {
  auto run = dtype == ASRQ_BF16 ? add_rmsnorm_as<true> : add_rmsnorm_as<false>;
  return run(in_ptr(x), in_ptr(delta), in_ptr(gamma), eps, out_ptr(x_out), out_ptr(h_out), int(rows), int(dim), stream);
}

int silu_mul(const void* gu, void* out, int64_t rows, int64_t inter, int dtype, int sm_count, cudaStream_t stream) {
  const unsigned gx = unsigned((inter / 8 + 255) / 256);
  const int64_t passes = (rows + kSiluRows - 1) / kSiluRows;
  const unsigned gy = unsigned(std::max<int64_t>(1, std::min<int64_t>({passes, int64_t(sm_count) * 16 / gx + 1, 65535})));
  return launch_pdl(dtype == ASRQ_BF16 ? silu_mul_kernel<true> : silu_mul_kernel<false>, dim3(gx, gy), dim3(256), stream, in_ptr(gu), out_ptr(out),
                    int(rows), int(inter));
}

int qk_norm_rope(const void* qkv, const void* qw, const void* kw, const void* cos_t, const void* sin_t, const long long* pos_dev,
                 long long pos_host, void* q_out, void* k_cache, void* v_cache, int64_t B, int64_t T, int nq, int nkv, int hd,
                 int64_t max_len, float eps, int dtype, cudaStream_t stream) {
  const dim3 grid(unsigned((B * T + 7) / 8), unsigned((nq + 2 * nkv + kRopeHeads - 1) / kRopeHeads)), block(256);
  bool vec = true;
  for (const void* q : {qkv, qw, kw, cos_t, sin_t, static_cast<const void*>(q_out), static_cast<const void*>(k_cache), static_cast<const void*>(v_cache)})
    vec = vec && aligned16(q);
  auto run = [&](auto kern) {
    return launch_pdl(kern, grid, block, stream, in_ptr(qkv), in_ptr(qw), in_ptr(kw), in_ptr(cos_t), in_ptr(sin_t), pos_dev, pos_host, out_ptr(q_out),
                      out_ptr(k_cache), out_ptr(v_cache), int(B * T), int(T), nq, nkv, int(max_len), eps);
  };
  const bool bf16 = dtype == ASRQ_BF16;
  if (hd == 128) {
    if (vec) return bf16 ? run(qk_norm_rope_kernel<128, true, true>) : run(qk_norm_rope_kernel<128, false, true>);
    return bf16 ? run(qk_norm_rope_kernel<128, true, false>) : run(qk_norm_rope_kernel<128, false, false>);
  }
  if (vec) return bf16 ? run(qk_norm_rope_kernel<64, true, true>) : run(qk_norm_rope_kernel<64, false, true>);
  return bf16 ? run(qk_norm_rope_kernel<64, true, false>) : run(qk_norm_rope_kernel<64, false, false>);
}

// y = act(y) / y = residual + y over M x N 16-bit elements (M*N a multiple of 8, pointers 16-byte aligned)
int epilogue16_apply(void* y, const void* residual, int64_t M, int64_t N, int act, int dtype, int sm_count, cudaStream_t stream) {
  const size_t n_vec = size_t(M) * size_t(N) / 8;
  const size_t per_block = 256 * (residual ? kEpiVecsResidual : kEpiVecsActivation), all = (n_vec + per_block - 1) / per_block;
  const unsigned blocks = unsigned(std::max<size_t>(1, std::min<size_t>(all, residual ? size_t(sm_count) * 8 : 0x7fffffffu)));
  auto run = [&](auto kern) { return launch_pdl(kern, dim3(blocks), dim3(256), stream, out_ptr(y), in_ptr(residual), n_vec); };
  const bool gelu = act == kActGelu;
  if (dtype == ASRQ_BF16) {
    if (residual) return gelu ? run(epilogue16_kernel<true, true, true>) : run(epilogue16_kernel<true, false, true>);
    return gelu ? run(epilogue16_kernel<true, true, false>) : run(epilogue16_kernel<true, false, false>);
  }
  if (residual) return gelu ? run(epilogue16_kernel<false, true, true>) : run(epilogue16_kernel<false, false, true>);
  return gelu ? run(epilogue16_kernel<false, true, false>) : run(epilogue16_kernel<false, false, false>);
}

}  // namespace asrq
