// W4A4 GEMM, register-tile variants (mma.sync.m16n8k32 s8): w4a4_few_kernel for up to 64 tokens, w4a4_mma_kernel for the other
// shapes that the tcgen05 kernel does not take (ragged N tiles, wide groups) and as its cross-check.
//
// Both operands are packed signed nibbles.  A nibble pair word q is split into
// E = (q << 4) & 0xf0f0f0f0 (even k) and O = q & 0xf0f0f0f0 (odd k): each byte is
// then 16x the signed value, so a product is 256x the true one and the exact group
// sum is (acc >> 8).  The k order inside a lane's 32-k span is the same for both
// operands, which is all a contraction needs.
//
// Per 128-k step (one weight group) the int32 tile is scaled by sW[n, group] and
// added to an fp32 running sum; the per-token scale and the bias come last.
#include <algorithm>

#include "common.cuh"

namespace asrq {

int ensure_dynamic_smem(const void* kernel, size_t bytes);

struct W4A4Params {
  const uint8_t* qa;
  const float* sa;
  const uint8_t* qw;
  const __half* sw;
  const __half* bias;
  uint16_t* y;
  int32_t* acc_dump;
  int M, N, K, group_size, groups, bf16;
};

__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// block: 4 warps as 2(m) x 2(n); warp tile 32(m) x 32(n); block tile 64 x 64.
__global__ void __launch_bounds__(128) w4a4_mma_kernel(const W4A4Params p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const int m_base = blockIdx.y * 64 + (warp >> 1) * 32;
  const int n_base = blockIdx.x * 64 + (warp & 1) * 32;
  const size_t row_bytes = size_t(p.K) / 2;
  const int steps_per_group = p.group_size / 128;

  float accf[2][4][4];
  int acc[2][4][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        accf[a][b][i] = 0.f;
        acc[a][b][i] = 0;
      }

  const int nsteps = p.K / 128;
  for (int step = 0; step < nsteps; ++step) {
    const size_t koff = size_t(step) * 64 + c * 16;  // bytes
    uint4 ar[2][2], br[4];
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m_base + 16 * f + 8 * h + g;
        ar[f][h] = m < p.M ? __ldg(reinterpret_cast<const uint4*>(p.qa + m * row_bytes + koff))
                           : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int n = n_base + 8 * f + g;
      br[f] = __ldg(reinterpret_cast<const uint4*>(p.qw + n * row_bytes + koff));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t ae[2][2], ao[2][2], be[4], bo[4];
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t q = (&ar[f][h].x)[j];
          ae[f][h] = (q << 4) & 0xf0f0f0f0u;
          ao[f][h] = q & 0xf0f0f0f0u;
        }
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const uint32_t q = (&br[f].x)[j];
        be[f] = (q << 4) & 0xf0f0f0f0u;
        bo[f] = q & 0xf0f0f0f0u;
      }
#pragma unroll
      for (int fm = 0; fm < 2; ++fm)
#pragma unroll
        for (int fn = 0; fn < 4; ++fn)
          mma_s8(acc[fm][fn], ae[fm][0], ae[fm][1], ao[fm][0], ao[fm][1], be[fn], bo[fn]);
    }
    if ((step + 1) % steps_per_group == 0) {
      const int gi = step / steps_per_group;
#pragma unroll
      for (int fn = 0; fn < 4; ++fn) {
        const int n0 = n_base + 8 * fn + 2 * c;
        const float s0 = __half2float(__ldg(p.sw + size_t(n0) * p.groups + gi));
        const float s1 = __half2float(__ldg(p.sw + size_t(n0 + 1) * p.groups + gi));
#pragma unroll
        for (int fm = 0; fm < 2; ++fm)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int v = acc[fm][fn][i] >> 8;
            accf[fm][fn][i] += float(v) * ((i & 1) ? s1 : s0);
            if (p.acc_dump) {
              const int m = m_base + 16 * fm + 8 * (i >> 1) + g;
              if (m < p.M) p.acc_dump[(size_t(m) * p.N + n0 + (i & 1)) * p.groups + gi] = v;
            }
            acc[fm][fn][i] = 0;
          }
      }
    }
  }
#pragma unroll
  for (int fm = 0; fm < 2; ++fm)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = m_base + 16 * fm + 8 * h + g;
      if (m >= p.M) continue;
      const float s = __ldg(p.sa + m);
#pragma unroll
      for (int fn = 0; fn < 4; ++fn) {
        const int n0 = n_base + 8 * fn + 2 * c;
        float v0 = accf[fm][fn][2 * h] * s, v1 = accf[fm][fn][2 * h + 1] * s;
        if (p.bias) {
          v0 += ldg_half(p.bias + n0);
          v1 += ldg_half(p.bias + n0 + 1);
        }
        const uint32_t o = uint32_t(float_to_out16(v0, p.bf16)) | (uint32_t(float_to_out16(v1, p.bf16)) << 16);
        *reinterpret_cast<uint32_t*>(p.y + size_t(m) * p.N + n0) = o;
      }
    }
}

// ---- up to 64 tokens, groups of 128 ------------------------------------------------------------------------------------
// A block owns 16 features, its warps the groups of K in turn; a warp's operands are fragments as they lie in memory (16 bytes of a
// row per lane: words j = 0..3 of four lanes make the 32 k of step j, the same for both operands).  Weights are the MMA's A operand, up
// to eight tiles of eight tokens its B.  Weights and scales are constants and are fetched ahead of the stream dependency.  The groups'
// exact sums meet in shared memory as 16-bit integers (at most 128 * 7 * 8) and are scaled and added there in group order, so that a call
// has the bits of w4a4_mma_kernel: behind four bits a last place can move a later layer's codes.
// Bound: latency (launch, one L2 trip for the codes, the sums' way through shared memory).  The kernel above gives 64 features and all
// of K to four warps and launches behind the end of the quantisation: 4096 -> 1024 ran on 16 SMs, 32 dependent trips to L2 each.
// Chains of quantisation and GEMM, that -> this, us: 1024 -> 1024, one token 9.7 -> 3.5, 63 tokens 11.7 -> 5.7; 1024 -> 4096 10.0 -> 3.7 and 11.7 -> 6.2;
// 4096 -> 1024 29.5 -> 5.4 and 32.8 -> 9.5.  Calls: 12.3 -> 8.5, 30.8 -> 8.6 (the host).
constexpr int kFewMaxWarps = 16, kFewAhead = 2;
constexpr size_t kFewMaxSmem = 200 * 1024;
constexpr size_t few_smem(int groups, int nt) { return size_t(groups) * (size_t(nt) * 2 * 32 * 4 + 16 * 4); }
template <int NT>
__global__ void __launch_bounds__(32 * kFewMaxWarps) w4a4_few_kernel(const W4A4Params p) {
  extern __shared__ uint32_t sums[];                                              // [group][2 t + feature half][lane]: tokens 8 t + 2 c, + 1
  float* const scales = reinterpret_cast<float*>(sums + size_t(p.groups) * NT * 2 * 32);  // [group][16]
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g = lane >> 2, c = lane & 3, n0 = blockIdx.x * 16 + g;
  const size_t row_bytes = size_t(p.K) / 2;
  uint4 wr[kFewAhead][2];
  auto fetch = [&](int gi, int at) {
    const size_t off = size_t(gi) * 64 + c * 16;
    wr[at][0] = __ldg(reinterpret_cast<const uint4*>(p.qw + size_t(n0) * row_bytes + off));
    wr[at][1] = __ldg(reinterpret_cast<const uint4*>(p.qw + size_t(n0 + 8) * row_bytes + off));
  };
#pragma unroll
  for (int a = 0; a < kFewAhead; ++a)
    if (warp + a * nw < p.groups) fetch(warp + a * nw, a);
  for (int i = threadIdx.x; i < p.groups * 16; i += blockDim.x)
    scales[i] = ldg_half(p.sw + size_t(blockIdx.x * 16 + (i & 15)) * p.groups + (i >> 4));
  asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
  for (int g0 = warp; g0 < p.groups; g0 += kFewAhead * nw) {
#pragma unroll
    for (int a = 0; a < kFewAhead; ++a) {
      const int gi = g0 + a * nw;
      if (gi >= p.groups) break;
      uint4 xr[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        xr[t] = make_uint4(0, 0, 0, 0);
        const int m = t * 8 + g;
        if (m < p.M)  // (volatile: not ahead of the wait)
          asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(xr[t].x), "=r"(xr[t].y), "=r"(xr[t].z), "=r"(xr[t].w)
                       : "l"(p.qa + size_t(m) * row_bytes + size_t(gi) * 64 + c * 16) : "memory");
      }
      int acc[NT][4];
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t q0 = (&wr[a][0].x)[j], q1 = (&wr[a][1].x)[j];
        const uint32_t e0 = (q0 << 4) & 0xf0f0f0f0u, e1 = (q1 << 4) & 0xf0f0f0f0u, o0 = q0 & 0xf0f0f0f0u, o1 = q1 & 0xf0f0f0f0u;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const uint32_t q = (&xr[t].x)[j];
          mma_s8(acc[t], e0, e1, o0, o1, (q << 4) & 0xf0f0f0f0u, q & 0xf0f0f0f0u);
        }
      }
      if (gi + kFewAhead * nw < p.groups) fetch(gi + kFewAhead * nw, a);
      // acc[t][i]: feature g + 8 * (i / 2), token 8 t + 2 c + i % 2
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          sums[((gi * NT + t) * 2 + h) * 32 + lane] = uint32_t((acc[t][2 * h] >> 8) & 0xffff) | (uint32_t(acc[t][2 * h + 1] >> 8) << 16);
    }
  }
  __syncthreads();
  // two tokens of a feature per thread and turn, features fastest: 32 contiguous bytes of a token's row by 16 threads
  for (int o = threadIdx.x; o < NT * 4 * 16; o += blockDim.x) {
    const int f = o & 15, m = (o >> 4) * 2;
    if (m >= p.M) break;
    const uint32_t* src = sums + ((m >> 3) * 2 + (f >> 3)) * 32 + (f & 7) * 4 + ((m & 7) >> 1);
    float v0 = 0.f, v1 = 0.f;
    for (int gi = 0; gi < p.groups; ++gi) {
      const uint32_t w = src[gi * (NT * 2 * 32)];
      const float s = scales[gi * 16 + f];
      v0 += float(int16_t(w & 0xffffu)) * s;
      v1 += float(int16_t(w >> 16)) * s;
    }
    const int n = blockIdx.x * 16 + f;
    float s0, s1 = 0.f;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(s0) : "l"(p.sa + m) : "memory");
    if (m + 1 < p.M) asm volatile("ld.global.f32 %0, [%1];" : "=f"(s1) : "l"(p.sa + m + 1) : "memory");
    v0 *= s0;
    v1 *= s1;
    if (p.bias) {
      const float b = ldg_half(p.bias + n);
      v0 += b;
      v1 += b;
    }
    p.y[size_t(m) * p.N + n] = float_to_out16(v0, p.bf16);
    if (m + 1 < p.M) p.y[size_t(m + 1) * p.N + n] = float_to_out16(v1, p.bf16);
  }
}

template <int NT>
int launch_few(const W4A4Params& p, cudaStream_t stream) {
  const size_t smem = few_smem(p.groups, NT);
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(w4a4_few_kernel<NT>), smem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(p.N / 16));
  cfg.blockDim = dim3(32 * std::min(p.groups, kFewMaxWarps));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, w4a4_few_kernel<NT>, p));
  return ASRQ_OK;
}

int w4a4_gemm_mma(const uint8_t* qa, const float* sa, const uint8_t* qw, const void* sw, const void* bias,
                  void* y, int32_t* acc_dump, int64_t M, int64_t N, int64_t K, int group_size, int dtype,
                  cudaStream_t stream) {
  if (group_size <= 0 || N % 64 || K % 128 || group_size % 128 || K % group_size)
    return fail(ASRQ_ERR_SHAPE,
                "w4a4 gemm: need N%%64==0, K%%128==0, group_size%%128==0, K%%group_size==0 "
                "(N=%lld K=%lld g=%d)", (long long)N, (long long)K, group_size);
  if (M <= 0) return ASRQ_OK;
  W4A4Params p;
  p.qa = qa; p.sa = sa; p.qw = qw;
  p.sw = static_cast<const __half*>(sw);
  p.bias = static_cast<const __half*>(bias);
  p.y = static_cast<uint16_t*>(y);
  p.acc_dump = acc_dump;
  p.M = int(M); p.N = int(N); p.K = int(K);
  p.group_size = group_size;
  p.groups = int(K / group_size);
  p.bf16 = dtype == ASRQ_BF16;
  if (M <= 64 && group_size == 128 && !acc_dump && few_smem(p.groups, M <= 8 ? 1 : (M <= 16 ? 2 : (M <= 32 ? 4 : 8))) <= kFewMaxSmem) {
    if (M <= 8) return launch_few<1>(p, stream);
    if (M <= 16) return launch_few<2>(p, stream);
    return M <= 32 ? launch_few<4>(p, stream) : launch_few<8>(p, stream);
  }
  dim3 grid(unsigned(N / 64), unsigned((M + 63) / 64));
  w4a4_mma_kernel<<<grid, 128, 0, stream>>>(p);
  ASRQ_CUDA_TRY(cudaGetLastError());
  return ASRQ_OK;
}

}  // namespace asrq
