// The floating-point output head of a decoding step: y[M, N] = x[M, K] . W[N, K]^T for M <= 32 tokens and a
// vocabulary-sized N (Whisper's proj_out 1280 -> 51 866, Qwen3's lm_head 2048 -> 151 936; the reference keeps
// these layers as nn.Linear: asrq/models/transformers/whisper.py:268, asrq/models/nemo/canary_qwen.py:179).
//
// Bound: HBM (the weight is read once: 133 MB and 622 MB for the two heads above, against a few hundred KB of
// activations and logits).  The decode kernel's skeleton without the unpacking: a warp owns 16 weight rows, every
// lane reads 16 bytes of rows g and g + 8 per 32-wide K step straight from global memory (its own fragment of
// mma.sync.m16n8k16 under a fixed permutation of k inside the step, which the activation fragments follow), the
// activations sit in shared memory for the whole block, accumulation in fp32.
//
// Shared memory, MMAs and the loads in flight follow the number of token tiles (NT: 8, 16 or 32 tokens).  With one form for
// 32 tokens a single token paid for four tiles of MMAs, and at K = 2048 its 133 KB allowed one block of 12 warps with four
// steps ahead: 49 KB in flight on an SM, about what the memory's latency takes at full rate -- 213 us for 622 MB.  Two blocks of
// six steps, or one of eight where the activations fill the shared memory, hold 98-147 KB in flight.
#include <algorithm>

#include "common.cuh"

namespace asrq {

int ensure_dynamic_smem(const void* kernel, size_t bytes);

namespace {

constexpr int kHeadWarps = 12;

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, bool bf16) {
  if (bf16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

__device__ __forceinline__ uint4 ldg_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// The next token of every row: the index of the largest logit (the first of equals; a NaN is larger than any number, as in torch),
// in kArgmaxParts blocks per row that meet by one atomic maximum of (ordered value, ~index) and a counter; the last of a row
// writes and leaves both at zero.  Bound: latency, some hundred KB per row from L2; the library's reduction in one block per row
// took 8 to 23 us of a step, and a copy and an indexed copy followed it.
constexpr int kArgmaxParts = 16;
template <bool BF16, bool PAIRS>
__global__ void __launch_bounds__(256)
argmax_rows_kernel(const uint16_t* __restrict__ y, long long* __restrict__ tok, long long* __restrict__ ids, const long long* __restrict__ pos,
                   unsigned long long* __restrict__ best, unsigned* __restrict__ arrived, int N) {
  __shared__ unsigned long long part[8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  y = behind_wait(y);
  pos = behind_wait(pos);
  const int row = blockIdx.y;
  const uint16_t* src = y + size_t(row) * N;
  auto ordered = [](uint32_t b) {  // monotone in the value; zeros equal; NaN above everything
    if ((b & 0x7fffu) > (BF16 ? 0x7f80u : 0x7c00u)) return 0xffffu;
    if (b == 0x8000u) b = 0u;
    return (b & 0x8000u) ? (~b & 0xffffu) : (b | 0x8000u);
  };
  uint32_t top = 0, at = 0;  // every number's order is above zero
  auto see = [&](uint32_t bits, int i) {
    const uint32_t o = ordered(bits);
    if (o > top) {
      top = o;
      at = uint32_t(i);
    }
  };
  if (PAIRS) {
    const int n2 = N / 2, lo = int((long long)n2 * blockIdx.x / kArgmaxParts), hi = int((long long)n2 * (blockIdx.x + 1) / kArgmaxParts);
#pragma unroll 4
    for (int i = lo + threadIdx.x; i < hi; i += 256) {
      const uint32_t w = reinterpret_cast<const uint32_t*>(src)[i];
      see(w & 0xffffu, 2 * i);
      see(w >> 16, 2 * i + 1);
    }
  } else {
    const int lo = int((long long)N * blockIdx.x / kArgmaxParts), hi = int((long long)N * (blockIdx.x + 1) / kArgmaxParts);
    for (int i = lo + threadIdx.x; i < hi; i += 256) see(src[i], i);
  }
  unsigned long long key = (static_cast<unsigned long long>(top) << 32) | (top ? 0xffffffffu - at : 0u);
  auto larger = [](unsigned long long a, unsigned long long b) { return a > b ? a : b; };
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) key = larger(key, __shfl_xor_sync(0xffffffffu, key, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = key;
  __syncthreads();
  if (threadIdx.x) return;
#pragma unroll
  for (int i = 1; i < 8; ++i) key = larger(key, part[i]);
  atomicMax(best + row, key);
  __threadfence();
  if (atomicAdd(arrived + row, 1u) != kArgmaxParts - 1) return;
  __threadfence();
  const long long t = static_cast<long long>(0xffffffffu - uint32_t(atomicExch(best + row, 0ull)));
  arrived[row] = 0u;
  tok[row] = t;
  if (ids) ids[*pos * gridDim.y + row] = t;
}

// x: M x K, w: N x K, y: M x N, all 16-bit of one type; K a multiple of 32; shared memory: head_smem(NT, K) bytes.
// PER_SM: blocks that share an SM; AHEAD: K steps of weight loads in flight per warp.
template <bool BF16, int NT, int PER_SM>
__global__ void __launch_bounds__(32 * kHeadWarps, PER_SM)
dense_head_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, uint16_t* __restrict__ y, int M, int N, int K) {
  constexpr int kHeadTokens = 8 * NT, kHeadAhead = PER_SM == 1 ? 8 : (NT == 4 ? 4 : 6);
  extern __shared__ __align__(16) uint16_t xs[];
  // row pitch = 64 bytes modulo 128: the eight lanes of a quarter warp (two token rows x four 16-byte pieces) then
  // read eight distinct 16-byte bank groups
  const int pitch = K + ((K & 63) ? 0 : 32);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n_tiles = (N + 15) / 16;
  const int steps = K / 32;
  int tile = blockIdx.x * kHeadWarps + warp;
  const int tile_stride = gridDim.x * kHeadWarps;

  // the weights do not depend on the kernel before this one on the stream: the first loads go out before the wait
  uint4 wa[kHeadAhead], wb[kHeadAhead];
  auto rows_of = [&](int tl, const uint16_t*& ra, const uint16_t*& rb) {
    const int r0 = tl * 16 + g, r1 = r0 + 8;
    ra = w + size_t(min(r0, N - 1)) * K + 8 * t;  // rows past the end read the last row; their results are not stored
    rb = w + size_t(min(r1, N - 1)) * K + 8 * t;
  };
  const uint16_t *ra = w, *rb = w;
  if (tile < n_tiles) {
    rows_of(tile, ra, rb);
#pragma unroll
    for (int i = 0; i < kHeadAhead; ++i) {
      if (i < steps) {
        wa[i] = ldg_stream16(ra + 32 * i);
        wb[i] = ldg_stream16(rb + 32 * i);
      }
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  x = behind_wait(x);
  // activations -> shared memory (rows beyond M are zero)
  for (int i = threadIdx.x; i < kHeadTokens * (K / 8); i += blockDim.x) {
    const int r = i / (K / 8), c = (i - r * (K / 8)) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < M) v = *reinterpret_cast<const uint4*>(x + size_t(r) * K + c);
    *reinterpret_cast<uint4*>(xs + r * pitch + c) = v;
  }
  __syncthreads();

  for (; tile < n_tiles; tile += tile_stride) {
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    for (int s0 = 0; s0 < steps; s0 += kHeadAhead) {
#pragma unroll
      for (int i = 0; i < kHeadAhead; ++i) {
        const int s = s0 + i;
        if (s < steps) {
          const uint4 a = wa[i], b = wb[i];
          if (s + kHeadAhead < steps) {  // refill this slot
            wa[i] = ldg_stream16(ra + 32 * (s + kHeadAhead));
            wb[i] = ldg_stream16(rb + 32 * (s + kHeadAhead));
          }
          // k slots (2t, 2t+1 | 2t+8, 2t+9) of the two MMAs of this step hold actual k = 8t + (0,1 | 2,3) and 8t + (4,5 | 6,7)
          const uint32_t a0[4] = {a.x, b.x, a.y, b.y}, a1[4] = {a.z, b.z, a.w, b.w};
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint4 xv = *reinterpret_cast<const uint4*>(xs + (8 * j + g) * pitch + 32 * s + 8 * t);
            mma16816(acc[j], a0, xv.x, xv.y, BF16);
            mma16816(acc[j], a1, xv.z, xv.w, BF16);
          }
        }
      }
    }
    // the next tile's first loads go out before this tile's stores
    const int next = tile + tile_stride;
    if (next < n_tiles) {
      rows_of(next, ra, rb);
#pragma unroll
      for (int i = 0; i < kHeadAhead; ++i) {
        if (i < steps) {
          wa[i] = ldg_stream16(ra + 32 * i);
          wb[i] = ldg_stream16(rb + 32 * i);
        }
      }
    }
    const int r0 = tile * 16 + g, r1 = r0 + 8;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int m0 = 8 * j + 2 * t, m1 = m0 + 1;
      if (m0 < M) {
        if (r0 < N) y[size_t(m0) * N + r0] = float_to_out16(acc[j][0], BF16);
        if (r1 < N) y[size_t(m0) * N + r1] = float_to_out16(acc[j][2], BF16);
      }
      if (m1 < M) {
        if (r0 < N) y[size_t(m1) * N + r0] = float_to_out16(acc[j][1], BF16);
        if (r1 < N) y[size_t(m1) * N + r1] = float_to_out16(acc[j][3], BF16);
      }
    }
  }
}

size_t head_smem(int tiles, int64_t K) { return size_t(8 * tiles) * size_t(K + ((K & 63) ? 0 : 32)) * 2; }

using HeadKernel = void (*)(const uint16_t*, const uint16_t*, uint16_t*, int, int, int);
template <bool BF16>
HeadKernel head_kernel(int tiles, int per_sm) {
  if (tiles == 1) return dense_head_kernel<BF16, 1, 2>;
  if (tiles == 2) return per_sm == 2 ? dense_head_kernel<BF16, 2, 2> : dense_head_kernel<BF16, 2, 1>;
  return per_sm == 2 ? dense_head_kernel<BF16, 4, 2> : dense_head_kernel<BF16, 4, 1>;
}

}  // namespace

int dense_head(const void* x, const void* w, void* y, int64_t M, int64_t N, int64_t K, int dtype, int sm_count, cudaStream_t stream) {
  const int tiles = M <= 8 ? 1 : (M <= 16 ? 2 : 4);
  const size_t smem = head_smem(tiles, K);
  const int blocks_per_sm = smem <= 100 * 1024 ? 2 : 1;  // (K <= 3200: always 2 for one tile)
  const HeadKernel kern = dtype == ASRQ_BF16 ? head_kernel<true>(tiles, blocks_per_sm) : head_kernel<false>(tiles, blocks_per_sm);
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
  const int64_t n_tiles = (N + 15) / 16;
  const int grid = int(std::min<int64_t>(int64_t(sm_count) * blocks_per_sm, (n_tiles + kHeadWarps - 1) / kHeadWarps));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * kHeadWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(w),
                                   static_cast<uint16_t*>(y), int(M), int(N), int(K)));
  return ASRQ_OK;
}

// scratch: 16 bytes per row, zero between calls
int argmax_rows(const void* y, long long* tok, long long* ids, const long long* pos, void* scratch, int64_t B, int64_t N, int dtype, cudaStream_t stream) {
  unsigned long long* best = static_cast<unsigned long long*>(scratch);
  unsigned* arrived = reinterpret_cast<unsigned*>(best + B);
  const bool pairs = N % 2 == 0 && reinterpret_cast<uintptr_t>(y) % 4 == 0;
  auto kern = dtype == ASRQ_BF16 ? (pairs ? argmax_rows_kernel<true, true> : argmax_rows_kernel<true, false>)
                                 : (pairs ? argmax_rows_kernel<false, true> : argmax_rows_kernel<false, false>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kArgmaxParts, unsigned(B));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<const uint16_t*>(y), tok, ids, pos, best, arrived, int(N)));
  return ASRQ_OK;
}

}  // namespace asrq
