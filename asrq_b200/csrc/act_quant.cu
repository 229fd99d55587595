// W4A4 prologue: optional online Hadamard rotation + per-token symmetric int4
// quantisation, one warp per token, everything in fp32 registers.
//
// The rotation is the normalised Walsh-Hadamard transform computed as butterflies
// with strides 1, 2, 4, ... K/2 in that order, (a, b) -> (a + b, a - b), followed by
// a division by sqrt(K).  Each output of a stage is a single fp32 add or subtract of
// two values of the previous stage, so the result is bit-identical to any other
// evaluation that keeps the stage order, however the butterflies are spread over
// lanes.  A lane holds V = K/32 consecutive elements: the strides below V are
// register-to-register, the five strides V..16V are warp shuffles.
//
// Quantisation: s = absmax/7 (0 -> 1e-3), q = rint(v/s) with IEEE division and
// round-half-even, packed two's-complement nibbles, even k in the low nibble.
#include <cuda_fp8.h>

#include <algorithm>

#include "tcgen05.cuh"

namespace asrq {

int current_device_sm_count(int* sm_count);

constexpr int kQuantWarps = 4;

__device__ __forceinline__ float in16_to_float(uint16_t b, bool bf16) {
  return bf16 ? bf16_bits_to_float(b) : __half2float(__ushort_as_half(b));
}

// Per-token scale and its reciprocal.
struct QScale {
  float s, inv;
};

// rint(v / s) with IEEE division, bit for bit, without a division per element: r = v * (1/s) is
// within 1.3e-6 of the correctly rounded quotient (|r| <= 7), so both round to the same integer
// unless r lies within 1e-5 of a tie; only then is the true quotient computed.  Rounding to
// nearest-even is done by adding 1.5 * 2^23, which also leaves the two's-complement code in the
// low mantissa bits, so there is no float->int conversion either.  |code| <= 7 by construction
// (s = absmax / 7), as in the reference formula, which has no clamp.
__device__ __forceinline__ int quant1(float v, QScale qs) {
  const float magic = 12582912.f;
  const float r = __fmul_rn(v, qs.inv);
  float t = __fadd_rn(r, magic);
  const float d = fabsf(__fsub_rn(r, __fsub_rn(t, magic)));
  if (d > 0.49999f) t = __fadd_rn(rintf(__fdiv_rn(v, qs.s)), magic);
  return __float_as_int(t) - 0x4B400000;
}

__device__ __forceinline__ QScale make_qscale(float amax) {
  QScale q;
  q.s = __fdiv_rn(amax, 7.f);
  if (q.s == 0.f) q.s = 1e-3f;
  q.inv = __fdiv_rn(1.f, q.s);
  return q;
}

__device__ __forceinline__ uint32_t pack8_int4(const float* v, QScale s) {
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) w |= (uint32_t(quant1(v[i], s)) & 0xFu) << (4 * i);
  return w;
}

// Four codes as int8 bytes holding 16x the value (the operand format of the tcgen05 W4A4 GEMM).
__device__ __forceinline__ uint32_t pack4_int8x16(const float* v, QScale s) {
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) w |= ((uint32_t(quant1(v[i], s)) << 4) & 0xFFu) << (8 * i);
  return w;
}

// OUT = 0: packed nibbles (K/2 bytes per token); OUT = 1: int8 holding 16*q (K bytes per token).
// Four codes as FP8 e4m3 bytes holding the value itself (the operand format of the kind::f8f6f4 GEMM).
__device__ __forceinline__ uint32_t e4m3x2(float a, float b) {
  return uint32_t(__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ uint32_t pack4_e4m3(const float* v, QScale s) {
  return e4m3x2(float(quant1(v[0], s)), float(quant1(v[1], s))) |
         (e4m3x2(float(quant1(v[2], s)), float(quant1(v[3], s))) << 16);
}
template <int OUT>
__device__ __forceinline__ uint32_t pack4_operand(const float* v, QScale s) {
  return OUT == 2 ? pack4_e4m3(v, s) : pack4_int8x16(v, s);
}

template <int V, int OUT>
__global__ void __launch_bounds__(kQuantWarps * 32)
hadamard_quant_kernel(const uint16_t* __restrict__ x, uint8_t* __restrict__ qa,
                      float* __restrict__ sa, int M, int K, int bf16) {
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * kQuantWarps + (threadIdx.x >> 5);
  if (token >= M) return;
  float v[V];
  const uint4* src = reinterpret_cast<const uint4*>(x + size_t(token) * K + lane * V);
#pragma unroll
  for (int i = 0; i < V / 8; ++i) {
    const uint4 u = __ldg(src + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[8 * i + 2 * j] = in16_to_float(uint16_t(w[j] & 0xffffu), bf16);
      v[8 * i + 2 * j + 1] = in16_to_float(uint16_t(w[j] >> 16), bf16);
    }
  }
  // strides 1 .. V/2: inside the lane
#pragma unroll
  for (int h = 1; h < V; h <<= 1) {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if ((j & h) == 0) {
        const float a = v[j], b = v[j + h];
        v[j] = a + b;
        v[j + h] = a - b;
      }
    }
  }
  // strides V .. 16V: across lanes
#pragma unroll
  for (int mask = 1; mask < 32; mask <<= 1) {
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float o = __shfl_xor_sync(0xffffffffu, v[j], mask);
      v[j] = upper ? (o - v[j]) : (v[j] + o);
    }
  }
  const float root = sqrtf(float(K));
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    v[j] = __fdiv_rn(v[j], root);
    amax = fmaxf(amax, fabsf(v[j]));
  }
#pragma unroll
  for (int mask = 16; mask > 0; mask >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, mask));
  const QScale s = make_qscale(amax);
  if (lane == 0) sa[token] = s.s;
  if (OUT >= 1) {
    uint32_t* d8 = reinterpret_cast<uint32_t*>(qa + size_t(token) * K + lane * V);
    if (V >= 16) {
#pragma unroll
      for (int i = 0; i < V / 16; ++i)
        reinterpret_cast<uint4*>(d8)[i] = make_uint4(pack4_operand<OUT>(v + 16 * i, s), pack4_operand<OUT>(v + 16 * i + 4, s),
                                                     pack4_operand<OUT>(v + 16 * i + 8, s), pack4_operand<OUT>(v + 16 * i + 12, s));
    } else {
#pragma unroll
      for (int i = 0; i < V / 4; ++i) d8[i] = pack4_operand<OUT>(v + 4 * i, s);
    }
    return;
  }
  uint32_t* dst = reinterpret_cast<uint32_t*>(qa + size_t(token) * (K / 2) + lane * (V / 2));
  if (V >= 32) {
#pragma unroll
    for (int i = 0; i < V / 32; ++i) {
      uint4 o;
      o.x = pack8_int4(v + 32 * i, s);
      o.y = pack8_int4(v + 32 * i + 8, s);
      o.z = pack8_int4(v + 32 * i + 16, s);
      o.w = pack8_int4(v + 32 * i + 24, s);
      reinterpret_cast<uint4*>(dst)[i] = o;
    }
  } else {
#pragma unroll
    for (int i = 0; i < V / 8; ++i) dst[i] = pack8_int4(v + 8 * i, s);
  }
}

// No rotation: any K that is a multiple of 8.  Two passes over the token (the second
// one hits L1/L2).
template <int OUT>
__global__ void __launch_bounds__(kQuantWarps * 32)
quant_int4_kernel(const uint16_t* __restrict__ x, uint8_t* __restrict__ qa, float* __restrict__ sa,
                  int M, int K, int bf16) {
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * kQuantWarps + (threadIdx.x >> 5);
  if (token >= M) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + size_t(token) * K);
  const int units = K / 8;
  float amax = 0.f;
  for (int i = lane; i < units; i += 32) {
    const uint4 u = __ldg(src + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      amax = fmaxf(amax, fabsf(in16_to_float(uint16_t(w[j] & 0xffffu), bf16)));
      amax = fmaxf(amax, fabsf(in16_to_float(uint16_t(w[j] >> 16), bf16)));
    }
  }
#pragma unroll
  for (int mask = 16; mask > 0; mask >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, mask));
  const QScale s = make_qscale(amax);
  if (lane == 0) sa[token] = s.s;
  uint32_t* dst = reinterpret_cast<uint32_t*>(qa + size_t(token) * (OUT >= 1 ? K : K / 2));
  for (int i = lane; i < units; i += 32) {
    const uint4 u = __ldg(src + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = in16_to_float(uint16_t(w[j] & 0xffffu), bf16);
      v[2 * j + 1] = in16_to_float(uint16_t(w[j] >> 16), bf16);
    }
    if (OUT >= 1) {
      reinterpret_cast<uint2*>(dst)[i] = make_uint2(pack4_operand<OUT>(v, s), pack4_operand<OUT>(v + 4, s));
    } else {
      dst[i] = pack8_int4(v, s);
    }
  }
}

// K = 1024 and 4096: 32 and 64 threads per token, each with 32 and 64 values, and ONE transpose through shared memory where the
// kernel above has five levels of shuffles:
//   phase A  thread t holds the T consecutive elements t * T + e: strides 1 .. T / 2;
//   phase B  thread u holds the elements o * T + u, o = 0..T-1: strides T .. K / 2.  Four neighbouring threads transpose their
//            4 x 4 bytes of codes by two shuffles per word, so that a warp stores whole 32-byte sectors.
// The strides are taken in ascending order, as everywhere in this file: another order rounds differently, and behind four bits a
// difference in the last place can move a code.
// Values live as pairs, so every butterfly but the one inside the pair is a packed fp32 add and a packed subtract (add.f32x2 /
// fma.f32x2) on two pairs.  Rows of the transpose are padded by four floats: its 4-byte writes and 16-byte reads are free of bank
// conflicts.
// 256, 512 and 2048, which no layer of the models here has, stay with the kernel above: 512 and 2048 are no squares.
// The division by sqrt(K) = 32 or 64 is exact and is applied to the scale only: rint((v/64) / (s/64)) is rint(v/s) bit for bit.
// Quantisation without a division per element: t_lo = fma(v, inv_lo, magic), t_hi = fma(v, inv_hi,
// magic) with inv_lo < 1/s < inv_hi (2^-22 apart) bracket the exact quotient, and adding 1.5*2^23
// rounds to nearest-even and leaves the two's-complement code in the low mantissa bits; where the
// two agree (all but a few elements in a million) that is rint(v/s); where they differ the true
// quotient is computed.
__device__ __forceinline__ float2 sub2(float2 a, float2 c) { return __ffma2_rn(c, make_float2(-1.f, -1.f), a); }

// The rare path of quant8_bytes, out of line so that its call sites do not swell the kernel: IEEE division and round-half-even,
// as magic + code.
__device__ __noinline__ float4 quant4_exact(float2 v01, float2 v23, float s) {
  return make_float4(__fadd_rn(rintf(__fdiv_rn(v01.x, s)), 12582912.f), __fadd_rn(rintf(__fdiv_rn(v01.y, s)), 12582912.f),
                     __fadd_rn(rintf(__fdiv_rn(v23.x, s)), 12582912.f), __fadd_rn(rintf(__fdiv_rn(v23.y, s)), 12582912.f));
}

// Codes of eight values as two words: OUT 0 and 1 as bytes b0..b3 = low byte of each t (t = magic + code), OUT 2 as e4m3 bytes
template <int OUT>
__device__ __forceinline__ void quant8_bytes(const float2 (&v)[4], float2 inv_lo, float2 inv_hi, float s, uint32_t (&out)[2]) {
  const float2 magic = make_float2(12582912.f, 12582912.f);
  float2 a[4];
  uint32_t diff = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[i] = __ffma2_rn(v[i], inv_lo, magic);
    const float2 h = __ffma2_rn(v[i], inv_hi, magic);
    diff |= __float_as_uint(a[i].x) ^ __float_as_uint(h.x);
    diff |= __float_as_uint(a[i].y) ^ __float_as_uint(h.y);
  }
  if (diff != 0) {  // an element within 4e-6 of a rounding boundary: IEEE division
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 e = quant4_exact(v[2 * i], v[2 * i + 1], s);
      a[2 * i] = make_float2(e.x, e.y);
      a[2 * i + 1] = make_float2(e.z, e.w);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float2 p = a[2 * i], q = a[2 * i + 1];
    if (OUT == 2) {
      const float2 nm = make_float2(-12582912.f, -12582912.f);
      p = __fadd2_rn(p, nm);  // exact: the code as a float
      q = __fadd2_rn(q, nm);
      out[i] = e4m3x2(p.x, p.y) | (e4m3x2(q.x, q.y) << 16);
    } else {
      out[i] = prmt(prmt(__float_as_uint(p.x), __float_as_uint(p.y), 0x0040u), prmt(__float_as_uint(q.x), __float_as_uint(q.y), 0x0040u), 0x5410u);
    }
  }
}

// log2 levels over an array of pairs: strides of 1 .. N / 2 pairs
template <int N>
__device__ __forceinline__ void butterflies(float2 (&P)[N]) {
#pragma unroll
  for (int h = 1; h < N; h <<= 1)
#pragma unroll
    for (int j = 0; j < N; ++j)
      if ((j & h) == 0) {
        const float2 a = P[j], c = P[j + h];
        P[j] = __fadd2_rn(a, c);
        P[j + h] = sub2(a, c);
      }
}
template <int N>
__device__ __forceinline__ void inside_pairs(float2 (&P)[N]) {
#pragma unroll
  for (int j = 0; j < N; ++j) P[j] = make_float2(P[j].x + P[j].y, P[j].x - P[j].y);
}

template <int N>
__device__ __forceinline__ float largest(const float2 (&P)[N]) {
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) amax = fmaxf(amax, fmaxf(fabsf(P[j].x), fabsf(P[j].y)));
#pragma unroll
  for (int mask = 16; mask > 0; mask >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, mask));
  return amax;
}
// scale of the unnormalised values, with the bracket of its reciprocal; the token's scale is that / sqrt(K) (exact)
struct CodeScale {
  float s;
  float2 inv_lo, inv_hi;
};
template <int K>
__device__ __forceinline__ CodeScale code_scale(float amax, float* sa) {
  CodeScale c;
  c.s = __fdiv_rn(amax, 7.f);
  const bool zero = c.s == 0.f;
  if (sa) *sa = zero ? 1e-3f : c.s * (K == 4096 ? 0.015625f : 0.03125f);
  if (zero) c.s = 1.f;  // every value is 0: any scale gives code 0
  const float inv = __fdiv_rn(1.f, c.s);
  const float il = inv * (1.f - 2.384185791015625e-07f), ih = inv * (1.f + 2.384185791015625e-07f);  // 2^-22
  c.inv_lo = make_float2(il, il);
  c.inv_hi = make_float2(ih, ih);
  return c;
}
// Codes of twice four values that lie a row of memory apart each, held by each of four neighbouring lanes at neighbouring places
// of these rows: after the exchange a lane has four neighbouring places of row (lane & 3) of either four, which go to elements
// at0 and at1 of the token.
template <int K, int OUT>
__device__ __forceinline__ void store_codes(const float2 (&v)[4], const CodeScale& c, int lane, uint8_t* __restrict__ qa, int64_t token, int at0, int at1) {
  const uint32_t sel1 = (lane & 2) ? 0x3276u : 0x5410u, sel2 = (lane & 1) ? 0x3715u : 0x6240u;
  uint32_t w[2];
  quant8_bytes<OUT>(v, c.inv_lo, c.inv_hi, c.s, w);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t b = prmt(w[i], __shfl_xor_sync(0xffffffffu, w[i], 2), sel1);
    b = prmt(b, __shfl_xor_sync(0xffffffffu, b, 1), sel2);
    const int at = i ? at1 : at0;
    if (OUT >= 1) {
      *reinterpret_cast<uint32_t*>(qa + size_t(token) * K + at) = OUT == 1 ? (b << 4) & 0xf0f0f0f0u : b;
    } else {
      const uint32_t n = b & 0x0f0f0f0fu, m = n | (n >> 4);  // bytes 0 and 2 hold two nibbles each, element 0 lowest
      *reinterpret_cast<uint16_t*>(qa + size_t(token) * (K / 2) + at / 2) = uint16_t((m & 0xffu) | ((m >> 8) & 0xff00u));
    }
  }
}
template <bool BF16, int N>
__device__ __forceinline__ void unpack8(const uint4& q, float2 (&P)[N], int at) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int e = 0; e < 4; ++e)
    P[at + e] = BF16 ? make_float2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u)) : __half22float2(u32_as_h2(w[e]));
}
// K = 1024: a warp per token, four to a block
template <int OUT, bool BF16>
__global__ void __launch_bounds__(128, 5)
hadamard_1024_quant_kernel(const uint16_t* __restrict__ x, uint8_t* __restrict__ qa, float* __restrict__ sa, int M) {
  constexpr int K = 1024, T = 32, PITCH = T + 4, UNITS = T / 8;  // 16-byte units per thread
  __shared__ __align__(16) float rows_all[4][T * PITCH];  // the 16-bit input is staged in its first half
  // A GEMM launched behind this kernel with programmatic stream serialisation may be scheduled once
  // every block of this grid has started, and set itself up on SMs the last wave leaves idle; it
  // orders itself with griddepcontrol.wait before it touches this kernel's output.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = threadIdx.x % T, token = blockIdx.x * 4 + threadIdx.x / T;
  float* rows = rows_all[threadIdx.x / T];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (token >= M) return;  // a whole warp, which meets no other
  const uint4* src = reinterpret_cast<const uint4*>(x + size_t(token) * K) + t;
  uint4* stage = reinterpret_cast<uint4*>(rows);
  auto slot = [](int owner, int j) { return owner * UNITS + (j ^ ((owner >> 1) & 3)); };  // conflict-free both ways
  uint4 raw[UNITS];
#pragma unroll
  for (int i = 0; i < UNITS; ++i)  // (behind the wait: __ldg could be moved ahead of it)
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(raw[i].x), "=r"(raw[i].y), "=r"(raw[i].z), "=r"(raw[i].w) : "l"(src + i * T) : "memory");
#pragma unroll
  for (int i = 0; i < UNITS; ++i) stage[slot((i * T + t) / UNITS, (i * T + t) % UNITS)] = raw[i];
  __syncwarp();
  {
    float2 P[T / 2];
#pragma unroll
    for (int i = 0; i < UNITS; ++i) unpack8<BF16>(stage[slot(t, i)], P, 4 * i);
    inside_pairs(P);
    butterflies(P);
    __syncwarp();  // the staged rows have been read
#pragma unroll
    for (int i = 0; i < T / 2; ++i) {
      rows[(2 * i) * PITCH + t] = P[i].x;
      rows[(2 * i + 1) * PITCH + t] = P[i].y;
    }
  }
  __syncwarp();
  float2 Q[T / 2];
#pragma unroll
  for (int k = 0; k < T / 4; ++k) {
    const float4 z = *reinterpret_cast<const float4*>(rows + t * PITCH + 4 * k);
    Q[2 * k] = make_float2(z.x, z.y);
    Q[2 * k + 1] = make_float2(z.z, z.w);
  }
  inside_pairs(Q);
  butterflies(Q);
  const CodeScale c = code_scale<K>(largest(Q), t == 0 ? sa + token : nullptr);
#pragma unroll
  for (int k = 0; k < T / 8; ++k) {
    const float2 v[4] = {Q[4 * k], Q[4 * k + 1], Q[4 * k + 2], Q[4 * k + 3]};
    const int at = (8 * k + (t & 3)) * T + (t & ~3);
    store_codes<K, OUT>(v, c, t, qa, token, at, at + 4 * T);
  }
}

// The wait for this block's own copy, bounded like every wait of the library.
__device__ __forceinline__ bool wait_landed(uint32_t bar, uint32_t parity) {
  if (tc::mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (clock64() - t0 <= tc::kWaitCycles)
    if (tc::mbar_try_wait(bar, parity)) return true;
  return false;
}

// K = 4096: 64 threads per token, each with 64 values, in blocks that walk the tokens.
// A token's 8 KB arrive by one bulk copy, asked for as soon as the token before has been read from the same place, and lie as in
// memory.  Thread t's 128 bytes all start in the same bank, so it takes its eight 16-byte units in the order i ^ r, r = t % 8.  Place i
// then holds unit i ^ r, and for the strides between units (8, 16, 32) the partners of a butterfly have changed places where their
// bit of r is set: the sum is the same, the difference has the other sign, which changes nothing in how it rounds.  After phase A
// place i holds unit i with the sign (-1)^popcount(i & r): over the o of phase B a Walsh function, under which the butterflies of
// strides T, 2 T and 4 T exchange their results.  Place m after phase B is o = m ^ s, s = t / 8, and the codes are stored accordingly;
// no sign is ever put back.
// Bound: no single one.  About 2 300 warp instructions a token, a third of them packed ones and conversions that issue at half rate
// or less (ncu: 56% of the issue slots), with three barriers a token between them; the bytes go at half the copy rate.  128 threads of 32 values with two transposes and 32 warps per SM: 24.9 us for 6 000
// tokens; more warps of this code, at 80 registers: no change.  Chains of launches, loads in the chain and a branch per four codes -> this
// form, us: one token 2.6 -> 2.3, 250 4.95 -> 4.4, 6 000 22.2 -> 21.5, 16 000 57.6 -> 53.5; the 1024-wide kernel with a branch per eight codes
// 1.70 -> 1.56, 2.0 -> 1.9, 6.2 -> 6.0, 12.85 -> 12.67.
template <int OUT, bool BF16>
__global__ void __launch_bounds__(64, 8)
hadamard_4096_quant_kernel(const uint16_t* __restrict__ x, uint8_t* __restrict__ qa, float* __restrict__ sa, int M) {
  constexpr int K = 4096, T = 64, PITCH = T + 4, UNITS = T / 8;
  __shared__ __align__(128) uint4 stage[K / 8];
  __shared__ __align__(16) float rows[T * PITCH];
  __shared__ float part[2];
  __shared__ __align__(8) uint64_t full;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = threadIdx.x;
  const uint32_t bar = tc::smem_u32(&full), dst = tc::smem_u32(stage);
  auto fetch = [&](int token) {
    tc::mbar_arrive_expect_tx(bar, K * 2);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(x + size_t(token) * K), "r"(K * 2), "r"(bar)
                 : "memory");
  };
  if (t == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_barrier_init();
    tc::fence_proxy_async_smem();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (t == 0) fetch(blockIdx.x);
  __syncthreads();
  const int s = t >> 3;
  uint32_t ph = 0;
  for (int token = blockIdx.x; token < M; token += gridDim.x, ph ^= 1u) {
    const bool landed = wait_landed(bar, ph);
    {
      float2 P[T / 2];
#pragma unroll
      for (int i = 0; i < UNITS; ++i) unpack8<BF16>(stage[t * UNITS + (i ^ (t & 7))], P, 4 * i);
      inside_pairs(P);
      butterflies(P);
#pragma unroll
      for (int i = 0; i < T / 2; ++i) {
        rows[(2 * i) * PITCH + t] = P[i].x;
        rows[(2 * i + 1) * PITCH + t] = P[i].y;
      }
    }
    __syncthreads();  // the transpose is written and the staged bytes have been read
    if (t == 0 && token + int(gridDim.x) < M) fetch(token + gridDim.x);
    float2 Q[T / 2];
#pragma unroll
    for (int k = 0; k < T / 4; ++k) {
      const float4 z = *reinterpret_cast<const float4*>(rows + t * PITCH + 4 * k);
      Q[2 * k] = make_float2(z.x, z.y);
      Q[2 * k + 1] = make_float2(z.z, z.w);
    }
    inside_pairs(Q);
    butterflies(Q);
    const float m = largest(Q);
    if ((t & 31) == 0) part[t >> 5] = m;
    __syncthreads();  // also: the transpose has been read, the next token's may be written
    const CodeScale c = code_scale<K>(fmaxf(part[0], part[1]), t == 0 ? sa + token : nullptr);
    if (!landed && t == 0) sa[token] = __int_as_float(0x7fc00000);  // gave up waiting: the token's outputs are NaN
#pragma unroll
    for (int k = 0; k < T / 8; ++k) {
      const float2 v[4] = {Q[4 * k], Q[4 * k + 1], Q[4 * k + 2], Q[4 * k + 3]};
      const int at = ((8 * k + (t & 3)) ^ s) * T + (t & ~3);
      store_codes<K, OUT>(v, c, t, qa, token, at, at ^ (4 * T));
    }
  }
}

static int launch_had(void (*kern)(const uint16_t*, uint8_t*, float*, int), int64_t blocks, int threads, const uint16_t* xp, uint8_t* qa, float* sa,
                      int64_t M, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, xp, qa, sa, int(M)));
  return ASRQ_OK;
}

template <int OUT>
static int launch_quant(const uint16_t* xp, uint8_t* qa, float* sa, int64_t M, int64_t K, int hadamard, int bf16,
                        cudaStream_t stream) {
  int sm_count = 0;
  if (const int rc = current_device_sm_count(&sm_count)) return rc;
  const int blocks = int((M + kQuantWarps - 1) / kQuantWarps);
  const int thr = kQuantWarps * 32;
  if (!hadamard) {
    if (K % 8 || K <= 0) return fail(ASRQ_ERR_SHAPE, "quant_int4: K %% 8 != 0 (K=%lld)", (long long)K);
    quant_int4_kernel<OUT><<<blocks, thr, 0, stream>>>(xp, qa, sa, int(M), int(K), bf16);
  } else {
    switch (K) {
      case 256: hadamard_quant_kernel<8, OUT><<<blocks, thr, 0, stream>>>(xp, qa, sa, int(M), int(K), bf16); break;
      case 512: hadamard_quant_kernel<16, OUT><<<blocks, thr, 0, stream>>>(xp, qa, sa, int(M), int(K), bf16); break;
      case 1024:
        return launch_had(bf16 ? hadamard_1024_quant_kernel<OUT, true> : hadamard_1024_quant_kernel<OUT, false>, (M + 3) / 4, 128, xp, qa, sa, M, stream);
      case 2048: hadamard_quant_kernel<64, OUT><<<blocks, thr, 0, stream>>>(xp, qa, sa, int(M), int(K), bf16); break;
      case 4096:
        return launch_had(bf16 ? hadamard_4096_quant_kernel<OUT, true> : hadamard_4096_quant_kernel<OUT, false>, std::min<int64_t>(M, 8 * sm_count), 64, xp,
                          qa, sa, M, stream);
      default:
        return fail(ASRQ_ERR_SHAPE, "hadamard_quant_int4: K must be 256, 512, 1024, 2048 or 4096 (K=%lld)",
                    (long long)K);
    }
  }
  ASRQ_CUDA_TRY(cudaGetLastError());
  return ASRQ_OK;
}

// out_fmt = 0: qa receives packed nibbles (M x K/2); 1: int8 holding 16*q (M x K); 2: e4m3 holding q (M x K).
int hadamard_quant_int4(const void* x, uint8_t* qa, float* sa, int64_t M, int64_t K, int hadamard, int dtype,
                        int out_fmt, cudaStream_t stream) {
  if (M <= 0) return ASRQ_OK;
  const uint16_t* xp = static_cast<const uint16_t*>(x);
  const int bf16 = dtype == ASRQ_BF16;
  if (out_fmt == 2) return launch_quant<2>(xp, qa, sa, M, K, hadamard, bf16, stream);
  return out_fmt ? launch_quant<1>(xp, qa, sa, M, K, hadamard, bf16, stream)
                 : launch_quant<0>(xp, qa, sa, M, K, hadamard, bf16, stream);
}

}  // namespace asrq
