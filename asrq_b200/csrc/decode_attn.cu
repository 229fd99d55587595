// Attention of one decoding step: one new query per sequence (and query head) against a cache of keys and values.
//
//   self    the new key and value come out of the same fused projection row as the query and are written to the cache;
//   cross   keys and values are given (the encoder's, projected once), at any row and head stride;
//   grouped QH query heads share a key head; per-head RMS norm of queries and keys and the rotary embedding happen here too
//           (what qk_norm_rope_kernel does for a prompt), then as self.
//
// Bound: the bytes of the cache when there are many (sequence, head) items, else latency: a launch of 64 keys for one
// sequence took 8.5 us with one warp per item, each lane walking its keys' 128-byte rows alone.  Here an item is a block
// of 2, 4 or 8 warps, or a cluster of up to 8 such blocks when that fills the chip better.  HD / 8 lanes share a key (16 bytes
// each), a warp has eight such loads of keys and eight of values in flight, and the first of them go out BEFORE the stream
// dependency where the caller says that the cache is settled: in a decoder everything below the new position was written by
// earlier steps.  Eight keys' partial scores are summed over the
// lanes together by halving (7-8 shuffles instead of 24-32), after which every lane holds other keys' scores and the
// exponentials are not computed twice.  Warps and blocks meet as (maximum, sum, weighted values), blocks through the shared
// memory of the cluster's first.  fp32 scores, softmax and accumulation.
#include <atomic>
#include <cstdint>

#include "tcgen05.cuh"

namespace asrq {
namespace {

constexpr int kAttnWarps = 8;   // at most
constexpr int kU = 8;           // key loads in flight per lane
enum AttnKind { kAttnSelf = 0, kAttnCross = 1, kAttnGrouped = 2 };

struct AttnParams {
  const uint16_t* qkv;     // B rows of q_row values: [queries | keys | values] or queries only (cross)
  uint16_t* k;             // key of (sequence b, key head h, position t): k + b * sb + h * sh + t * st
  uint16_t* v;             // values: the same strides
  uint16_t* out;           // B x (hkv * QH * HD)
  const long long* pos;    // position of the new key (self, grouped)
  const uint16_t *qw, *kw, *cos_t, *sin_t;  // grouped
  long long sb, sh, st;
  int q_row, hkv, keys;    // keys: cross only
  float scale, eps;
  int bf16, q_vec;          // q_vec: the projection's rows are 16-byte aligned
  int early;                // keys and values in memory may be read ahead of the stream dependency
};

__device__ __forceinline__ float2 pair_to_float(uint32_t w, bool bf16) {
  if (bf16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return __half22float2(u32_as_h2(w));
}
__device__ __forceinline__ void eight(const uint4& u, bool bf16, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = pair_to_float(w[i], bf16);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8], bool bf16) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = uint32_t(float_to_out16(f[2 * i], bf16)) | (uint32_t(float_to_out16(f[2 * i + 1], bf16)) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 ld_stream(const uint16_t* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ uint4 ld_row(const uint16_t* p, bool vec) {
  if (vec) return *reinterpret_cast<const uint4*>(p);
  auto two = [&](int i) { return uint32_t(p[i]) | (uint32_t(p[i + 1]) << 16); };
  return make_uint4(two(0), two(2), two(4), two(6));
}

// RMS norm over the head (its HD / 8 lanes), weight, rotary embedding; rounded where the module sequence rounds
template <int LPK>
__device__ __forceinline__ void norm_rope8(float (&f)[8], const float (&w)[8], const float (&cs)[8], const float (&sn)[8], int sub, float eps, bool bf16) {
  auto r16 = [&](float x) { return out16_to_float(float_to_out16(x, bf16), bf16); };
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) sq = fmaf(f[i], f[i], sq);
#pragma unroll
  for (int o = 1; o < LPK; o *= 2) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  const float rs = rsqrtf(sq / float(8 * LPK) + eps);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float y = r16(w[i] * r16(f[i] * rs));
    const float partner = __shfl_xor_sync(0xffffffffu, y, LPK / 2);  // the element half a head away
    const float rot = sub < LPK / 2 ? -partner : partner;
    f[i] = r16(r16(y * cs[i]) + r16(rot * sn[i]));
  }
}

template <int HD, int QH, int KIND>
__global__ void __launch_bounds__(32 * kAttnWarps, 2)
decode_attn_kernel(const AttnParams p) {
  constexpr int LPK = HD / 8, KPI = 32 / LPK;   // lanes per key, keys per load
  constexpr int BATCH = kU * KPI;               // keys a warp has in flight
  constexpr float kLog2e = 1.4426950408889634f;
  __shared__ __align__(16) float part[kAttnWarps][QH][HD + 4];   // (values, maximum, sum) per warp, then per block of the cluster
  __shared__ __align__(16) float gathered[8][QH][HD + 4];        // first block of the cluster: one per block
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane % LPK, kg = lane / LPK, nw = blockDim.x >> 5;
  uint32_t rank = 0, nsplit = 1;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nsplit));
  // a block's shared memory may be written by another only once it is known to run: arrived here, waited for before the first write
  if (nsplit > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int item = int(blockIdx.x / nsplit), b = item / p.hkv, h = item - b * p.hkv;
  const bool bf16 = p.bf16 != 0;
  if (!p.early) asm volatile("griddepcontrol.wait;" ::: "memory");
  // the position is advanced by a kernel of the step before: complete, whatever runs just ahead of this one
  const int n = KIND == kAttnCross ? p.keys : int(*p.pos);  // keys in memory
  const uint16_t* kb = p.k + b * p.sb + h * p.sh + sub * 8;
  const uint16_t* vb = p.v + b * p.sb + h * p.sh + sub * 8;
  const int first = (int(rank) * nw + warp) * BATCH, stride = int(nsplit) * nw * BATCH;
  uint4 kr[kU], vr[kU];
  auto load = [&](const uint16_t* base, int t0, uint4 (&r)[kU]) {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * KPI + kg;
      r[u] = t < n ? ld_stream(base + t * p.st) : make_uint4(0, 0, 0, 0);
    }
  };
  if (first < n) {
    load(kb, first, kr);
    load(vb, first, vr);
  }
  // constants of the grouped form
  float wq[8], cs[8], sn[8];
  if constexpr (KIND == kAttnGrouped) {
    eight(__ldg(reinterpret_cast<const uint4*>(p.qw + sub * 8)), bf16, wq);
    eight(__ldg(reinterpret_cast<const uint4*>(p.cos_t + size_t(n) * HD + sub * 8)), bf16, cs);
    eight(__ldg(reinterpret_cast<const uint4*>(p.sin_t + size_t(n) * HD + sub * 8)), bf16, sn);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint16_t* row = p.qkv + size_t(b) * p.q_row;
  const int qw = p.hkv * QH * HD;
  uint4 qraw[QH], knew = make_uint4(0, 0, 0, 0), vnew = knew;
#pragma unroll
  for (int j = 0; j < QH; ++j) qraw[j] = ld_row(row + (h * QH + j) * HD + sub * 8, p.q_vec);
  const bool newest = KIND != kAttnCross && rank == 0 && warp == nw - 1;  // the warp that takes the new key
  if (newest) {
    knew = ld_row(row + qw + h * HD + sub * 8, p.q_vec);
    vnew = ld_row(row + qw + (p.hkv + h) * HD + sub * 8, p.q_vec);
  }
  float q[QH][8], o[QH][8], m[QH], l[QH];
#pragma unroll
  for (int j = 0; j < QH; ++j) {
    eight(qraw[j], bf16, q[j]);
    if constexpr (KIND == kAttnGrouped) norm_rope8<LPK>(q[j], wq, cs, sn, sub, p.eps, bf16);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      q[j][e] *= p.scale;
      o[j][e] = 0.f;
    }
    m[j] = -INFINITY;
    l[j] = 0.f;
  }
  if (newest) {
    float kf[8], vf[8];
    eight(knew, bf16, kf);
    eight(vnew, bf16, vf);
    if constexpr (KIND == kAttnGrouped) {
      float wk[8];
      eight(__ldg(reinterpret_cast<const uint4*>(p.kw + sub * 8)), bf16, wk);
      norm_rope8<LPK>(kf, wk, cs, sn, sub, p.eps, bf16);
      knew = pack8(kf, bf16);
    }
    if (kg == 0) {
      *reinterpret_cast<uint4*>(p.k + b * p.sb + h * p.sh + n * p.st + sub * 8) = knew;
      *reinterpret_cast<uint4*>(p.v + b * p.sb + h * p.sh + n * p.st + sub * 8) = vnew;
      __threadfence();
    }
#pragma unroll
    for (int j = 0; j < QH; ++j) {
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(q[j][e], kf[e], s);
#pragma unroll
      for (int x = 1; x < LPK; x *= 2) s += __shfl_xor_sync(0xffffffffu, s, x);
      m[j] = s;
      l[j] = lane == 0 ? 1.f : 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[j][e] = kg == 0 ? vf[e] : 0.f;
    }
  }
  // Only now may the next kernel start: a later step's launch of this one reads the cache before it waits for anything, so
  // the new key has to be in memory by the time the chain of early starts can reach it.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll 1
  for (int t0 = first; t0 < n; t0 += stride) {
    // scores: s[u] over this lane's eight dimensions, then summed over the key's lanes
    float s[QH][kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      float kf[8];
      eight(kr[u], bf16, kf);
#pragma unroll
      for (int j = 0; j < QH; ++j) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) a = fmaf(q[j][e], kf[e], a);
        s[j][u] = a;
      }
    }
    if (t0 + stride < n) load(kb, t0 + stride, kr);
    float pr[QH];
    const int mine = ((lane & 1) << 2) | (lane & 2) | ((lane >> 2) & 1);  // the load whose key's score this lane ends up with
    const bool live = t0 + mine * KPI + kg < n && (LPK == 8 || (lane & 8) == 0);
#pragma unroll
    for (int j = 0; j < QH; ++j) {
#pragma unroll
      for (int step = 0; step < 3; ++step) {
        const int hf = 4 >> step;
        const bool up = lane & (1 << step);
#pragma unroll
        for (int i = 0; i < hf; ++i) {
          const float give = up ? s[j][i] : s[j][i + hf], keep = up ? s[j][i + hf] : s[j][i];
          s[j][i] = keep + __shfl_xor_sync(0xffffffffu, give, 1 << step);
        }
      }
      float sc = s[j][0];
      if (LPK == 16) sc += __shfl_xor_sync(0xffffffffu, sc, 8);
      float mx = live ? sc : -INFINITY;
#pragma unroll
      for (int x = 16; x >= 1; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      mx = fmaxf(mx, m[j]);  // the batch holds a key: finite
      const float corr = exp2f((m[j] - mx) * kLog2e);
      m[j] = mx;
      const float e = exp2f((sc - mx) * kLog2e);
      l[j] = fmaf(l[j], corr, live ? e : 0.f);
      pr[j] = t0 + mine * KPI + kg < n ? e : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[j][i] *= corr;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      float vf[8];
      eight(vr[u], bf16, vf);
      const int src = (lane & ~7) | ((u & 1) << 2) | (u & 2) | ((u >> 2) & 1);
#pragma unroll
      for (int j = 0; j < QH; ++j) {
        const float w = __shfl_sync(0xffffffffu, pr[j], src);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[j][i] = fmaf(w, vf[i], o[j][i]);
      }
    }
    if (t0 + stride < n) load(vb, t0 + stride, vr);
  }
  // the warp's key groups, then its part of the block's result
#pragma unroll
  for (int j = 0; j < QH; ++j) {
#pragma unroll
    for (int x = 16; x >= 1; x >>= 1) l[j] += __shfl_xor_sync(0xffffffffu, l[j], x);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int x = 16; x >= LPK; x >>= 1) o[j][i] += __shfl_xor_sync(0xffffffffu, o[j][i], x);
    if (kg == 0) {
      float* d = &part[warp][j][sub * 8];
      *reinterpret_cast<float4*>(d) = make_float4(o[j][0], o[j][1], o[j][2], o[j][3]);
      *reinterpret_cast<float4*>(d + 4) = make_float4(o[j][4], o[j][5], o[j][6], o[j][7]);
      if (sub == 0) {
        part[warp][j][HD] = m[j];
        part[warp][j][HD + 1] = l[j];
      }
    }
  }
  __syncthreads();
  auto merge = [&](const float (*src)[QH][HD + 4], int count, int j, int e, float& mx, float& lt) {
    mx = -INFINITY;
    for (int w = 0; w < count; ++w) mx = fmaxf(mx, src[w][j][HD]);
    float acc = 0.f;
    lt = 0.f;
    for (int w = 0; w < count; ++w) {
      const float mw = src[w][j][HD], wt = mw == -INFINITY ? 0.f : exp2f((mw - mx) * kLog2e);
      acc = fmaf(wt, src[w][j][e], acc);
      lt = fmaf(wt, src[w][j][HD + 1], lt);
    }
    return acc;
  };
  uint16_t* out = p.out + size_t(b) * qw + size_t(h) * QH * HD;
  if (nsplit == 1) {
    for (int i = threadIdx.x; i < QH * HD; i += blockDim.x) {
      float mx, lt;
      const float acc = merge(part, nw, i / HD, i % HD, mx, lt);
      out[i] = float_to_out16(acc / lt, bf16);
    }
    return;
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t dst0 = tc::mapa(tc::smem_u32(&gathered[rank][0][0]), 0);
  for (int i = threadIdx.x; i < QH * HD; i += blockDim.x) {
    const int j = i / HD, e = i % HD;
    float mx, lt;
    const float acc = merge(part, nw, j, e, mx, lt);
    const uint32_t d = dst0 + uint32_t(j * (HD + 4) + e) * 4u;
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(d), "f"(acc) : "memory");
    if (e == 0) {
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(d + HD * 4u), "f"(mx) : "memory");
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(d + HD * 4u + 4u), "f"(lt) : "memory");
    }
  }
  tc::cluster_sync();  // the parts have arrived; the first block is still there to receive them
  if (rank == 0)
    for (int i = threadIdx.x; i < QH * HD; i += blockDim.x) {
      float mx, lt;
      const float acc = merge(gathered, int(nsplit), i / HD, i % HD, mx, lt);
      out[i] = float_to_out16(acc / lt, bf16);
    }
}

// Blocks of `warps` warps, in clusters of `split`, that the device holds at once (the clusters of a size leave SMs unused)
template <int HD, int QH, int KIND>
int resident_blocks(int split, int warps, int sm_count) {
  static std::atomic<int> known[9][9];  // one kind of device: asked once per process
  std::atomic<int>& k = known[split][warps];
  int n = k.load(std::memory_order_relaxed);
  if (n) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(split));
  cfg.blockDim = dim3(32 * warps);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, decode_attn_kernel<HD, QH, KIND>, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 2 * sm_count / split;
  }
  k.store(n * split, std::memory_order_relaxed);
  return n * split;
}

template <int HD, int QH, int KIND>
int launch_attn(const AttnParams& p, int64_t items, int64_t max_keys, int sm_count, cudaStream_t stream) {
  // Blocks per item and warps per block: the pair with the least (waves of resident blocks) x (batches a warp walks, plus 2 for
  // the launch, the query and the merge, plus 1 for the cluster's merge); the fewest blocks among equals, since the cache may be
  // much shorter than max_keys.  Two warps keep many items of few keys in one wave (640 items, us: 10 keys 4.6 -> 3.2, 64
  // 5.5 -> 4.1, 128 8.3 -> 6.9; 320 items of 1500 keys in clusters of three 29 -> 23).  Clusters of more than two blocks count a
  // sixteenth fewer slots than the occupancy query gives: behind a running launch they do not pack as tightly (377 clusters of
  // three by the query; 340 take one wave and 23.4 us, 360 take 32.4, and 29.7 as single blocks of four warps).
  constexpr int BATCH = kU * 32 / (HD / 8);
  int split = 1, warps = kAttnWarps;
  int64_t best = INT64_MAX;
  for (int sp = 1; sp <= 8; ++sp)
    for (int w : {8, 4, 2}) {
      const int64_t held = resident_blocks<HD, QH, KIND>(sp, w, sm_count), slots = sp > 2 ? held * 15 / 16 : held;
      const int64_t waves = (items * sp + slots - 1) / slots;
      const int64_t cost = waves * ((max_keys + sp * w * BATCH - 1) / (sp * w * BATCH) + (sp > 1 ? 3 : 2));
      if (cost < best) {
        best = cost;
        split = sp;
        warps = w;
      }
    }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(items * split));
  cfg.blockDim = dim3(32 * warps);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 1 : 2;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, decode_attn_kernel<HD, QH, KIND>, p));
  return ASRQ_OK;
}

}  // namespace

int decode_self_attention(const void* qkv, void* kv, const long long* pos_dev, void* out, int64_t B, int H, int hd, int64_t max_len,
                          float scale, bool settled, int dtype, int sm_count, cudaStream_t stream) {
  AttnParams p = {};
  p.qkv = static_cast<const uint16_t*>(qkv);
  p.k = static_cast<uint16_t*>(kv);
  p.v = p.k + size_t(B) * H * max_len * hd;
  p.out = static_cast<uint16_t*>(out);
  p.pos = pos_dev;
  p.sb = (long long)H * max_len * hd;
  p.sh = (long long)max_len * hd;
  p.st = hd;
  p.q_row = 3 * H * hd;
  p.early = settled;
  p.hkv = H;
  p.scale = scale;
  p.bf16 = dtype == ASRQ_BF16;
  p.q_vec = aligned16(p.qkv);
  if (hd == 64) return launch_attn<64, 1, kAttnSelf>(p, B * H, max_len, sm_count, stream);
  return launch_attn<128, 1, kAttnSelf>(p, B * H, max_len, sm_count, stream);
}

int decode_cross_attention(const void* q, const void* k, const void* v, void* out, int64_t B, int H, int hd, int64_t keys, int64_t row_stride,
                           float scale, bool settled, int dtype, int sm_count, cudaStream_t stream) {
  AttnParams p = {};
  p.qkv = static_cast<const uint16_t*>(q);
  p.k = static_cast<uint16_t*>(const_cast<void*>(k));
  p.v = static_cast<uint16_t*>(const_cast<void*>(v));
  p.out = static_cast<uint16_t*>(out);
  p.sb = keys * row_stride;
  p.sh = hd;
  p.st = row_stride;
  p.q_row = H * hd;
  p.hkv = H;
  p.keys = int(keys);
  p.early = settled;
  p.scale = scale;
  p.bf16 = dtype == ASRQ_BF16;
  p.q_vec = aligned16(p.qkv);
  if (hd == 64) return launch_attn<64, 1, kAttnCross>(p, B * H, keys, sm_count, stream);
  return launch_attn<128, 1, kAttnCross>(p, B * H, keys, sm_count, stream);
}

int decode_grouped_attention(const void* qkv, const void* qw, const void* kw, const void* cos_t, const void* sin_t, const long long* pos_dev,
                             void* k_cache, void* v_cache, void* out, int64_t B, int nkv, int64_t max_len, float eps, float scale, int dtype,
                             int sm_count, cudaStream_t stream) {
  constexpr int hd = 128, qh = 2;
  AttnParams p = {};
  p.qkv = static_cast<const uint16_t*>(qkv);
  p.k = static_cast<uint16_t*>(k_cache);
  p.v = static_cast<uint16_t*>(v_cache);
  p.out = static_cast<uint16_t*>(out);
  p.pos = pos_dev;
  p.qw = static_cast<const uint16_t*>(qw);
  p.kw = static_cast<const uint16_t*>(kw);
  p.cos_t = static_cast<const uint16_t*>(cos_t);
  p.sin_t = static_cast<const uint16_t*>(sin_t);
  p.sb = (long long)nkv * max_len * hd;
  p.sh = (long long)max_len * hd;
  p.st = hd;
  p.q_row = (qh + 2) * nkv * hd;
  p.hkv = nkv;
  p.early = 1;
  p.eps = eps;
  p.scale = scale;
  p.bf16 = dtype == ASRQ_BF16;
  p.q_vec = aligned16(p.qkv);
  return launch_attn<hd, qh, kAttnGrouped>(p, B * nkv, max_len, sm_count, stream);
}

}  // namespace asrq
