// Large W{2,4}A16 calls: the weights dequantised once per call, then a plain 16-bit GEMM on CTA pairs with the epilogue in it.
//
// The kernels that unpack weights inside the GEMM do it again for every token tile: at 48 000 tokens the same 128 x 64 block of
// weights is unpacked 188 times, beside the MMAs and at the same power budget, and their few epilogue warps have no issue slots
// left for an activation.  Here `unpack_kernel` writes the layer's 16-bit weights into scratch of the call's own (13 MB for
// 1280 -> 5120, which stay in L2) and `gemm_dense_kernel` takes both operands by TMA:
//
//   * activations are the MMA's A operand (256 tokens of a CTA pair, 128 per CTA = TMEM lanes), weights the B operand (up to
//     256 features = TMEM columns, each CTA loads half): tcgen05.mma.cta_group::2, M = 256;
//   * a ring of stages of 64 elements of K; two accumulator buffers of 256 columns, so that a tile's epilogue runs under the next
//     tile's main loop;
//   * warp 0 TMA producer (both CTAs), warp 1 MMA issuer (CTA 0), from warp 4 on the epilogue: a warp owns 32 tokens and takes
//     32 features at a time.  A lane holds one token's row, so bias, rounding, GELU and residual act on registers; the 32 x 32 tile
//     goes through 2 KB of swizzled shared memory and leaves by TMA, which clips the ragged edges.  The residual comes the same
//     way into the same place.
//
// Bound: the MMAs, at the clock that the power limit leaves; in a call of a few rounds also the two launches with the unpacking
// between them (about 9 us together with the first fetches and the last stores).  Measured, chains of calls, W4 fp16, unpacking in
// the GEMM and a pass for the epilogue -> this form, us: 48 000 tokens of 5120 -> 1280 with residual 643 -> 432 (1457 TFLOP/s), of
// 1280 -> 5120 with GELU 863 -> 520, without epilogue 526 -> 424; 6 000 tokens of 1280 -> 5120 with residual 113 -> 66; 1500 with GELU
// 32 -> 27.  Same bits: the products are summed in the same order.
#include <algorithm>

#include "tcgen05.cuh"
#include "dequant.cuh"

namespace asrq {

int ensure_dynamic_smem(const void* kernel, size_t bytes);

namespace {

constexpr int kDnMaxStages = 10;
constexpr int kDnProducerWarp = 0, kDnMmaWarp = 1, kDnFirstEpilogueWarp = 4;
constexpr uint32_t kDnXBytes = 128 * 128;   // a CTA's 128 tokens x 64 elements
constexpr uint32_t kDnRingBytes = 6 * 2 * kDnXBytes;  // six stages with half of 256 features beside the tokens, more of narrower ones
constexpr uint32_t kDnBoxBytes = 32 * 64;   // an epilogue warp's 32 tokens x 32 features

struct DenseParams {
  const __half* bias;
  unsigned* status;
  int M, N, nkb;
  // Units: tiles of 256 tokens x 256 features, features fastest, as long as every CTA pair has one (`whole` of them); what is left
  // in tiles of `w` granules of 32 features: `head` of them from granule g0 of token tile tt0, then `per_tt` per token tile.
  int n_ftiles, whole, n_units, tt0, g0, head, per_tt, w;
  int stages;
  unsigned stage_bytes;
};

// unit u -> token tile, first feature, number of features (a multiple of 32)
__device__ __forceinline__ void dense_unit(const DenseParams& p, int u, int& tt, int& f0, int& n) {
  if (u < p.whole) {
    tt = u / p.n_ftiles;
    f0 = (u - tt * p.n_ftiles) * 256;
    n = min(256, p.N - f0);
    return;
  }
  u -= p.whole;
  int g;
  if (u < p.head) {
    tt = p.tt0;
    g = p.g0 + u * p.w;
  } else {
    u -= p.head;
    const int t = u / p.per_tt;
    tt = p.tt0 + (p.head ? 1 : 0) + t;
    g = (u - t * p.per_tt) * p.w;
  }
  f0 = g * 32;
  n = min(p.w * 32, p.N - f0);
}

// ---- packed weights -> 16-bit weights, (N, K) row-major ------------------------------------------------------------
// A thread takes 32-bit words of packed weights (8 or 16 outputs, one or two 16-byte stores; a warp reads 128 and writes 512 or
// 1024 contiguous bytes); words, scales and zeros are constants and are fetched ahead of the stream dependency, the stores wait,
// because a kernel before on the stream may still use that memory.
constexpr int kUnpackWords = 4;
template <int BITS, bool BF16>
__global__ void __launch_bounds__(256)
unpack_kernel(const uint32_t* __restrict__ w, const __half* __restrict__ scales, const __half* __restrict__ zeros, uint4* __restrict__ out,
              unsigned n_words, unsigned words_per_row, unsigned words_per_group, unsigned groups_per_row) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int PW = 32 / BITS / 2;  // output pairs per word
  const unsigned i0 = blockIdx.x * (256u * kUnpackWords) + threadIdx.x;
  uint32_t q[kUnpackWords], s2[kUnpackWords], z2[kUnpackWords];
#pragma unroll
  for (int j = 0; j < kUnpackWords; ++j) {
    const unsigned i = i0 + j * 256u;
    q[j] = s2[j] = z2[j] = 0u;
    if (i < n_words) {
      const unsigned row = i / words_per_row, g = row * groups_per_row + (i - row * words_per_row) / words_per_group;
      q[j] = __ldg(w + i);
      const unsigned short s = __ldg(reinterpret_cast<const unsigned short*>(scales) + g);
      const unsigned short z = __ldg(reinterpret_cast<const unsigned short*>(zeros) + g);
      if (BF16) {
        s2[j] = __float_as_uint(__half2float(__ushort_as_half(s)));
        z2[j] = __float_as_uint(__half2float(__ushort_as_half(z)));
      } else {
        s2[j] = uint32_t(s) * 0x10001u;
        z2[j] = uint32_t(z) * 0x10001u;
      }
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
  for (int j = 0; j < kUnpackWords; ++j) {
    const unsigned i = i0 + j * 256u;
    if (i >= n_words) break;
    uint32_t o[PW];
    dequant_word<BITS, BF16>(q[j], s2[j], z2[j], o);
#pragma unroll
    for (int c = 0; c < PW / 4; ++c) out[size_t(i) * (PW / 4) + c] = make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
  }
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, int c0, int c1, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(m)),
               "r"(c0), "r"(c1), "r"(src)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(LEFT) : "memory");
}

// Groups of four epilogue warps.  An erf per output keeps a tile's epilogue (two groups: about 13 000 clocks) longer than the main loop
// of 1280 inputs (10 200): four groups measured 6 % faster over 2 000 to 16 512 tokens there, and nothing without GELU or from 2048 on.
template <bool GELU>
constexpr int kDnGroups = GELU ? 4 : 2;

// y[M, N] = x[M, K] . w[N, K]^T + bias, then GELU and / or the residual
template <bool BF16, bool GELU, bool RES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(128 + 128 * kDnGroups<GELU>, 1)
gemm_dense_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw, const __grid_constant__ CUtensorMap tmwt,
                  const __grid_constant__ CUtensorMap tmy, const __grid_constant__ CUtensorMap tmr, const DenseParams p) {
  constexpr int kGroups = kDnGroups<GELU>, kDnEpilogueWarps = 4 * kGroups, kBoxes = 4 / kGroups;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kDnMaxStages + 4 + kBoxes * kDnEpilogueWarps];
  __shared__ __align__(16) uint16_t bias_s[kDnEpilogueWarps][32];  // halves
  __shared__ uint32_t tmem_slot;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t boxes = base + kDnRingBytes;  // kBoxes per epilogue warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = tc::cluster_ctarank();
  const int cluster = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  const uint32_t bar0 = tc::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto free_bar = [&](int s) { return bar0 + 8u * (kDnMaxStages + s); };
  auto accf_bar = [&](uint32_t b) { return bar0 + 8u * (2 * kDnMaxStages + b); };
  auto acce_bar = [&](uint32_t b) { return bar0 + 8u * (2 * kDnMaxStages + 2 + b); };
  auto res_bar = [&](int i) { return bar0 + 8u * (2 * kDnMaxStages + 4 + i); };

  {
    const int i = threadIdx.x;
    if (i < 2 * kDnMaxStages + 4 + kBoxes * kDnEpilogueWarps) {
      // a drained accumulator: the epilogue warps of both CTAs
      tc::mbar_init(bar0 + 8u * i, (i >= 2 * kDnMaxStages + 2 && i < 2 * kDnMaxStages + 4) ? 2 * kDnEpilogueWarps : 1);
      tc::fence_barrier_init();
      tc::fence_proxy_async_smem();
    }
    if (threadIdx.x == 32 * kDnProducerWarp) {
      tc::prefetch_tmap(&tmx);
      tc::prefetch_tmap(&tmw);
    }
    if (threadIdx.x == 32 * kDnFirstEpilogueWarp) tc::prefetch_tmap(&tmy);
  }
  if (warp == kDnMmaWarp) {
    tc::tmem_alloc_pair(tc::smem_u32(&tmem_slot), 512);
    tc::tmem_relinquish_pair();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync();  // the peer's barriers are initialised before anything arrives on them
  tc::fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);

  int tt, f0, n;  // of the current unit: every role walks the list cluster, cluster + nclusters, ...

  if (warp == kDnProducerWarp) {
    if (lane == 0) {
      const uint32_t full0 = tc::mapa(full_bar(0), 0);  // CTA 0's full barriers, as seen from here
      asm volatile("griddepcontrol.wait;" ::: "memory");
      uint32_t ph = 0;
      int s = 0;
      bool ok = true;
      for (int unit = cluster; unit < p.n_units && ok; unit += nclusters) {
        dense_unit(p, unit, tt, f0, n);
        const int row_x = tt * 256 + int(rank) * 128, row_w = f0 + int(rank) * (n / 2);
        // a box per unit width; the last unit of a token tile may need fewer rows than its box brings
        const CUtensorMap* const map_w = unit < p.whole ? &tmw : &tmwt;
        const uint32_t bytes = 2u * kDnXBytes + (unit < p.whole ? 256u : uint32_t(p.w) * 32u) * 128u;
        for (int kb = 0; kb < p.nkb; ++kb) {
          if (!tc::mbar_wait(free_bar(s), ph ^ 1u, p.status, 31)) { ok = false; break; }
          if (rank == 0) tc::mbar_arrive_expect_tx(full_bar(s), bytes);
          const uint32_t dst = base + uint32_t(s) * p.stage_bytes;
          tc::tma_load_2d_pair(dst, &tmx, kb * 64, row_x, full0 + 8u * s);
          tc::tma_load_2d_pair(dst + kDnXBytes, map_w, kb * 64, row_w, full0 + 8u * s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == kDnMmaWarp) {
    // whole warp, tcgen05 instructions in one elected lane; the next stage's barrier is tested ahead of this stage's MMAs
    if (rank == 0) {
      const uint32_t el = tc::elect_one() ? 1u : 0u;
      uint32_t ph = 0, ucount = 0, ready = 0;
      int s = 0;
      bool ok = true;
      for (int unit = cluster; unit < p.n_units && ok; unit += nclusters, ++ucount) {
        dense_unit(p, unit, tt, f0, n);
        const uint32_t buf = ucount & 1u, d_tmem = tmem_base + buf * 256u;
        const uint32_t idesc = tc::instr_desc(1u, BF16 ? 1u : 0u, 256u, uint32_t(n));
        ok = tc::mbar_wait_spin(acce_bar(buf), ((ucount >> 1) & 1u) ^ 1u, p.status, 32);
        tc::fence_after_sync();
        for (int kb = 0; kb < p.nkb && ok; ++kb) {
          if (!ready) {
            ok = tc::mbar_wait_spin(full_bar(s), ph, p.status, 33);
            if (!ok) break;
          }
          tc::fence_after_sync();
          int sn = s + 1;
          uint32_t phn = ph;
          if (sn == p.stages) { sn = 0; phn ^= 1u; }
          const uint32_t a = base + uint32_t(s) * p.stage_bytes;
          ready = tc::mma4_commit_probe_pair(el, d_tmem, tc::smem_desc_sw128(a), tc::smem_desc_sw128(a + kDnXBytes), idesc, uint32_t(kb != 0),
                                             free_bar(s), full_bar(sn), full_bar(sn), phn);
          if (el && kb + 1 == p.nkb) tc::mma_commit_pair(accf_bar(buf), 3);
          s = sn;
          ph = phn;
        }
      }
    }
  } else if (warp >= kDnFirstEpilogueWarp) {
    const int e = warp - kDnFirstEpilogueWarp, qd = warp & 3, group = e >> 2;
    const uint32_t box0 = boxes + uint32_t(e * kBoxes) * kDnBoxBytes;
    // a lane's row of a box: 64 bytes, its 16-byte chunk c at position c ^ (row / 2 % 4) (64-byte swizzle)
    const uint32_t row_off = uint32_t(lane) * 64u, row_xor = uint32_t((lane >> 1) & 3);
    uint32_t ucount = 0, nbox = 0, rph = 0;  // boxes used so far; bit b of rph: parity of box b's residual barrier
    if (RES) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int unit = cluster; unit < p.n_units; unit += nclusters, ++ucount) {
      dense_unit(p, unit, tt, f0, n);
      const bool last = unit + nclusters >= p.n_units;
      const uint32_t buf = ucount & 1u;
      const int row0 = tt * 256 + int(rank) * 128 + qd * 32;
      const int nch = n / 32;
      const bool rows = row0 < p.M;
      // the residual of this warp's chunk ch into the box it will use; the box's last store has been read
      auto fetch_residual = [&](int ch, uint32_t b) {
        if (RES && lane == 0 && rows && ch < nch) {
          tc::mbar_arrive_expect_tx(res_bar(kBoxes * e + int(b)), kDnBoxBytes);
          tc::tma_load_2d(box0 + b * kDnBoxBytes, &tmr, f0 + ch * 32, row0, res_bar(kBoxes * e + int(b)));
        }
      };
      if (RES) {
        if (lane == 0) bulk_wait_read<0>();
        __syncwarp();
        fetch_residual(group, nbox % kBoxes);
      }
      if (!__all_sync(0xffffffffu, tc::mbar_wait(accf_bar(buf), (ucount >> 1) & 1u, p.status, 34))) break;
      __syncwarp();
      tc::fence_after_sync();
      const uint32_t taddr = tmem_base + (uint32_t(qd * 32) << 16) + buf * 256u;
      // "this warp's part of the accumulator is in registers": not for the last unit, nobody waits for that, and an arrival in
      // flight must not land in shared memory of the next kernel's block
      auto drained = [&]() {
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0 && !last) {
          if (rank == 0) tc::mbar_arrive(acce_bar(buf));
          else tc::mbar_arrive_cluster_relaxed(tc::mapa(acce_bar(buf), 0));
        }
      };
      if (group >= nch) drained();
      bool ok = true;
      for (int ch = group; ch < nch; ch += kGroups, ++nbox) {
        const uint32_t b = nbox % kBoxes, box = box0 + b * kDnBoxBytes;
        uint32_t r[32];
        tc::tmem_ld_32x32(taddr + ch * 32, r);
        bias_s[e][lane] = p.bias ? __ldg(reinterpret_cast<const unsigned short*>(p.bias) + f0 + ch * 32 + lane) : uint16_t(0);
        tc::tmem_ld_wait();
        if (ch + kGroups >= nch) drained();
        if (RES) {
          // the other box: its store (if any) has been read, then the next chunk's residual goes there
          if (kBoxes > 1) {
            if (lane == 0) bulk_wait_read<0>();
            __syncwarp();
            fetch_residual(ch + kGroups, b ^ 1u);
          }
          if (rows) {
            ok = __all_sync(0xffffffffu, tc::mbar_wait(res_bar(kBoxes * e + int(b)), (rph >> b) & 1u, p.status, 35));
            rph ^= 1u << b;
            if (!ok) break;
          }
        } else {
          if (lane == 0) bulk_wait_read<kBoxes - 1>();
        }
        __syncwarp();
        if (rows) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 bq = *reinterpret_cast<const uint4*>(&bias_s[e][c * 8]);
            const float2 b01 = __half22float2(u32_as_h2(bq.x)), b23 = __half22float2(u32_as_h2(bq.y)), b45 = __half22float2(u32_as_h2(bq.z)),
                         b67 = __half22float2(u32_as_h2(bq.w));
            const float bv[8] = {b01.x, b01.y, b23.x, b23.y, b45.x, b45.y, b67.x, b67.y};
            const uint32_t addr = box + row_off + ((uint32_t(c) ^ row_xor) << 4);
            uint32_t rv[4] = {0u, 0u, 0u, 0u};
            if (RES) {
              const uint4 t = tc::ld_shared_v4(addr);
              rv[0] = t.x; rv[1] = t.y; rv[2] = t.z; rv[3] = t.w;
            }
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint16_t h[2];
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const uint16_t v = float_to_out16(__uint_as_float(r[c * 8 + 2 * j + k]) + bv[2 * j + k], BF16);
                h[k] = (GELU || RES) ? epilogue16(v, GELU ? kActGelu : kActNone, RES, uint16_t(rv[j] >> (16 * k)), BF16) : v;
              }
              o[j] = uint32_t(h[0]) | (uint32_t(h[1]) << 16);
            }
            tc::st_shared_v4(addr, o[0], o[1], o[2], o[3]);
          }
          tc::fence_proxy_async_smem();
        }
        __syncwarp();
        if (rows && lane == 0) {
          tma_store_2d(&tmy, f0 + ch * 32, row0, box);
          bulk_commit();
        }
        if (RES && kBoxes == 1 && ch + kGroups < nch) {
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
          fetch_residual(ch + kGroups, 0u);
        }
      }
      if (!ok) break;
    }
    if (lane == 0) bulk_wait_read<0>();  // shared memory is given back only when the stores have been read
  }

  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync_relaxed();
  if (warp == kDnMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc_pair(tmem_base, 512);
  }
}

template <typename... KArgs, typename... Args>
int launch(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t stream, Args... args) {
  if (smem)
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 0 : 1;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, KArgs(args)...));
  return ASRQ_OK;
}

// Clocks of a K block of 64 elements for a tile of w granules of 32 features: the MMAs, or the operands from L2, of which the
// ring holds 192 KB for a trip of 1.4 us (1280 and 6144 inputs, 300 to 2000 tokens: 0.23-0.25 us a block whatever its width, with six stages)
double block_clocks(int w) { return std::max(64.0 * w, (16384.0 + 2048.0 * w) / 70.0); }

// Whole rounds of 256 x 256 tiles, and the width of the tiles that share out the rest.  Returns the clocks per K block over all rounds.
double pick_units(DenseParams* p, int64_t M, int64_t N, int max_clusters) {
  const int64_t n_tt = (M + 255) / 256, n_ft = (N + 255) / 256, granules = N / 32;
  const int64_t rounds = n_tt * n_ft / max_clusters, whole = rounds * max_clusters;
  double best = 1e30;
  const int64_t tt0 = whole / n_ft, g0 = whole % n_ft * 8;
  for (int w = 8; w >= 1; --w) {
    const int64_t head = g0 ? (granules - g0 + w - 1) / w : 0, per_tt = (granules + w - 1) / w;
    const int64_t tail = head + (n_tt - tt0 - (g0 ? 1 : 0)) * per_tt;
    const double cost = double((tail + max_clusters - 1) / max_clusters) * block_clocks(w);
    if (cost >= best) continue;
    best = cost;
    if (p) {
      p->n_ftiles = int(n_ft);
      p->whole = int(whole);
      p->n_units = int(whole + tail);
      p->tt0 = int(tt0);
      p->g0 = int(g0);
      p->head = int(head);
      p->per_tt = int(per_tt);
      p->w = w;
    }
  }
  return best + double(rounds) * block_clocks(8);
}

}  // namespace

// The 16-bit weights.
size_t gemm_a16_dense_scratch_bytes(int64_t N, int64_t K) { return size_t(2) * size_t(N) * size_t(K); }

// Estimated time in us, epilogue included: unpacking and two launches, and the rounds' K blocks at the clock that the power limit
// leaves (1.8 GHz for a call of 20 us, 1.3 from about 70 us on).  Measured, W4, fp16, us: 21.1 for 1500 tokens of 1280 -> 5120, 33.7 for
// 12 000 of 1280 -> 1280, 65.6 for 6 000 of 5120 -> 1280, 193 for 16 512 of 2048 -> 4096, 424 for 48 000 of 1280 -> 5120.
double gemm_a16_dense_estimate(int64_t M, int64_t N, int64_t K, int sm_count, bool gelu, bool residual) {
  const double clocks = pick_units(nullptr, M, N, sm_count / 2) * double(K / 64);
  const double mn = double(M) * double(N);
  return 9.0 + 0.4e-6 * double(N) * double(K) + clocks / 1800.0 * (1.0 + std::min(0.4, std::max(0.0, clocks - 2e4) / 1.5e5)) +
         (gelu ? (4.0 + 0.5e-6 * mn) * std::min(1.0, 1280.0 / double(K)) : 0.0) + (residual ? 3.0 : 0.0);
}

bool gemm_a16_dense_supports(int64_t M, int64_t N, int64_t K, int group_size) {
  return M >= 1 && M <= (1ll << 30) && N % 128 == 0 && K % 64 == 0 && N * K <= (1ll << 30) && (M + 255) / 256 * (N / 32) < (1ll << 31) - 1024 && group_size > 0 && group_size % 64 == 0 && K % group_size == 0;
}

int gemm_a16_dense(int bits, const void* x, const uint8_t* w, const void* scales, const void* zeros, const void* bias, void* y, int64_t M,
                   int64_t N, int64_t K, int group_size, int dtype, void* workspace, void* scratch, size_t scratch_bytes, int sm_count,
                   cudaStream_t stream, const Epilogue& ep) {
  if (!gemm_a16_dense_supports(M, N, K, group_size))
    return fail(ASRQ_ERR_SHAPE, "w%da16 gemm (dense): unsupported shape N=%lld K=%lld g=%d", bits, (long long)N, (long long)K, group_size);
  if (!scratch || scratch_bytes < gemm_a16_dense_scratch_bytes(N, K)) return fail(ASRQ_ERR_WORKSPACE, "w%da16 gemm (dense): scratch too small", bits);
  if (!aligned16(x) || !aligned16(w) || !aligned16(y) || !aligned16(ep.residual) || !aligned16(scratch))
    return fail(ASRQ_ERR_ALIGN, "w%da16 gemm (dense): x, w, y, residual and scratch must be 16-byte aligned", bits);
  const bool bf16 = dtype == ASRQ_BF16;

  const unsigned words_per_row = unsigned(K * bits / 32), n_words = unsigned(N) * words_per_row;
  const int blocks = int((n_words + 256u * kUnpackWords - 1) / (256u * kUnpackWords));
  auto unpack = [&](auto kern) {
    return launch(kern, blocks, 256, 0, stream, reinterpret_cast<const uint32_t*>(w), static_cast<const __half*>(scales),
                  static_cast<const __half*>(zeros), static_cast<uint4*>(scratch), n_words, words_per_row, unsigned(group_size * bits / 32),
                  unsigned(K / group_size));
  };
  int rc = bits == 4 ? (bf16 ? unpack(unpack_kernel<4, true>) : unpack(unpack_kernel<4, false>))
                     : (bf16 ? unpack(unpack_kernel<2, true>) : unpack(unpack_kernel<2, false>));
  if (rc) return rc;

  const int max_clusters = sm_count / 2;
  DenseParams p;
  p.bias = static_cast<const __half*>(bias);
  p.status = static_cast<unsigned*>(workspace);
  p.M = int(M);
  p.N = int(N);
  p.nkb = int(K / 64);
  pick_units(&p, M, N, max_clusters);
  p.stage_bytes = kDnXBytes + (p.whole ? 8u : unsigned(p.w)) * 2048u;
  p.stages = int(std::min<unsigned>(kDnMaxStages, kDnRingBytes / p.stage_bytes));
  CUtensorMap tmx, tmw, tmwt, tmy, tmr;
  if ((rc = make_tmap_2d(&tmx, x, 2, bf16, uint64_t(K), uint64_t(M), 64, 128, kSwizzle128))) return rc;
  if ((rc = make_tmap_2d(&tmw, scratch, 2, bf16, uint64_t(K), uint64_t(N), 64, 128, kSwizzle128))) return rc;
  if ((rc = make_tmap_2d(&tmwt, scratch, 2, bf16, uint64_t(K), uint64_t(N), 64, uint32_t(p.w * 16), kSwizzle128))) return rc;
  if ((rc = make_tmap_2d(&tmy, y, 2, bf16, uint64_t(N), uint64_t(M), 32, 32, kSwizzle64))) return rc;
  tmr = tmy;
  if (ep.residual && (rc = make_tmap_2d(&tmr, ep.residual, 2, bf16, uint64_t(N), uint64_t(M), 32, 32, kSwizzle64))) return rc;
  const size_t smem = 1024 + kDnRingBytes + size_t(16) * kDnBoxBytes;
  const int clusters = std::min(p.n_units, max_clusters);
  const bool gelu = ep.act == kActGelu, res = ep.residual != nullptr;
  auto gemm = [&](auto kern) { return launch(kern, 2 * clusters, 128 + 128 * (gelu ? kDnGroups<true> : kDnGroups<false>), smem, stream, tmx, tmw, tmwt, tmy, tmr, p); };
  if (bf16) {
    if (res) return gelu ? gemm(gemm_dense_kernel<true, true, true>) : gemm(gemm_dense_kernel<true, false, true>);
    return gelu ? gemm(gemm_dense_kernel<true, true, false>) : gemm(gemm_dense_kernel<true, false, false>);
  }
  if (res) return gelu ? gemm(gemm_dense_kernel<false, true, true>) : gemm(gemm_dense_kernel<false, false, true>);
  return gelu ? gemm(gemm_dense_kernel<false, true, false>) : gemm(gemm_dense_kernel<false, false, false>);
}

}  // namespace asrq
