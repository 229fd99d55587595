// Decode batches and short prompts on the tensor cores: y[M,N] = x[M,K] . dequant(W)[N,K]^T (+ bias), 17 <= M <= 2048, in one wave.
//
// At these token counts the mma.sync decode kernel is bound by the legacy MMA pipe (one m16n8k16 per ~13
// clocks per scheduler, one per 8 tokens per 256 codes), and the persistent prefill kernel by its fixed
// costs (set-up, first TMA and first dequantisation pass before the first MMA, an epilogue nothing
// overlaps): 10-15 us for a 1-3 MB layer either way.  This kernel is built for a CHAIN of such layers:
//
//   * a block owns ONE work item -- a tile of 128 features x BT tokens and a part of K.  Its activation tiles and packed
//     weights pass through a ring of stages in shared memory, which for decode batches holds all of them at once;
//   * weights are unpacked into TENSOR MEMORY, as the MMA's A operand (tcgen05.st; a lane is a weight row, 32 columns a K block of 64;
//     three or six such slots beside the accumulator).  Through shared memory a K block cost 128 clocks of stores, 128 of the
//     MMA's reads and a proxy fence beside the 190 that packed weights and activations take: shared memory was busy for three
//     quarters of the block's 620 clocks;
//   * it triggers its dependents as its first instruction, and up to 64 tokens two blocks share an SM where the plan's shared memory
//     allows (up to 112 KB).  Packed weights are fetched by TMA and the first three or six K blocks are dequantised BEFORE
//     griddepcontrol.wait: weights do not depend on the kernel before, so the next launch's weight traffic and unpacking run under
//     this launch's tail where it has an SM by then;
//   * after the wait only the activation tiles (tokens as the MMA's N dimension: 32 to 256 TMEM columns)
//     are fetched, as many as there are stages at once; tcgen05.mma kind::f16 128 x BT x 16, fp32 accumulator in tensor memory;
//   * the K parts of a tile are a thread-block cluster and meet in distributed shared memory: every block leaves its
//     fp32 part in its own shared memory (over the stages, whose MMAs are done), and after one cluster barrier each
//     adds its share of the tokens over all parts in part order, with all of its threads, adds the bias, converts
//     and stores.  Through the workspace (partial tiles, a counter per tile, the last block adding) the same step
//     cost a release to memory, an atomic and two to four L2 round trips of one block while the others were done.
//
// Roles (14 warps): warp 0 TMA producer, warp 1 MMA issuer (owns the tensor-memory allocation), warps
// 2-13 three dequant groups of 128 threads (one weight row per thread, group d takes K blocks d, d+3, ...); the first group
// (warps 2-5, one per TMEM lane quadrant) then runs the epilogue.  No TMA multicast.  Every wait is bounded.
//
// Bound: the chain's latencies and, where a block has many K blocks, the dequant groups' own (0.27 us a block; 0.23 with the
// arithmetic left out).  Chains of launches, W4, unpacking through shared memory -> this form, us at 32 / 64 / 128 / 259 tokens:
// 1280 -> 1280 4.3 / 4.6 / 5.9 / 6.6 -> 3.9 / 4.1 / 5.5 / 6.4; 1280 -> 5120 6.1 / 6.8 / 8.1 / 11.8 -> 5.0 / 6.0 / 8.0 / 11.0; 2048 -> 4096 6.7 / 7.5 /
// 8.7 / 12.6 -> 5.3 / 6.6 / 8.7 / 11.3; 2048 -> 12288 15.3 / 16.1 / 17.9 -> 12.9 / 14.0 / 15.6; 6144 -> 2048 10.5 / 11.4 / 12.4 / 16.5 -> 8.5 / 10.0 / 12.1 /
// 15.7; bf16 2048 -> 4096 at 64 / 80 / 96 / 128 tokens 7.6 / 7.9 / 8.05 / 8.8 -> 6.6 / 7.85 / 8.0 / 8.7.  More slots than the MMAs' round trip needs changed nothing.
//
// Prompts of some hundred tokens: the persistent kernels give a tile the whole of K, and with few tiles most SMs idle (1280 x 5120
// at 260 to 1500 tokens: 31 us on 20 to 60 of them).  Here K is cut so that one wave fills the chip.
#include <algorithm>
#include <atomic>

#include "dequant.cuh"
#include "tcgen05.cuh"

namespace asrq {

int ensure_dynamic_smem(const void* kernel, size_t bytes);

namespace {

constexpr int kSkWarps = 14;
constexpr int kSkThreads = 32 * kSkWarps;
constexpr int kSkMaxStages = 16;                // K blocks of 64 in shared memory at once
constexpr int kSkMaxSplit = 8;
constexpr int kSkMaxSlots = 6;
constexpr uint32_t kSkSlotCols = 32;            // a dequantised A slot in tensor memory: 128 lanes x 64 16-bit elements
constexpr int kSkMaxM = 2048;
constexpr size_t kSkMaxSmem = 226 * 1024;
constexpr size_t kSkTwoPerSm = 112 * 1024;      // two blocks share an SM
constexpr uint32_t kSkWSlot = 4096;             // packed weights of one K block (<= 128 x 32 B)

// Columns of tensor memory to allocate (a power of two).  256 at most up to 128 tokens: two blocks share an SM's 512.
__host__ __device__ constexpr uint32_t skinny_tmem_cols(int bt, int slots) {
  const uint32_t need = uint32_t(bt) + uint32_t(slots) * kSkSlotCols;
  return need <= 128 ? 128u : (need <= 256 ? 256u : 512u);
}

struct SkinnyParams {
  const __half* scales;
  const __half* zeros;
  const __half* bias;
  const uint16_t* residual;  // fused epilogue: y = residual + layer output (NULL: none)
  int act;                   // fused epilogue: activation on the layer output (kActNone / kActGelu)
  uint16_t* y;
  unsigned* status;
  int M, N, K, group_size, groups_per_row, bt, n_tt, ksplit, nkb, stages;
  int slots;  // A slots in tensor memory, a multiple of three: K block kb is in slot kb % slots
  unsigned long long* trace;  // builds with -DASRQ_TRACE: 8 globaltimer marks per block, NULL otherwise
};

#ifdef ASRQ_TRACE
#define SK_MARK(i)                                                                   \
  do {                                                                               \
    if (p.trace) {                                                                   \
      unsigned long long t__;                                                        \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t__)::"memory");              \
      p.trace[size_t(blockIdx.x) * 8 + (i)] = t__;                                   \
    }                                                                                \
  } while (0)
#else
#define SK_MARK(i) do { } while (0)
#endif

// RING: parts longer than the ring of stages.  Without it every K block has a stage of its own: one barrier for all activation
// tiles and nothing to count (with both forms in one kernel a launch of 32 tokens took 0.5 to 1 us more).
template <int BITS, bool BF16, bool RING>
__global__ void __launch_bounds__(kSkThreads, 2)
gemm_a16_skinny_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw,
                       const SkinnyParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * kSkMaxStages + 1 + 2 * kSkMaxSlots];
  __shared__ uint32_t tmem_slot;
  // the next launch on the stream may start its own set-up, weight fetch and first dequantisation now
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (threadIdx.x == 0) SK_MARK(0);
  const uint32_t raw_addr = tc::smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work item: feature tile ft, token tile tt, K part ks (parts of a tile on neighbouring blocks: a cluster)
  const int ks = blockIdx.x % p.ksplit, tile = blockIdx.x / p.ksplit, tt = tile % p.n_tt, ft = tile / p.n_tt;
  const int kb0 = ks * p.nkb / p.ksplit, kb1 = (ks + 1) * p.nkb / p.ksplit, kbn = kb1 - kb0, nst = p.stages;
  const uint32_t xbytes = uint32_t(p.bt) * 128u;
  // [activation tile x stages] [packed weights x stages]
  const uint32_t x_base = 0, w_base = uint32_t(nst) * xbytes;
  constexpr uint32_t wbytes = 128u * 8u * BITS;
  const uint32_t bar0 = tc::smem_u32(bars);
  auto w_bar = [&](int st) { return bar0 + 8u * st; };
  auto x_bar = [&](int st) { return bar0 + 8u * (kSkMaxStages + st); };
  auto sfree_bar = [&](int st) { return bar0 + 8u * (2 * kSkMaxStages + st); };  // the stage's MMAs are done
  const uint32_t accf_bar = bar0 + 8u * (3 * kSkMaxStages);
  auto deq_bar = [&](int a) { return accf_bar + 8u + 8u * a; };
  auto afree_bar = [&](int a) { return accf_bar + 8u + 8u * (kSkMaxSlots + a); };
  // tensor memory: [accumulator, bt columns] [A slots]
  const uint32_t a_col = uint32_t(p.bt), tmem_cols = skinny_tmem_cols(p.bt, p.slots);

  // The bias of the four features this thread stores (the same in each of its steps): a constant, and fetched here a first touch
  // of memory that the last step would otherwise wait for.
  uint2 bias4 = make_uint2(0u, 0u);
  if (p.bias) bias4 = __ldg(reinterpret_cast<const uint2*>(p.bias + ft * 128 + lane * 4));

  if (threadIdx.x == 0) {
    for (int st = 0; st < nst; ++st) {
      tc::mbar_init(w_bar(st), 1);
      if (st && !RING) continue;
      tc::mbar_init(x_bar(st), 1);
      tc::mbar_init(sfree_bar(st), 1);
    }
    tc::mbar_init(accf_bar, 1);
    for (int a = 0; a < p.slots; ++a) {
      tc::mbar_init(deq_bar(a), 4);  // the four warps of the group
      tc::mbar_init(afree_bar(a), 1);
    }
    tc::fence_barrier_init();
    tc::fence_proxy_async_smem();
    tc::prefetch_tmap(&tmx);
    tc::prefetch_tmap(&tmw);
  }
  if (warp == 1) {
    tc::tmem_alloc(tc::smem_u32(&tmem_slot), tmem_cols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
  if (threadIdx.x == 0) SK_MARK(1);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      auto fetch_w = [&](int kb, int st) {
        tc::mbar_arrive_expect_tx(w_bar(st), wbytes);
        tc::tma_load_2d(base + w_base + st * kSkWSlot, &tmw, (kb0 + kb) * 8 * BITS, ft * 128, w_bar(st));
      };
      auto fetch_x = [&](int kb, int st) {
        if (RING) tc::mbar_arrive_expect_tx(x_bar(st), xbytes);
        tc::tma_load_2d(base + x_base + st * xbytes, &tmx, (kb0 + kb) * 64, tt * p.bt, x_bar(RING ? st : 0));
      };
      for (int kb = 0; kb < kbn && kb < nst; ++kb) fetch_w(kb, kb);  // constants: ahead of the stream dependency
      SK_MARK(2);
      // activations belong to this kernel only once its predecessor on the stream is complete
      asm volatile("griddepcontrol.wait;" ::: "memory");
      SK_MARK(3);
      if (!RING) tc::mbar_arrive_expect_tx(x_bar(0), uint32_t(kbn) * xbytes);
      for (int kb = 0; kb < kbn && kb < nst; ++kb) fetch_x(kb, kb);
      if constexpr (RING) {
        int st = 0;
        uint32_t ph = 0;
        for (int kb = nst; kb < kbn; ++kb) {
          if (!tc::mbar_wait(sfree_bar(st), ph, p.status, 36)) break;
          fetch_w(kb, st);
          fetch_x(kb, st);
          if (++st == nst) { st = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The warp's own latency is part of every K block's chain: the next block's barriers are tested in the stream of this block's MMAs
    // (see mma4_ts_commit_probe), and waited for only where that found one incomplete.
    const uint32_t el = tc::elect_one() ? 1u : 0u;
    const uint32_t idesc = tc::instr_desc(1u, BF16 ? 1u : 0u, 128u, uint32_t(p.bt));
    int st = 0, a = 0;
    uint32_t ph = 0, aph = 0, ready = 0;
    bool ok = tc::mbar_wait_spin(x_bar(0), 0u, p.status, 31);
    if (lane == 0) SK_MARK(4);
    for (int kb = 0; kb < kbn && ok; ++kb) {
      if (!ready) {
        if (RING && kb) ok = tc::mbar_wait_spin(x_bar(st), ph, p.status, 31);
        ok = ok && tc::mbar_wait_spin(deq_bar(a), aph, p.status, 32);
        if (!ok) break;
      }
      tc::fence_after_sync();
      int st_n = st + 1, a_n = a + 1;
      uint32_t ph_n = ph, aph_n = aph;
      if (st_n == nst && RING) { st_n = 0; ph_n ^= 1u; }
      if (a_n == p.slots) { a_n = 0; aph_n ^= 1u; }
      ready = tc::mma4_ts_commit_probe(el, tmem_base, tmem_base + a_col + uint32_t(a) * kSkSlotCols, tc::smem_desc_sw128(base + x_base + st * xbytes), idesc,
                                       uint32_t(kb != 0), afree_bar(a), RING && kb + nst < kbn, sfree_bar(RING ? st : 0), deq_bar(a_n), aph_n,
                                       x_bar(RING ? st_n : 0), RING ? ph_n : 0u);
      if (el && kb + 1 == kbn) tc::mma_commit(accf_bar);
      st = st_n; a = a_n; ph = ph_n; aph = aph_n;
    }
    if (lane == 0) SK_MARK(5);
  } else {
    // ------------------------------ dequant (three groups) ------------------------------
    const int dgroup = (warp - 2) >> 2;
    const int t = (warp & 3) * 32 + lane;  // weight row inside the tile = lane of tensor memory (a warp reaches quadrant warp % 4)
    const uint32_t a_lane = tmem_base + (uint32_t((warp & 3) * 32) << 16) + a_col;
    const int kbpg = p.group_size / 64;
    bool ok = true;
    auto load_sz = [&](int kb) {
      const size_t idx = (size_t(ft) * 128 + t) * p.groups_per_row + (kb0 + kb) / kbpg;
      return uint32_t(__half_as_ushort(__ldg(p.scales + idx))) | (uint32_t(__half_as_ushort(__ldg(p.zeros + idx))) << 16);
    };
    uint32_t sz_next = dgroup < kbn ? load_sz(dgroup) : 0u;  // a block of this group ahead
    int st = dgroup, a = dgroup;  // a ring that goes round has at least four stages
    uint32_t ph = 0, aph = 1;     // aph: parity of the slot's last release; the first pass waits for none
    for (int kb = dgroup; kb < kbn && ok; kb += 3) {
      const uint32_t sz = sz_next;
      if (kb + 3 < kbn) sz_next = load_sz(kb + 3);
      const __half sh = __ushort_as_half(uint16_t(sz & 0xffffu)), zh = __ushort_as_half(uint16_t(sz >> 16));
      uint32_t s2, z2;
      if (BF16) {
        s2 = __float_as_uint(__half2float(sh));
        z2 = __float_as_uint(__half2float(zh));
      } else {
        s2 = h2_as_u32(__half2half2(sh));
        z2 = h2_as_u32(__half2half2(zh));
      }
      bool okw = tc::mbar_wait(w_bar(st), ph, p.status, 34);
      // the slot's previous K block must have been consumed by its MMAs
      if (kb >= p.slots) okw = okw && tc::mbar_wait(afree_bar(a), aph, p.status, 33);
      // one decision for the warp, and its lanes together: the store to tensor memory is a warp-wide instruction
      ok = __all_sync(0xffffffffu, okw);
      if (!ok) break;
      __syncwarp();
      const uint4* wp = reinterpret_cast<const uint4*>(smem + w_base + st * kSkWSlot + t * (8 * BITS));
      constexpr int NV = BITS / 2;  // 16-byte vectors of packed weights per row per K block
      uint32_t o[32];               // the row's 64 elements in pairs, in k order: one 32-bit column of tensor memory each
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const uint4 qv = wp[v];
        const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w};
        constexpr int PW = 32 / BITS / 2;  // output pairs per word: 4 or 8
#pragma unroll
        for (int j = 0; j < 4; ++j) dequant_word<BITS, BF16>(qw[j], s2, z2, o + (v * 4 + j) * PW);
      }
      if (kb >= p.slots) tc::fence_after_sync();
      tc::tmem_st_32x32(a_lane + uint32_t(a) * kSkSlotCols, o);
      tc::tmem_st_wait();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(deq_bar(a));
      a += 3;
      if (a >= p.slots) { a -= p.slots; aph ^= 1u; }
      st += 3;
      if (RING && st >= nst) { st -= nst; ph ^= 1u; }
    }
    if (dgroup == 0 && ok) {
      // ------------------------------ epilogue (warps 2-5: lane quadrants 2, 3, 0, 1) ------------------------------
      const int qd = warp & 3;
      // one decision for the warp, and the lanes together again after the polling loop: the tensor-memory loads
      // below are warp-wide instructions
      if (__all_sync(0xffffffffu, tc::mbar_wait(accf_bar, 0u, p.status, 35))) {
        __syncwarp();
        tc::fence_after_sync();
        if (warp == 2 && lane == 0) SK_MARK(6);
        const uint32_t taddr = tmem_base + (uint32_t(qd * 32) << 16);
        // this block's part of the tile, fp32 [token][128 features], over the stages
        float* part = reinterpret_cast<float*>(smem) + qd * 32 + lane;
        for (int ch = 0; ch < p.bt / 32; ++ch) {
          uint32_t r[32];
          tc::tmem_ld_32x32(taddr + ch * 32, r);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) part[(ch * 32 + j) * 128] = __uint_as_float(r[j]);
        }
      }
    }
  }

  __syncwarp();
  tc::fence_before_sync();
  // every part is in its block's shared memory
  if (p.ksplit == 1) {
    __syncthreads();
  } else {
    tc::cluster_sync();
  }
  {
    const int rows = min(p.bt, p.M - tt * p.bt);  // tokens of this tile
    const int m0 = ks * rows / p.ksplit, count = ((ks + 1) * rows / p.ksplit - m0) * 32;  // four features of a token per step
    uint32_t part[kSkMaxSplit];
#pragma unroll
    for (int s = 0; s < kSkMaxSplit; ++s) part[s] = s < p.ksplit ? tc::mapa(base, s) : 0u;
    for (int o4 = threadIdx.x; o4 < count; o4 += kSkThreads) {
      const int tok = m0 + (o4 >> 5), f = ft * 128 + (o4 & 31) * 4;
      const size_t idx = size_t(tt * p.bt + tok) * p.N + f;
      uint2 res = make_uint2(0u, 0u);
      if (p.residual) res = *reinterpret_cast<const uint2*>(p.residual + idx);
      float4 a[kSkMaxSplit];
#pragma unroll
      for (int s = 0; s < kSkMaxSplit; ++s)
        if (s < p.ksplit) a[s] = tc::ld_dsmem_v4(part[s] + uint32_t(tok * 128 + (o4 & 31) * 4) * 4u);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int s = 0; s < kSkMaxSplit; ++s)
        if (s < p.ksplit) {
          v.x += a[s].x; v.y += a[s].y; v.z += a[s].z; v.w += a[s].w;
        }
      const float2 b01 = __half22float2(u32_as_h2(bias4.x)), b23 = __half22float2(u32_as_h2(bias4.y));
      v.x += b01.x; v.y += b01.y; v.z += b23.x; v.w += b23.y;
      const float vv[4] = {v.x, v.y, v.z, v.w};
      const uint16_t rr[4] = {uint16_t(res.x & 0xffffu), uint16_t(res.x >> 16), uint16_t(res.y & 0xffffu), uint16_t(res.y >> 16)};
      uint16_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[e] = float_to_out16(vv[e], BF16);
        if (p.act != kActNone || p.residual) o[e] = epilogue16(o[e], p.act, p.residual != nullptr, rr[e], BF16);
      }
      *reinterpret_cast<uint2*>(p.y + idx) = make_uint2(uint32_t(o[0]) | (uint32_t(o[1]) << 16), uint32_t(o[2]) | (uint32_t(o[3]) << 16));
    }
    if (p.ksplit > 1) tc::cluster_sync_relaxed();  // no block leaves while another reads its part
  }
  if (threadIdx.x == 0) SK_MARK(7);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, tmem_cols);
  }
}

struct SkinnyPlan {
  int bt, n_tt, ksplit, nkb, stages, slots, grid;
  size_t smem;
  double us;  // estimate
};

// Blocks of one launch that run at once as clusters of `split` (the size leaves some SMs without a whole cluster): the
// answer of the driver for the kernel's block at one block per SM, or two where its shared memory allows.
int skinny_capacity(int split, size_t smem) {
  static std::atomic<int> known[kSkMaxSplit + 1][2];  // one kind of device: asked once per process
  const bool two = smem <= kSkTwoPerSm;
  std::atomic<int>& k = known[split][two];
  int n = k.load(std::memory_order_relaxed);
  if (n) return n;
  auto kern = gemm_a16_skinny_kernel<4, false, false>;
  const size_t ask = two ? kSkTwoPerSm : kSkMaxSmem;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), ask)) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(split));
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = ask;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  k.store(n * split, std::memory_order_relaxed);
  return n * split;
}

// Token tile and K parts: the pair with the least estimated time among those whose blocks run in one wave.  The estimate (us)
// follows the measurements of 17 to 1500 tokens on eight layer shapes: 4 for launch, first fetches and stores, 0.31 per K block
// (dequantisation and its hand-over; the MMAs of 256 columns hide behind it), 0.011 per column of the tile for its way out of
// tensor memory, 0.6 for the clusters' two barriers.  It has no term for two blocks on an SM: no plan counts on a second one.
bool skinny_search(int64_t M, int64_t N, int64_t K, int sm_count, SkinnyPlan* pl) {
  const int64_t nft = N / 128, nkb = K / 64;
  pl->us = 1e30;
  for (int bt : {32, 64, 96, 128, 192, 256}) {
    if (bt - 32 >= M && bt != 32) break;
    const int64_t n_tt = (M + bt - 1) / bt, tiles = nft * n_tt;
    if (tiles > sm_count) continue;
    const size_t stage = size_t(bt) * 128 + kSkWSlot;
    const int64_t fit = std::min<int64_t>(kSkMaxStages, int64_t((kSkMaxSmem - 1024) / stage));
    for (int64_t sp = 1; sp <= kSkMaxSplit && sp <= nkb && tiles * sp <= sm_count; ++sp) {
      const int64_t kb = (nkb + sp - 1) / sp, stages = std::min(kb, fit);
      const int slots = kb <= 3 || bt + 6 * int(kSkSlotCols) > 256 ? 3 : 6;
      // A block with all of tensor memory shares its SM with nobody: one of another launch's cluster could hold it up in its allocation
      // while it is itself waited for in its own.  From 96 tokens on a block has its SM to itself, too: two of one launch on one SM beside
      // SMs that the launch before still held took 7.4-8.7 us where one each takes 6.6-7.4 (1280 -> 3840 at 96 and 128 tokens, 2048 -> 2048 at 96).
      const size_t smem = skinny_tmem_cols(bt, slots) == 512 ? kSkMaxSmem : std::max(bt >= 96 ? kSkTwoPerSm + 1024 : 0, 1024 + std::max(size_t(stages) * stage, size_t(bt) * 512));
      const double us = 4.0 + 0.31 * double(kb) + 0.011 * bt + (sp > 1 ? 0.6 : 0.0);
      if (us >= pl->us || (sp > 1 && skinny_capacity(int(sp), smem) < tiles * sp)) continue;
      *pl = {bt, int(n_tt), int(sp), int(nkb), int(stages), slots, int(tiles * sp), smem, us};
    }
  }
  return pl->us < 1e30;
}

bool skinny_plan(int64_t M, int64_t N, int64_t K, int group_size, int sm_count, size_t workspace_bytes, SkinnyPlan* pl) {
  if (M < 1 || M > kSkMaxM || N % 128 || K % 64 || group_size <= 0 || group_size % 64 || K % group_size) return false;
  if (workspace_bytes < kStatusBytes) return false;
  struct Entry {
    int64_t M, N, K;
    int sms;
    bool ok;
    SkinnyPlan plan;
  };
  thread_local Entry known[16];  // a program's layers come round again; a few thousand candidates' arithmetic does not have to
  thread_local unsigned next = 0;
  for (const Entry& e : known)
    if (e.M == M && e.N == N && e.K == K && e.sms == sm_count) {
      *pl = e.plan;
      return e.ok;
    }
  Entry& e = known[next++ % 16];
  e = {M, N, K, sm_count, false, {}};
  e.ok = skinny_search(M, N, K, sm_count, &e.plan);
  *pl = e.plan;
  return e.ok;
}

template <int BITS, bool BF16>
int launch_skinny(const CUtensorMap& tmx, const CUtensorMap& tmw, const SkinnyParams& p, int grid, size_t smem,
                  cudaStream_t stream) {
  auto kern = int64_t(p.nkb + p.ksplit - 1) / p.ksplit > p.stages ? gemm_a16_skinny_kernel<BITS, BF16, true> : gemm_a16_skinny_kernel<BITS, BF16, false>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.ksplit;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = option(kOptNoPdl) ? 1 : 2;
  ASRQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmx, tmw, p));
  return ASRQ_OK;
}

}  // namespace

// Estimated time in us, or a negative number where the kernel does not cover the call (in one wave).
double gemm_a16_skinny_estimate(int64_t M, int64_t N, int64_t K, int group_size, int sm_count, size_t workspace_bytes) {
  SkinnyPlan pl;
  return skinny_plan(M, N, K, group_size, sm_count, workspace_bytes, &pl) ? pl.us : -1.0;
}

int gemm_a16_skinny(int bits, const void* x, const uint8_t* w, const void* scales, const void* zeros, const void* bias,
                    void* y, int64_t M, int64_t N, int64_t K, int group_size, int dtype, void* workspace,
                    size_t workspace_bytes, int sm_count, cudaStream_t stream, const Epilogue& ep) {
  SkinnyPlan pl;
  if (!skinny_plan(M, N, K, group_size, sm_count, workspace_bytes, &pl))
    return fail(ASRQ_ERR_SHAPE, "w%da16 skinny gemm: unsupported shape M=%lld N=%lld K=%lld g=%d", bits, (long long)M,
                (long long)N, (long long)K, group_size);
  if (!aligned16(x) || !aligned16(w)) return fail(ASRQ_ERR_ALIGN, "w%da16 skinny gemm: x and w must be 16-byte aligned", bits);
  SkinnyParams p;
  p.scales = static_cast<const __half*>(scales);
  p.zeros = static_cast<const __half*>(zeros);
  p.bias = static_cast<const __half*>(bias);
  p.residual = static_cast<const uint16_t*>(ep.residual);
  p.act = ep.act;
  p.y = static_cast<uint16_t*>(y);
  p.status = static_cast<unsigned*>(workspace);
  p.M = int(M);
  p.N = int(N);
  p.K = int(K);
  p.group_size = group_size;
  p.groups_per_row = int(K / group_size);
  p.bt = pl.bt;
  p.ksplit = pl.ksplit;
  p.nkb = pl.nkb;
  p.n_tt = pl.n_tt;
  p.stages = pl.stages;
  p.slots = pl.slots;
  p.trace = nullptr;
#ifdef ASRQ_TRACE
  if (option(kOptTrace) && workspace_bytes >= (8u << 20)) {  // marks of the launches since the option last changed
    static int launch_no = 0;
    static unsigned gen = 0;
    if (gen != options_generation()) { gen = options_generation(); launch_no = 0; }
    p.trace = reinterpret_cast<unsigned long long*>(static_cast<char*>(workspace) + (4u << 20)) + size_t(launch_no % 64) * 148 * 8;
    ++launch_no;
  }
#endif
  const bool bf16 = dtype == ASRQ_BF16;
  CUtensorMap tmx, tmw;
  int rc = make_tmap_2d(&tmx, x, 2, bf16, uint64_t(K), uint64_t(M), 64, uint32_t(pl.bt), kSwizzle128);
  if (rc) return rc;
  rc = make_tmap_2d(&tmw, w, 1, false, uint64_t(K) * bits / 8, uint64_t(N), uint32_t(8 * bits), 128, kSwizzleNone);
  if (rc) return rc;
  if (bits == 4)
    return bf16 ? launch_skinny<4, true>(tmx, tmw, p, pl.grid, pl.smem, stream)
                : launch_skinny<4, false>(tmx, tmw, p, pl.grid, pl.smem, stream);
  return bf16 ? launch_skinny<2, true>(tmx, tmw, p, pl.grid, pl.smem, stream)
              : launch_skinny<2, false>(tmx, tmw, p, pl.grid, pl.smem, stream);
}

}  // namespace asrq
