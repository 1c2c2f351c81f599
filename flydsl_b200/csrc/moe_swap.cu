// MoE stages for small routing blocks (tile_m <= 32, activations in routing order): decode batches,
// where an expert sees a handful of tokens and the layer is a stream of expert weights.
//
// Swap-AB: the WEIGHT rows are the MMA's M side (128 accumulator lanes = 128 output channels), the
// tokens its N side (NT = 32 or 64 columns). The tiled kernel (blockscale_gemm.cu) puts the tokens on
// the M side, so a block of 16 or 32 tokens is padded to 128 rows: four to eight times the tensor work,
// and the 48 KB stages that go with it leave three of them, 96 KB of weights in flight per SM. Neither
// costs time on a rested GPU, but under the power cap the padded MMAs take the clock down (1.97 ->
// 1.40 GHz at 1 kW in a steady stream of calls) and with it the weight stream. Here a stage is two
// 16 KB weight tiles and NT x 128 bytes of tokens, six stages fit, 192 KB of weights in flight.
// Steady stream of calls, 256 experts of 7168 x 2048, top 8, 16 hot experts: 32 tokens 630-695 -> 567 us,
// 256 tokens 2095-2120 -> 1686-1720 us (stage 1 at 6.9 TB/s of weights); per-token scales, 1000 tokens
// in blocks of 32: 2385 -> 1912 us, 1400 / 705 us for the stages without the merging of blocks and 1126 /
// 589 us with it.
//
// A CTA's tile is two 128-row weight tiles (stage 1: the gate and the up rows of the same 128
// intermediate channels, stage 2: two neighbouring 128-row tiles) against one routing block, or two
// that follow one another in the same expert: their rows are contiguous, and one pass over the weights
// serves both.
//   warp 0      producer: two bulk copies (weights) and one TMA tile (tokens) per K block
//   warp 1      MMA issuer: 2 x 4 tcgen05.mma 128 x NT x 32 per K block
//   warps 2-9   epilogue: a warp owns 32 channels of both weight tiles and half of the tokens; thread =
//               channel, registers = tokens. Block scales: every K block in a fresh accumulator buffer,
//               acc = fma(partial, sa[token] * sb, acc) as in the tiled kernel; per-token scales: the
//               whole K range in one buffer. Outputs are stored from registers: 32 lanes = 64
//               contiguous bytes of a row.
// Reference: the stage kernels of kernels/moe_blockscale_2stage.py (:206-1161, :1386-2387) and
// kernels/moe_gemm_2stage.py (:93-1264, :1267-2481).
#include "common.cuh"

namespace flyb200 {

int make_tensor_map_2d(CUtensorMap* map, const void* base, int rows, int cols, int elem_bytes, int box_rows);

namespace {

constexpr int kSwThreads = 320;
constexpr int kSwEpiWarp0 = 2;
constexpr int kSwEpiWarps = 8;
constexpr int kSwW = 128 * 128;   // bytes of a weight tile's K block

struct SwapParams {
  const uint8_t* b;
  const float* scale_a;    // [K/128, a_rows], per token: [a_rows]
  const float* scale_b;
  void* out;
  int* err;
  int M;                   // tokens
  int N;                   // stage 1: intermediate channels, stage 2: model channels
  int K;
  const int* sorted_ids;
  const int* expert_ids;
  const float* sorted_weights;
  const int* num_valid;
  int topk, tile_m, num_blocks, experts, doweight, accumulate, out_sorted, a_rows;
};

template <int NT>
struct SwapCfg {
  static constexpr int kStageBytes = 2 * kSwW + NT * 128;
  static constexpr int kStages = NT == 64 ? 5 : 6;
  static constexpr int kAccBufs = 512 / (2 * NT) > 8 ? 8 : 512 / (2 * NT);
  static constexpr int kTmemCols = 2 * NT * kAccBufs;
  static constexpr int kDone = kStages + kAccBufs;
  static constexpr int kListBytes = kMoeSwapListed * 2;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + kListBytes + 1024;
  static_assert(kSmemBytes <= 232448, "shared memory");
};

__device__ __forceinline__ void store1(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void store1(__half* p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store1(float* p, float v) { *p = v; }
// One output of each lane, 32 neighbouring columns from `p` (this lane's) on: added, two to a word.
__device__ __forceinline__ void add_row(__nv_bfloat16* p, float v, int lane) {
  const float hi = __shfl_xor_sync(0xffffffffu, v, 1);
  if (!(lane & 1))
    asm volatile("red.global.add.noftz.bf16x2 [%0], %1;" ::"l"(p), "r"(pack2(v, hi, __nv_bfloat16())) : "memory");
}
__device__ __forceinline__ void add_row(__half* p, float v, int lane) {
  const float hi = __shfl_xor_sync(0xffffffffu, v, 1);
  if (!(lane & 1))
    asm volatile("red.global.add.noftz.f16x2 [%0], %1;" ::"l"(p), "r"(pack2(v, hi, __half())) : "memory");
}
__device__ __forceinline__ void add_row(float* p, float v, int) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

template <int NT, int STAGE, bool PT, typename OutT>
__global__ void __launch_bounds__(kSwThreads, 1)
moe_swap_kernel(const __grid_constant__ CUtensorMap tmap_x, const SwapParams p) {
  using C = SwapCfg<NT>;
  constexpr int HT = NT / 2;   // tokens per epilogue warp
  constexpr int kSwStages = C::kStages, kSwAccBufs = C::kAccBufs, kSwDone = C::kDone;
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* misc = smem_raw + (smem_base - smem_u32(smem_raw)) + kSwStages * C::kStageBytes;
  const uint32_t bar_base = smem_base + kSwStages * C::kStageBytes;
  // full[s]: operands of stage s landed; done[i]: the MMAs of K-block iteration i (mod kSwDone) have
  // finished (stage free, and with block scales: partials in tensor memory); tempty[b]: buffer b has
  // been read; tfull[b]: per-token scales, tile accumulated
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto done_bar = [&](uint32_t i) { return bar_base + 8u * (kSwStages + i); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (kSwStages + kSwDone + b); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (kSwStages + kSwDone + kSwAccBufs + b); };
  constexpr int kNumBars = kSwStages + kSwDone + 2 * kSwAccBufs;
  static_assert(8 * kNumBars + 12 <= 1024, "barrier area");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(misc + 8 * kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 8 * kNumBars + 4);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSwStages; ++s) mbar_init(full_bar(s), 1);
    for (int i = 0; i < kSwDone; ++i) mbar_init(done_bar(i), 1);
    for (int b = 0; b < kSwAccBufs; ++b) {
      mbar_init(tempty_bar(b), kSwEpiWarps);
      mbar_init(tfull_bar(b), 1);
    }
    *abort_flag = 0;
    fence_proxy_async_smem();
    fence_barrier_init();
    prefetch_tensormap(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // Tiles: all channel tiles of a token tile, then the next token tile (those of an expert follow one
  // another, so its weights are still in L2 for the second one). Token tiles: warp 0 lists the routing
  // blocks that start one -- every other block of a run of blocks of the same expert -- as block number
  // and, in the top bit, whether the next block belongs to it too. With more blocks than the list
  // holds every block is a tile.
  const int KB = p.K / 128;
  constexpr int kCols = STAGE == 1 ? 128 : 256;   // output channels per tile
  const int num_n = (p.N + kCols - 1) / kCols;
  const int num_m = max(0, min(p.num_blocks, (p.num_valid[0] + p.tile_m - 1) / p.tile_m));
  const bool listed = num_m <= kMoeSwapListed;
  uint16_t* const list = reinterpret_cast<uint16_t*>(misc + 1024);
  volatile int* const list_len = reinterpret_cast<volatile int*>(misc + 8 * kNumBars + 8);
  if (warp == 0 && listed) {
    int run_start = 0, n = 0;
    for (int m0 = 0; m0 < num_m; m0 += 32) {
      const int m = m0 + lane;
      const int e = m < num_m ? p.expert_ids[m] : -1;
      const int before = m > 0 && m < num_m ? p.expert_ids[m - 1] : -1;
      const int after = m + 1 < num_m ? p.expert_ids[m + 1] : -1;
      const unsigned firsts = __ballot_sync(0xffffffffu, m < num_m && (m == 0 || before != e));
      const unsigned upto = firsts & (0xffffffffu >> (31 - lane));
      const int start = upto ? m0 + 31 - __clz(upto) : run_start;
      const bool leads = m < num_m && e >= 0 && e < p.experts && ((m - start) & 1) == 0;
      const unsigned mask = __ballot_sync(0xffffffffu, leads);
      if (leads)
        list[n + __popc(mask & ((1u << lane) - 1u))] = static_cast<uint16_t>(m | (after == e ? 0x8000 : 0));
      n += __popc(mask);
      if (firsts) run_start = m0 + 31 - __clz(firsts);
    }
    if (lane == 0) *list_len = n;
  }
  __syncthreads();
  const int total = (listed ? *list_len : num_m) * num_n;
  const int step = static_cast<int>(gridDim.x);
  // token tile, expert and first channel of tile t; false: a block without an expert
  struct Tile {
    int m_blk, blocks, e, n0;
  };
  auto tile_of = [&](int t, Tile& o) -> bool {
    const int i = t / num_n;
    o.n0 = (t - i * num_n) * kCols;
    o.m_blk = i;
    o.blocks = 1;
    if (listed) {
      const int v = list[i];
      o.m_blk = v & 0x7fff;
      o.blocks = 1 + (v >> 15);
    }
    o.e = p.expert_ids[o.m_blk];
    return o.e >= 0 && o.e < p.experts;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- producer ----------------
      uint32_t it = 0;
      bool alive = true;
      const uint64_t pol_evict_first = l2_policy_evict_first();
      for (int t = blockIdx.x; t < total && alive; t += step) {
        Tile tl;
        if (!tile_of(t, tl)) continue;
        const int e = tl.e, n0 = tl.n0, m_next = tl.m_blk + tl.blocks;
        // the last tile of an expert reads its weights for the last time: they leave L2 first
        const bool last_use = m_next >= num_m || p.expert_ids[m_next] != e;
        const int rows_w = STAGE == 1 ? 2 * p.N : p.N;   // weight rows of an expert
        const uint8_t* w0 = p.b + static_cast<size_t>(e) * rows_w * p.K + static_cast<size_t>(n0) * 128;
        const size_t second = STAGE == 1 ? static_cast<size_t>(p.N) * 128 : static_cast<size_t>(kSwW);
        const bool two = STAGE == 1 || n0 + 128 < p.N;
        const uint32_t bytes = (two ? 2 : 1) * kSwW + tl.blocks * p.tile_m * 128;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kSwStages;
          if (it >= kSwStages) {
            const uint32_t j = it - kSwStages;
            if (!mbar_wait(done_bar(j % kSwDone), (j / kSwDone) & 1, abort_flag, p.err, kErrWaitSmemEmpty)) {
              alive = false;
              break;
            }
          }
          const uint32_t base = smem_base + s * C::kStageBytes;
          const uint8_t* src = w0 + static_cast<size_t>(kb) * rows_w * 128;
          mbar_arrive_expect_tx(full_bar(s), bytes);
          if (last_use) {
            bulk_load_hint(base, src, kSwW, full_bar(s), pol_evict_first);
            if (two) bulk_load_hint(base + kSwW, src + second, kSwW, full_bar(s), pol_evict_first);
          } else {
            bulk_load(base, src, kSwW, full_bar(s));
            if (two) bulk_load(base + kSwW, src + second, kSwW, full_bar(s));
          }
          tma_load_2d(base + 2 * kSwW, &tmap_x, kb * 128, tl.m_blk * p.tile_m, full_bar(s));
          if (tl.blocks > 1)
            tma_load_2d(base + 2 * kSwW + p.tile_m * 128, &tmap_x, kb * 128, (tl.m_blk + 1) * p.tile_m, full_bar(s));
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool leader = elect_one();
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    uint32_t it = 0, tiles = 0;
    bool alive = true;
    for (int t = blockIdx.x; t < total && alive; t += step) {
      Tile tl;
      if (!tile_of(t, tl)) continue;
      const bool two = STAGE == 1 || tl.n0 + 128 < p.N;
      const uint32_t idesc = tl.blocks * p.tile_m <= HT ? umma_idesc_e4m3_f32(128, HT) : umma_idesc_e4m3_f32(128, NT);
      for (int kb = 0; kb < KB; ++kb, ++it) {
        const int s = it % kSwStages;
        const uint32_t n = PT ? tiles : it;   // what the accumulator buffers rotate with
        const int buf = n % kSwAccBufs;
        const uint32_t fph = (it / kSwStages) & 1, eph = ((n / kSwAccBufs) & 1) ^ 1;
        if (!__all_sync(0xffffffffu, mbar_test_both(full_bar(s), fph, tempty_bar(buf), eph))) {
          const bool ok = mbar_wait(full_bar(s), fph, abort_flag, p.err, kErrWaitSmemFull) &&
                          mbar_wait(tempty_bar(buf), eph, abort_flag, p.err, kErrWaitTmemEmpty);
          if (!__all_sync(0xffffffffu, ok)) {
            alive = false;
            break;
          }
        }
        tc_fence_after();
        const uint32_t base = smem_base + s * C::kStageBytes;
        const uint64_t wdesc = umma_desc_sw128(base);
        const uint64_t vdesc = umma_desc_sw128(base + kSwW);
        const uint64_t xdesc = umma_desc_sw128(base + 2 * kSwW);
        const uint32_t d = tmem_u + buf * 2 * NT;
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc_mma_f8(d, wdesc + 2 * k, xdesc + 2 * k, idesc, ((PT && kb) || k) ? 1u : 0u);
          if (two) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc_mma_f8(d + NT, vdesc + 2 * k, xdesc + 2 * k, idesc, ((PT && kb) || k) ? 1u : 0u);
          }
          tc_commit(done_bar(it % kSwDone));
          if (PT && kb + 1 == KB) tc_commit(tfull_bar(buf));
        }
        __syncwarp();
      }
      ++tiles;
    }
  } else {
    // ---------------- epilogue ----------------
    const int quad = warp & 3;                         // tensor-memory lanes this warp may read
    const int half = (warp - kSwEpiWarp0) >> 2;        // its tokens: [half * HT, half * HT + HT)
    const uint32_t t0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * HT;
    OutT* const out = static_cast<OutT*>(p.out);
    uint32_t it = 0, tiles = 0;
    bool alive = true;
    for (int t = blockIdx.x; t < total && alive; t += step) {
      Tile tl;
      if (!tile_of(t, tl)) continue;
      const int m_blk = tl.m_blk, e = tl.e, n0 = tl.n0;
      const int rows = tl.blocks * p.tile_m;   // tokens and padding
      const bool active = half * HT < rows;    // a warp without tokens hands its buffers back unread
      const bool two = STAGE == 1 || n0 + 128 < p.N;
      // lane j (< HT) looks after token j of this warp's half: output row, route weight, scale
      const int tok = half * HT + lane;
      const bool mine = lane < HT && tok < rows;
      const int pos = m_blk * p.tile_m + (mine ? tok : 0);
      long long row = -1;   // element offset of the token's output row
      float route_w = 1.f;
      {
        const int id = p.sorted_ids[pos];
        const int tt = id & 0xFFFFFF, slot = static_cast<unsigned>(id) >> 24;
        if (mine && tt < p.M && slot < p.topk) {
          if (STAGE == 1 && p.out_sorted) row = static_cast<long long>(pos) * p.N;
          else if (STAGE == 2 && p.accumulate) row = static_cast<long long>(tt) * p.N;
          else row = (static_cast<long long>(tt) * p.topk + slot) * p.N;
          if (p.doweight) route_w = p.sorted_weights[pos];
        }
      }
      float acc_a[HT], acc_b[HT];   // first / second weight tile
      constexpr int CW = 16;        // tokens per pair of tensor-memory loads
      uint32_t va[CW], vb[CW];
      if constexpr (!PT) {
#pragma unroll
        for (int j = 0; j < HT; ++j) acc_a[j] = acc_b[j] = 0.f;
        const long long nb_exp = (STAGE == 1 ? 2 * p.N : p.N) / 128;
        const float* sa = p.scale_a + pos;
        const float* sb_a = p.scale_b + (e * nb_exp + n0 / 128) * KB;
        const float* sb_b = STAGE == 1 ? sb_a + static_cast<long long>(p.N / 128) * KB : two ? sb_a + KB : sb_a;
        // scales four K blocks ahead (a K block's weights take about as long as one cold load)
        constexpr int kRing = 4;
        float ra[kRing], rb_a[kRing], rb_b[kRing];
#pragma unroll
        for (int j = 0; j < kRing; ++j) {
          const int kb = j < KB ? j : 0;
          ra[j] = __ldg(sa + static_cast<long long>(kb) * p.a_rows);
          rb_a[j] = __ldg(sb_a + kb);
          rb_b[j] = __ldg(sb_b + kb);
        }
        for (int kb0 = 0; kb0 < KB && alive; kb0 += kRing) {
#pragma unroll
          for (int u = 0; u < kRing; ++u) {
            const int kb = kb0 + u;
            if (kb < KB && alive) {
              // both products before the ring is loaded again (see the tiled kernel's K loop)
              const float sc_a = ra[u] * rb_a[u], sc_b = ra[u] * rb_b[u];
              asm volatile("" ::"f"(sc_a), "f"(sc_b));
              if (kb + kRing < KB) {
                ra[u] = __ldg(sa + static_cast<long long>(kb + kRing) * p.a_rows);
                rb_a[u] = __ldg(sb_a + kb + kRing);
                rb_b[u] = __ldg(sb_b + kb + kRing);
              }
              const int buf = it % kSwAccBufs;
              const bool got = mbar_wait(done_bar(it % kSwDone), (it / kSwDone) & 1, abort_flag, p.err,
                                         kErrWaitTmemFull);
              if (!__all_sync(0xffffffffu, got)) {
                alive = false;
                break;
              }
              tc_fence_after();
              auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(buf));
              };
              if (!active) {
                release();
              } else {
#pragma unroll
                for (int c = 0; c < HT; c += CW) {
                  tmem_ld<CW>(t0 + buf * 2 * NT + c, va);
                  tmem_ld<CW>(t0 + buf * 2 * NT + NT + c, vb);
                  tmem_wait_dep<CW>(va);
                  tmem_wait_dep<CW>(vb);
                  if (c + CW == HT) release();
#pragma unroll
                  for (int j = 0; j < CW; ++j) {
                    acc_a[c + j] = fmaf(__uint_as_float(va[j]), __shfl_sync(0xffffffffu, sc_a, c + j), acc_a[c + j]);
                    acc_b[c + j] = fmaf(__uint_as_float(vb[j]), __shfl_sync(0xffffffffu, sc_b, c + j), acc_b[c + j]);
                  }
                }
              }
              ++it;
            }
          }
        }
        if (!alive) break;
      } else {
        // per-token / per-channel scales: one drain per tile
        const float sa = __ldg(p.scale_a + pos);
        const float* sw = p.scale_b + static_cast<long long>(e) * (STAGE == 1 ? 2 * p.N : p.N) + n0 + quad * 32 + lane;
        const float sw_a = __ldg(sw);
        const float sw_b = two ? __ldg(sw + (STAGE == 1 ? p.N : 128)) : 0.f;
        const int buf = tiles % kSwAccBufs;
        const bool got = mbar_wait(tfull_bar(buf), (tiles / kSwAccBufs) & 1, abort_flag, p.err, kErrWaitTmemFull);
        if (!__all_sync(0xffffffffu, got)) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < HT; c += CW) {
          tmem_ld<CW>(t0 + buf * 2 * NT + c, va);
          tmem_ld<CW>(t0 + buf * 2 * NT + NT + c, vb);
          tmem_wait_dep<CW>(va);
          tmem_wait_dep<CW>(vb);
          if (c + CW == HT) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(buf));
          }
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            const float s = __shfl_sync(0xffffffffu, sa, c + j);
            acc_a[c + j] = __uint_as_float(va[j]) * (s * sw_a);
            acc_b[c + j] = __uint_as_float(vb[j]) * (s * sw_b);
          }
        }
      }
      ++tiles;

      // ---- output: this lane's channel of every token ----
      const int n = n0 + quad * 32 + lane;
#pragma unroll
      for (int j = 0; j < HT; ++j) {
        const long long off = __shfl_sync(0xffffffffu, row, j);
        const float w = __shfl_sync(0xffffffffu, route_w, j);
        if (off < 0) continue;   // the whole warp
        if constexpr (STAGE == 1) {
          store1(out + off + n, silu_mul(acc_a[j], acc_b[j]) * w);
        } else if (p.accumulate) {
          add_row(out + off + n, acc_a[j] * w, lane);
          if (two) add_row(out + off + n + 128, acc_b[j] * w, lane);
        } else {
          store1(out + off + n, acc_a[j] * w);
          if (two) store1(out + off + n + 128, acc_b[j] * w);
        }
      }
    }
  }

  // ---------------- teardown ----------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a role gave up: copies still in flight land before shared memory and TMEM are handed back
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int NT, int STAGE, bool PT, typename OutT>
int launch_swap(const CUtensorMap& tmap, const SwapParams& p, int grid, cudaStream_t stream) {
  using C = SwapCfg<NT>;
  auto kern = moe_swap_kernel<NT, STAGE, PT, OutT>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  FLYB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    FLYB200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(kSwThreads, 1, 1);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  FLYB200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmap, p));
  return FLYB200_OK;
}
template <int STAGE, bool PT, typename OutT>
int launch_nt(const CUtensorMap& tmap, const SwapParams& p, int grid, cudaStream_t stream) {
  return p.tile_m <= 16 ? launch_swap<32, STAGE, PT, OutT>(tmap, p, grid, stream)
                        : launch_swap<64, STAGE, PT, OutT>(tmap, p, grid, stream);
}

}  // namespace

// Entry of the MoE stages for routing-order activations in blocks of at most 32 tokens (tile_m a
// multiple of 8). Arguments have been checked by the caller; `a_rows` = rows of the activations.
int launch_moe_swap(int stage, bool pertoken, void* out, const void* act, const void* w_repacked,
                    const float* scale_x, const float* scale_w, const int32_t* sorted_ids, const int32_t* expert_ids,
                    const float* sorted_weights, const int32_t* num_valid_ids, int T, int n, int kdim, int num_blocks,
                    int E, int k, int tile_m, int doweight, int accumulate, int out_sorted, int a_rows, int out_dtype,
                    int max_ctas, cudaStream_t stream) {
  const int sms = sm_count();
  if (sms <= 0) return FLYB200_ERR_CUDA;
  SwapParams p{};
  p.b = static_cast<const uint8_t*>(w_repacked);
  p.scale_a = scale_x; p.scale_b = scale_w; p.out = out;
  p.err = device_error_word();
  if (!p.err) return FLYB200_ERR_CUDA;
  p.M = T; p.N = n; p.K = kdim;
  p.sorted_ids = sorted_ids; p.expert_ids = expert_ids; p.sorted_weights = sorted_weights;
  p.num_valid = num_valid_ids;
  p.topk = k; p.tile_m = tile_m; p.num_blocks = num_blocks; p.experts = E;
  p.doweight = doweight; p.accumulate = accumulate; p.out_sorted = out_sorted; p.a_rows = a_rows;
  const int cols = stage == 1 ? 128 : 256;
  const long tiles = static_cast<long>(num_blocks) * ((n + cols - 1) / cols);
  int grid = sms;
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (tiles < grid) grid = static_cast<int>(tiles);
  CUtensorMap tmap;
  int rc = make_tensor_map_2d(&tmap, act, a_rows, kdim, 1, tile_m);
  if (rc) return rc;
  if (stage == 1) {
    if (out_dtype == FLYB200_BF16)
      return pertoken ? launch_nt<1, true, __nv_bfloat16>(tmap, p, grid, stream)
                      : launch_nt<1, false, __nv_bfloat16>(tmap, p, grid, stream);
    return pertoken ? launch_nt<1, true, __half>(tmap, p, grid, stream)
                    : launch_nt<1, false, __half>(tmap, p, grid, stream);
  }
  if (out_dtype == FLYB200_BF16)
    return pertoken ? launch_nt<2, true, __nv_bfloat16>(tmap, p, grid, stream)
                    : launch_nt<2, false, __nv_bfloat16>(tmap, p, grid, stream);
  if (out_dtype == FLYB200_F16)
    return pertoken ? launch_nt<2, true, __half>(tmap, p, grid, stream)
                    : launch_nt<2, false, __half>(tmap, p, grid, stream);
  return pertoken ? launch_nt<2, true, float>(tmap, p, grid, stream)
                  : launch_nt<2, false, float>(tmap, p, grid, stream);
}

}  // namespace flyb200
