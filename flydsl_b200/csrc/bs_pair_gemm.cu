// FP8 block-scale GEMM on CTA pairs:
//   C[m,n] = sum_kb ( sum_{k in kb} A[m,k] * B[n,k] ) * sa[kb,m] * sb[n/128,kb]
//
// Two CTAs of a cluster share a 256 x 256 tile (tcgen05.mma.cta_group::2, M = 256): each fetches its own 128
// rows of A and half of the weight rows, 32 KB per K block instead of the 48 KB of a single CTA's 128 x 256
// tile, so five stages fit beside the staging tile instead of three, and the shared-memory traffic of a K block
// (operands written once and read by the MMAs) falls from 96 to 80 KB.
//
// A K block is issued as two groups of N = 128 instructions, one per column half of the tile, each half with
// two accumulator buffers of its own and four epilogue warps of its own. What bounds the single-CTA kernel is
// the chain MMAs -> completion seen -> drained -> buffer handed back, which has to fit into two K blocks: with
// one 256-wide group the MMAs take one of the two, with halves half of one.
//
// Measured, steady streams of calls, single-CTA tiles / pairs: 4096 x 7168 x 2048 72.1 / 69.0 us, 4096 x 4096 x
// 7168 131 / 125, 16384 x 4096 x 7168 487 / 462, 256 x 24576 x 1536 19.6 / 17.6 (rested: 60.7 / 57.9, 113 / 108, 419 /
// 396, 19.8 / 18.1). What bounds it now is the promotion and the power cap together: with the drain left out
// (a probe) 4096 x 4096 x 7168 takes 103 us, with the TMEM loads but no FMAs 113. Not kept: the next K block's first
// load requested ahead of its turn (a conditional tcgen05.ld; 6 % slower), 8- and 32-column loads (3 and 2 %
// slower), unpacked FMAs (6 %); without asking for the next completion ahead of time it is 6 % slower.
//
// Roles per CTA (384 threads): warp 0 producer, warp 1 MMA issuer (leader CTA) and TMEM allocation, warp 2 store
// thread, warp 3 relay (peer: tells the leader that a stage has landed), warps 4-11 epilogue. A completed group
// is announced to both CTAs by one multicast commit. Every wait is bounded; on expiry the role records a code in
// the device error word and all roles leave through the common teardown (both CTAs always reach the final
// cluster barrier). Bit-equal to the tiled kernel of blockscale_gemm.cu.
// Reference: kernels/blockscale_preshuffle_gemm.py:161-839, promotion :509-587.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "cluster.cuh"
#include "common.cuh"
#include "flyb200.h"
#include "pair.cuh"

namespace flyb200 {

int make_tensor_map_2d(CUtensorMap* map, const void* base, int rows, int cols, int elem_bytes, int box_rows);

namespace {

constexpr int kThreads = 384;
constexpr int kBK = 128;                         // K bytes per stage row = one scale block
constexpr int kStages = 5;
constexpr int kABytes = 128 * kBK;
constexpr int kChunkBytes = 64 * kBK;            // this CTA's 64 weight rows of one column half
constexpr int kStageBytes = kABytes + 2 * kChunkBytes;
constexpr int kRegionBytes = 128 * 128;          // 128 rows x 64 16-bit outputs
constexpr int kStagingBytes = 4 * kRegionBytes;
constexpr int kMisc = 2048;
constexpr int kSmem = kStages * kStageBytes + kStagingBytes + kMisc + 1024;
constexpr int kBufs = 2;                         // accumulator buffers per column half
// completion barriers per half, by K-block iteration: more than the stages, so that none is re-armed before the
// producer has seen its previous phase
constexpr int kDone = kStages + kBufs;
constexpr int kHalfWarps = 4;                    // epilogue warps per column half
static_assert(kSmem <= 232448 && kSmem >= tmem_share_bytes(512), "shared memory");

struct Params {
  const uint8_t* b;
  const float* scale_a;    // [K/128, M]
  const float* scale_b;    // [ceil(N/128), K/128]
  int* err;
  int M, N, K;
  int group_m;             // pair-row blocks per group of the tile order (0 = one group)
};

struct Tile {
  int pm, n;   // pair-row block (256 rows), column tile (256 columns)
};

template <typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
bs_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_c,
               const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  const uint32_t cstage_base = smem_base + kStages * kStageBytes;
  uint8_t* misc = smem_al + kStages * kStageBytes + kStagingBytes;
  const uint32_t bar_base = cstage_base + kStagingBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };   // own loads landed (leader: and the peer's)
  auto done_bar = [&](int h, uint32_t i) { return bar_base + 8u * (kStages + h * kDone + i); };
  auto tempty_bar = [&](int h, int b) { return bar_base + 8u * (kStages + 2 * kDone + h * kBufs + b); };   // leader
  auto cfull_bar = [&](int h) { return bar_base + 8u * (kStages + 2 * kDone + 2 * kBufs + h); };
  auto cfree_bar = [&](int h) { return bar_base + 8u * (kStages + 2 * kDone + 2 * kBufs + 2 + h); };
  constexpr int kNumBars = kStages + 2 * kDone + 2 * kBufs + 4;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(misc + 8 * kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 8 * kNumBars + 4);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(full_bar(s), leader ? 2 : 1);   // leader: + the peer relay's arrival
    for (int h = 0; h < 2; ++h) {
      for (int i = 0; i < kDone; ++i) mbar_init(done_bar(h, i), 1);
      for (int b = 0; b < kBufs; ++b) mbar_init(tempty_bar(h, b), 2 * kHalfWarps);   // the warps of both CTAs
      mbar_init(cfull_bar(h), kHalfWarps);
      mbar_init(cfree_bar(h), 1);
    }
    *abort_flag = 0;
    fence_proxy_async_smem();
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const int KB = p.K / kBK;
  const int num_pm = (p.M + 255) / 256;
  const int num_n = (p.N + 255) / 256;
  const int total = num_pm * num_n;
  const int pair = static_cast<int>(blockIdx.x >> 1);
  const int npairs = static_cast<int>(gridDim.x >> 1);
  const int gm = (p.group_m > 0 && p.group_m < num_pm) ? p.group_m : num_pm;
  auto decode = [&](int t) {
    Tile o;
    const int per_group = gm * num_n;
    const int g = t / per_group;
    const int r = t - g * per_group;
    const int rows_here = min(gm, num_pm - g * gm);
    o.n = r / rows_here;
    o.pm = g * gm + (r - o.n * rows_here);
    return o;
  };

  if (warp < 4) {
    reg_dealloc<40>();   // 40 x 128 + 232 x 256 = the 168 x 384 of the launch
    if (warp == 0 && lane == 0) {
      // ---------------- producer: this CTA's 128 rows of A and 64 weight rows of either half ----------------
      uint32_t it = 0;
      bool alive = true;
      for (int t = pair; t < total && alive; t += npairs) {
        const Tile tl = decode(t);
        const int row0 = tl.pm * 256 + static_cast<int>(rank) * 128;
        const int n0 = tl.n * 256 + static_cast<int>(rank) * 64, n1 = n0 + 128;
        const uint32_t bytes0 = static_cast<uint32_t>(max(0, min(64, p.N - n0))) * kBK;
        const uint32_t bytes1 = static_cast<uint32_t>(max(0, min(64, p.N - n1))) * kBK;
        const uint8_t* wsrc = p.b + static_cast<size_t>(n0) * kBK;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kStages;
          if (it >= kStages) {   // the second half's MMAs are the last to read a stage
            const uint32_t j = it - kStages;
            if (!mbar_wait(done_bar(1, j % kDone), (j / kDone) & 1, abort_flag, p.err, kErrWaitSmemEmpty)) {
              alive = false;
              break;
            }
          }
          const uint32_t sa = smem_base + s * kStageBytes;
          mbar_arrive_expect_tx(full_bar(s), kABytes + bytes0 + bytes1);
          tma_load_2d(sa, &tmap_a, kb * kBK, row0, full_bar(s));
          const uint8_t* w = wsrc + static_cast<size_t>(kb) * p.N * kBK;
          if (bytes0) bulk_load(sa + kABytes, w, bytes0, full_bar(s));
          if (bytes1) bulk_load(sa + kABytes + kChunkBytes, w + 128 * kBK, bytes1, full_bar(s));
        }
      }
    } else if (warp == 1 && leader) {
      // ---------------- MMA issuer (leader): two groups of 256 x 128 x 32 per K block ----------------
      const bool issue = elect_one();
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
      constexpr uint32_t idesc = umma_idesc_e4m3_f32(256, 128);
      // stage, completion barrier and accumulator buffer of the K block, and their phases, kept as counters
      uint32_t s = 0, ph = 0, dn = 0, b = 0, tph = 1;
      bool alive = true;
      for (int t = pair; t < total && alive; t += npairs) {
        for (int kb = 0; kb < KB; ++kb) {
          const uint32_t sa = smem_base + s * kStageBytes;
          const uint64_t adesc = umma_desc_sw128(sa);
          const uint64_t bdesc0 = umma_desc_sw128(sa + kABytes);
          const uint64_t bdesc1 = umma_desc_sw128(sa + kABytes + kChunkBytes);
          // the operands of both CTAs and the two halves' buffers, asked for together
          bool ready1;
          const bool ready0 = mbar_test_2_1(full_bar(s), ph, tempty_bar(0, b), tph, tempty_bar(1, b), tph, ready1);
          if (!__all_sync(0xffffffffu, ready0)) {
            const bool ok = mbar_wait(full_bar(s), ph, abort_flag, p.err, kErrWaitSmemFull) &&
                            mbar_wait(tempty_bar(0, b), tph, abort_flag, p.err, kErrWaitTmemEmpty);
            if (!__all_sync(0xffffffffu, ok)) {
              alive = false;
              break;
            }
          }
          tc_fence_after();
          if (issue) {
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              tc_mma_f8_2(tmem_u + b * 128, adesc + 2 * k, bdesc0 + 2 * k, idesc, k > 0 ? 1u : 0u);
            tc_commit2_both(done_bar(0, dn));
          }
          __syncwarp();
          if (!__all_sync(0xffffffffu, ready1)) {
            const bool ok = mbar_wait(tempty_bar(1, b), tph, abort_flag, p.err, kErrWaitTmemEmpty);
            if (!__all_sync(0xffffffffu, ok)) {
              alive = false;
              break;
            }
          }
          tc_fence_after();
          if (issue) {
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              tc_mma_f8_2(tmem_u + (kBufs + b) * 128, adesc + 2 * k, bdesc1 + 2 * k, idesc, k > 0 ? 1u : 0u);
            tc_commit2_both(done_bar(1, dn));
          }
          __syncwarp();
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
          if (++dn == kDone) dn = 0;
          tph ^= b;
          b ^= 1;
        }
      }
    } else if (warp == 2 && lane == 0) {
      // ---------------- store thread: staged halves -> TMA stores ----------------
      uint32_t n = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += npairs, ++n) {
        const Tile tl = decode(t);
        const int row0 = tl.pm * 256 + static_cast<int>(rank) * 128;
        for (int h = 0; h < 2; ++h) {
          if (!mbar_wait(cfull_bar(h), n & 1, abort_flag, p.err, kErrWaitEpilogue)) {
            ok = false;
            break;
          }
          if (row0 < p.M) {
#pragma unroll
            for (int reg = 0; reg < 2; ++reg) {
              const int col = tl.n * 256 + h * 128 + reg * 64;
              if (col < p.N) tma_store_2d(&tmap_c, cstage_base + (h * 2 + reg) * kRegionBytes, col, row0);
            }
            bulk_commit_group();
            bulk_wait_group_read0();
          }
          mbar_arrive(cfree_bar(h));
        }
      }
      bulk_wait_group0();
    } else if (warp == 3 && lane == 0 && !leader) {
      // ---------------- relay (peer): my stage has landed -> tell the leader ----------------
      uint32_t it = 0;
      bool alive = true;
      for (int t = pair; t < total && alive; t += npairs) {
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait(full_bar(s), (it / kStages) & 1, abort_flag, p.err, kErrWaitSmemFull)) {
            alive = false;
            break;
          }
          mbar_arrive_remote(full_bar(s), 0);
        }
      }
    }
  } else {
    reg_alloc<232>();
    // ---------------- epilogue: a warp owns 32 rows x 128 columns (one half) of this CTA's 128 rows ----------------
    const int quad = warp & 3, half = (warp - 4) >> 2;
    const int r = quad * 32 + lane;   // row inside the CTA's 128 rows = TMEM lane
    const uint32_t tmem_h = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * kBufs * 128;
    const int nblk_max = (p.N + 127) / 128 - 1;
    struct Scales {
      const float* sa;   // this row's scale of K block kb at sa + kb * M
      const float* sb;   // this half's at sb + kb
    };
    // rows beyond M take row 0's scales, halves beyond N the last block's: their results are not stored
    auto scales_of = [&](int t) {
      const Tile tl = decode(t);
      const int row = tl.pm * 256 + static_cast<int>(rank) * 128 + r;
      Scales c;
      c.sa = p.scale_a + (row < p.M ? row : 0);
      c.sb = p.scale_b + static_cast<size_t>(min(tl.n * 2 + half, nblk_max)) * KB;
      return c;
    };
    constexpr int kRing = 4;   // K blocks between a scale's load and its use: ~1.2 us, more than a cold load
    float ring_a[kRing], ring_b[kRing];
    Scales cur{};
    if (pair < total) {
      cur = scales_of(pair);
#pragma unroll
      for (int j = 0; j < kRing; ++j) {
        const int kb = j < KB ? j : 0;
        ring_a[j] = __ldg(cur.sa + static_cast<size_t>(kb) * p.M);
        ring_b[j] = __ldg(cur.sb + kb);
      }
    }
    uint32_t tiles = 0;
    int buf = 0;
    uint32_t dn_i = 0, dn_ph = 0;   // iteration % kDone and (iteration / kDone) & 1
    bool ready = false;             // the next K block's group is known to have completed (warp-uniform)
    // where this half's buffers are handed back: barriers of the leader CTA
    const uint32_t tempty0 = leader ? tempty_bar(half, 0) : map_to_cta(tempty_bar(half, 0), 0);
    const uint32_t tempty1 = leader ? tempty_bar(half, 1) : map_to_cta(tempty_bar(half, 1), 0);
    bool alive = true;
    for (int t = pair; t < total && alive; t += npairs, ++tiles) {
      float2 acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = make_float2(0.f, 0.f);
      const float* pf_a = cur.sa + static_cast<size_t>(kRing) * p.M;
      const float* pf_b = cur.sb + kRing;
      float nring_a[kRing], nring_b[kRing];
      for (int kb0 = 0; kb0 < KB && alive; kb0 += kRing) {
        if (kb0 + kRing >= KB && t + npairs < total) {
          // last trip: the next tile's first scales, so that their latency hides behind the store phase
          cur = scales_of(t + npairs);
#pragma unroll
          for (int j = 0; j < kRing; ++j) {
            const int kb = j < KB ? j : 0;
            nring_a[j] = __ldg(cur.sa + static_cast<size_t>(kb) * p.M);
            nring_b[j] = __ldg(cur.sb + kb);
          }
        }
#pragma unroll
        for (int j = 0; j < kRing; ++j) {
          const int kb = kb0 + j;
          if (kb < KB && alive) {
            if (!ready) {
              const bool got = mbar_wait(done_bar(half, dn_i), dn_ph, abort_flag, p.err, kErrWaitTmemFull);
              if (!__all_sync(0xffffffffu, got)) {
                alive = false;
                break;
              }
            }
            tc_fence_after();
            const uint32_t src = tmem_h + buf * 128;
            uint32_t va[16], vb[16];
            tmem_ld<16>(src, va);
            // in the shadow of the first load: the scale, the loads of later scales, the counters
            const float s = ring_a[j] * ring_b[j];
            asm volatile("" ::"f"(s));   // formed before the slot is loaded again (see blockscale_gemm.cu)
            if (kb + kRing < KB) {
              ring_a[j] = __ldg(pf_a);
              ring_b[j] = __ldg(pf_b);
            }
            pf_a += p.M;
            ++pf_b;
            const uint32_t rel = buf ? tempty1 : tempty0;
            if (++dn_i == kDone) {
              dn_i = 0;
              dn_ph ^= 1;
            }
            const float2 s2 = make_float2(s, s);
            tmem_wait_dep<16>(va);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              uint32_t* cv = (q & 1) ? vb : va;
              uint32_t* nv = (q & 1) ? va : vb;
              if (q < 7) tmem_ld<16>(src + (q + 1) * 16, nv);   // in flight during the FMAs
              if (q == 6) ready = mbar_test(done_bar(half, dn_i), dn_ph);   // the next K block's
              float2* a = acc + q * 8;
#pragma unroll
              for (int c = 0; c < 8; ++c)
                a[c] = __ffma2_rn(make_float2(__uint_as_float(cv[2 * c]), __uint_as_float(cv[2 * c + 1])), s2, a[c]);
              if (q < 7) tmem_wait_dep<16>(nv);
              // Everything has been read: the buffer goes back to the issuer. The wait above is one instruction
              // of the whole warp (.sync.aligned), for the loads of all its lanes, so lane 0 may speak for them
              // without a __syncwarp (which costs 1.5 %).
              if (q == 6) {
                tc_fence_before();
                mbar_arrive_if(rel, lane == 0 && leader);
                mbar_arrive_cluster_if(rel, lane == 0 && !leader);
              }
            }
            ready = __all_sync(0xffffffffu, ready);
            buf ^= 1;
          }
        }
      }
      if (!alive) break;
      if (tiles > 0) {   // the store of this half's previous tile has read the staging regions
        const bool ok = mbar_wait(cfree_bar(half), (tiles - 1) & 1, abort_flag, p.err, kErrWaitEpilogue);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
#pragma unroll
      for (int j = 0; j < 64; j += 4) {   // 8 columns
        const int col = 2 * j;            // inside the half
        const uint32_t addr = cstage_base + (half * 2 + (col >> 6)) * kRegionBytes + r * 128 +
                              ((((col & 63) >> 3) ^ (r & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(pack2(acc[j].x, acc[j].y, OutT())),
                     "r"(pack2(acc[j + 1].x, acc[j + 1].y, OutT())), "r"(pack2(acc[j + 2].x, acc[j + 2].y, OutT())),
                     "r"(pack2(acc[j + 3].x, acc[j + 3].y, OutT()))
                     : "memory");
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(cfull_bar(half));
#pragma unroll
      for (int j = 0; j < kRing; ++j) {
        ring_a[j] = nring_a[j];
        ring_b[j] = nring_b[j];
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();   // nobody frees tensor memory or leaves while the partner may still use it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
}

template <typename OutT>
int launch_bs_pair(const CUtensorMap& tmap_a, const CUtensorMap& tmap_c, const Params& p, int pairs,
                   cudaStream_t stream) {
  auto kern = bs_pair_kernel<OutT>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  FLYB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    FLYB200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  FLYB200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmap_a, tmap_c, p));
  return FLYB200_OK;
}

}  // namespace

// N % 16 == 0, K % 128 == 0, M >= 128 (see plan_dense in blockscale_gemm.cu for when it is taken).
int launch_blockscale_pair_gemm(void* c, const void* a, const void* b_repacked, const float* scale_a_t,
                                const float* scale_b, int M, int N, int K, int out_dtype, int ctas, int group_m,
                                cudaStream_t stream) {
  Params p{};
  p.b = static_cast<const uint8_t*>(b_repacked);
  p.scale_a = scale_a_t;
  p.scale_b = scale_b;
  p.err = device_error_word();
  if (!p.err) return FLYB200_ERR_CUDA;
  p.M = M; p.N = N; p.K = K;
  p.group_m = group_m / 2;
  CUtensorMap tmap_a, tmap_c;
  int rc;
  if ((rc = make_tensor_map_2d(&tmap_a, a, M, K, 1, 128))) return rc;
  if ((rc = make_tensor_map_2d(&tmap_c, c, M, N, 2, 128))) return rc;
  if (out_dtype == FLYB200_BF16) return launch_bs_pair<__nv_bfloat16>(tmap_a, tmap_c, p, ctas / 2, stream);
  return launch_bs_pair<__half>(tmap_a, tmap_c, p, ctas / 2, stream);
}

}  // namespace flyb200
