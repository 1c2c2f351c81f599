// Weight-only int4 x bf16 GEMM for decode-size M (<= 64 tokens): C[M, N] = A[M, K] * dequant(W)[N, K]^T,
// W signed 4-bit with one bf16 scale per (row, 128-wide K group). HBM-bound on the packed weights
// (N*K/2 bytes), so the kernel streams them once and does everything else on chip:
//
//   * swap-AB like the fp8 decode kernel: the 128-row weight tile is the MMA "A" operand
//     (accumulator lane = output column n), the tokens are the MMA "B" operand (NT = 16/32/64).
//   * one thread feeds a ring of shared-memory slots: the packed 128 x 128 group (8 KB, one bulk copy) and the
//     tokens' 128 K columns (two TMA tiles).
//   * two sets of four dequantiser warps, each taking every other group. A thread owns a weight row (= TMEM lane):
//     it reads the row's 64 packed bytes, turns them into EXACT bf16 values q / 4 and writes them with tcgen05.st
//     where tcgen05.mma takes its A operand from: tensor memory. The weights never go back to shared memory
//     (the image there is four times the packed bytes, written and read again). The unpacking takes 2.25
//     instructions per two weights, one of them on the FMA pipe (with 3.25 the integer pipe was 59 % busy and bound the
//     kernel, 14.6 us at N = K = 8192 and 16 tokens; now 33 % and 12.4 us): nibble n = q + 8 in the low bits, (n | 0x4300) is bf16 128 + n, times 1/4 minus 34 gives q / 4; n in bits 4-7 is the bf16 number n 2^-129
//     (bits up to 255 are subnormals or have the same spacing), times 2^127 minus 2 gives q / 4 without a shift.
//   * tcgen05.mma kind::f16 (bf16 x bf16 -> f32), 128 x NT x 16, eight per K group, each group into a
//     fresh accumulator buffer; the issuing warp stays converged (one elected lane issues).
//   * the epilogue applies the group scale per accumulator lane in fp32 --
//     acc[n][m] += scale[n][g] * sum_k q[n][k] / 4 * a[m][k] (times 4 when it is stored) -- the same promotion structure as the
//     block-scale kernels; this equals dequantise-then-matmul with the products q*a summed exactly
//     in fp32 before scaling.
//   * split-K over a thread-block cluster with the partials exchanged by bulk copies through
//     distributed shared memory and summed in rank order (deterministic), as in decode_gemm.cu.
//   * up to 32 tokens a CTA takes half an SM (448 threads of 64 registers, 256 TMEM columns, 113 KB), so
//     that two share one and hide each other's chain dequantise -> MMA -> completion -> dequantise. Each set owns one
//     operand buffer there, and that chain is what a group takes (0.31 us alone, 0.24 with two CTAs): ncu shows no unit
//     more than half busy (issue slots 44 %, integer pipe 33 %, DRAM 24 %, tensor pipe 7 %).
//
// The reference has no kernel for this exact format (its nearest code is the W4A16 path of
// kernels/moe_gemm_2stage.py:607-630 and the int4 unpack of kernels/mfma_preshuffle_pipeline.py:
// 202-222); the contract is "dequantise, then matmul".
//
// Packed layout (flyb200_int4_repack): wq [K/128][N/8][4][8][16 bytes] -- per 128-K group and block
// of 8 rows, four 16-byte chunks (32 K elements each), each chunk holding its 8 rows back to back,
// so that a warp reading one chunk of 8 consecutive rows touches 128 contiguous bytes. The 8 nibbles
// of each 32-bit word hold 8 consecutive K elements in the order e0 e2 e4 e6 e1 e3 e5 e7 (low nibble
// first), so that (word >> 4q) & 0x000F000F yields the pair (e_2q, e_2q+1) in the two 16-bit
// halves: a 32-bit column of the operand in tensor memory. Scales [K/128][N] bf16.
#include "common.cuh"
#include "cluster.cuh"

namespace flyb200 {

constexpr int kI4DqSets = 2;
constexpr int kI4MaxSlots = 16;
constexpr int kI4PackedBytes = 128 * 64;
constexpr int kI4ACols = 64;        // TMEM columns of a group's weights: 128 K, two per column

struct Int4Params {
  const uint8_t* wq;               // [K/128][N/8][4][8][16]
  const __nv_bfloat16* scales_t;   // [K/128][N]
  void* out;                       // [M, N] bf16
  int* err;
  int M, N, K;
  int splits, kbps, slots;
};

// A from tensor memory, B from shared memory.
__device__ __forceinline__ void tc_mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// (a & mask) | bits in one instruction; from the expression the compiler makes two, which bounded the dequantisers
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(bits));
  return d;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// registers -> TMEM: thread i of the warp writes lane (base lane + i), 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// bf16 x bf16 -> f32, both operands K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16_f32(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

template <int NT>
struct I4Cfg {
  // warp 0 copies, warp 1 MMA, then the epilogue warps (four for up to 32 token columns), then the dequantisers
  static constexpr int kEpiSets = NT > 32 ? NT / 32 : 1;
  static constexpr int kEpiCols = NT / kEpiSets;
  static constexpr int kDqWarp0 = 2 + 4 * kEpiSets;
  static constexpr int kThreads = 32 * (kDqWarp0 + 4 * kI4DqSets);
  static constexpr int kXSub = NT * 128;                     // one 64-K sub-tile of the tokens
  static constexpr int kSlotBytes = kI4PackedBytes + 2 * kXSub;
  static constexpr bool kHalfSm = NT <= 32;                  // two CTAs share an SM
  static constexpr int kTmemCols = kHalfSm ? 256 : 512;
  static constexpr int kABufs = kHalfSm ? 2 : 4;             // a multiple of the sets: buffer i % kABufs is set i % 2's
  static constexpr int kDBufs = (kTmemCols - kABufs * kI4ACols) / NT;
  static constexpr int kRecvBytes = (NT + 8) * 128 * 4;      // [sender][local token][128] fp32
  // completion barriers, by group: more than a waiter may lag behind (the ring's depth, the accumulator buffers)
  static constexpr int kDone = kI4MaxSlots + kDBufs;
  static constexpr int kMiscBytes = 1024;
  static int ring_bytes(int slots) {   // the ring doubles as the send buffer of the exchange
    return slots * kSlotBytes > NT * 512 ? slots * kSlotBytes : NT * 512;
  }
  // + the group scales of the CTA's K range: [kbps][128] bf16
  static int fixed_bytes(int kbps) { return kRecvBytes + kbps * 256 + kMiscBytes + 1024; }
  static int smem_bytes(int slots, int kbps) {
    const int bytes = ring_bytes(slots) + fixed_bytes(kbps);
    return bytes > tmem_share_bytes(kTmemCols) ? bytes : tmem_share_bytes(kTmemCols);
  }
};

template <int NT>
__global__ void __launch_bounds__(I4Cfg<NT>::kHalfSm ? 512 : I4Cfg<NT>::kThreads, I4Cfg<NT>::kHalfSm ? 2 : 1)
int4_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const Int4Params p) {
  using C = I4Cfg<NT>;
  constexpr int kABufs = C::kABufs, kDBufs = C::kDBufs, kDone = C::kDone;
  static_assert(kABufs % kI4DqSets == 0, "an operand buffer belongs to one set");
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int slots = p.slots;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const int ring = slots * C::kSlotBytes;
  const uint32_t recv_off = static_cast<uint32_t>(ring > NT * 512 ? ring : NT * 512);
  const uint32_t recv_base = smem_base + recv_off;
  const float* recv = reinterpret_cast<const float*>(smem_al + recv_off);
  const uint32_t scale_off = recv_off + C::kRecvBytes;                       // [kbps][128] bf16
  const __nv_bfloat16* sc_s = reinterpret_cast<const __nv_bfloat16*>(smem_al + scale_off);
  const uint32_t misc_off = scale_off + static_cast<uint32_t>(p.kbps) * 256u;
  const uint32_t bar_base = smem_base + misc_off;
  auto full_bar = [&](uint32_t s) { return bar_base + 8u * s; };                          // a slot has landed
  auto done_bar = [&](uint32_t i) { return bar_base + 8u * (kI4MaxSlots + i); };          // a group's MMAs are done
  auto aready_bar = [&](uint32_t b) { return bar_base + 8u * (kI4MaxSlots + kDone + b); };   // operand written
  auto dempty_bar = [&](uint32_t b) { return bar_base + 8u * (kI4MaxSlots + kDone + kABufs + b); };
  constexpr int kBars = kI4MaxSlots + kDone + kABufs + kDBufs + 2;
  const uint32_t recv_bar = bar_base + 8u * (kBars - 2);
  const uint32_t scale_bar = bar_base + 8u * (kBars - 1);
  static_assert(8 * kBars + 8 <= C::kMiscBytes, "barrier area");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_al + misc_off + 8 * kBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_al + misc_off + 8 * kBars + 4);

  const int split = static_cast<int>(cluster_ctarank());
  const int n_tile = blockIdx.x / p.splits;
  const int n0 = n_tile * 128;
  const int KBt = p.K / 128;
  const int kb_begin = split * p.kbps;
  const int kb_end = min(KBt, kb_begin + p.kbps);
  const int count = max(0, kb_end - kb_begin);
  const int cpc = (p.M + p.splits - 1) / p.splits;   // tokens each CTA of the cluster reduces and stores

  if (warp == 0) {
    if (lane < slots) mbar_init(full_bar(lane), 1);
    if (lane < kDone) mbar_init(done_bar(lane), 1);
    if (lane < kABufs) mbar_init(aready_bar(lane), 4);
    if (lane < kDBufs) mbar_init(dempty_bar(lane), 4 * C::kEpiSets);
    if (lane == 0) {
      mbar_init(recv_bar, 1);
      mbar_init(scale_bar, 1);
      *abort_flag = 0;
      prefetch_tensormap(&tmap_x);
    }
    fence_proxy_async_smem();
    fence_barrier_init();
    if (lane == 0) {
      const int own = min(p.M, (split + 1) * cpc) - split * cpc;
      if (own > 0) mbar_arrive_expect_tx(recv_bar, static_cast<uint32_t>(own * p.splits) * 512u);
    }
  }
  static_assert(kDone <= 32, "one lane initialises one barrier");
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_d = tmem_base + kABufs * kI4ACols;
  cluster_sync_all();   // the receive barriers of the whole cluster exist before anybody signals them

  // Programmatic dependent launch: the packed weights and group scales of the first ring fill are
  // requested BEFORE the dependency wait -- they are parameters, never the result of the kernel that
  // runs just before (a kernel of this library that lets its dependents start early writes no
  // weights; any other kernel has exited before this one starts). The tokens are read after it.
  const int first_fill = count < slots ? count : slots;
  const uint8_t* wsrc = p.wq + (static_cast<size_t>(kb_begin) * p.N + n0) * 64;   // the next group's weights
  const size_t wstep = static_cast<size_t>(p.N) * 64;
  // The whole of warp 0 runs the copy loop and one elected lane issues: as a chain of scalar instructions in one
  // thread, with two token copies per group, it took 760 cycles a group and bounded the kernel.
  const bool copier = warp == 0 && elect_one();
  auto load_weights = [&](uint32_t bar, uint32_t dst) {
    if (copier) {
      mbar_arrive_expect_tx(bar, C::kSlotBytes);
      bulk_load(dst, wsrc, kI4PackedBytes, bar);
    }
    wsrc += wstep;
  };
  if (warp == 0) {
    for (int i = 0; i < first_fill; ++i) load_weights(full_bar(i), smem_base + i * C::kSlotBytes);
    if (copier && count > 0) {
      mbar_arrive_expect_tx(scale_bar, static_cast<uint32_t>(count) * 256u);
      for (int i = 0; i < count; ++i)   // all in flight at once: one by one they cost a DRAM latency per group
        bulk_load(smem_base + scale_off + i * 256, p.scales_t + static_cast<size_t>(kb_begin + i) * p.N + n0, 256,
                  scale_bar);
    }
    __syncwarp();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ---------------- copies ----------------
    int k64 = kb_begin * 2;   // the tokens' next 64-column slab
    auto load_tokens = [&](uint32_t bar, uint32_t slot) {
      if (copier) tma_load_3d(slot + kI4PackedBytes, &tmap_x, 0, 0, k64, bar);
      k64 += 2;
    };
    for (int i = 0; i < first_fill; ++i)   // of the slots whose weights are on their way
      load_tokens(full_bar(i), smem_base + i * C::kSlotBytes);
    uint32_t s = 0, slot = smem_base, dn = 0, dph = 0;
    for (int i = first_fill; i < count; ++i) {   // first_fill == slots here: the slot's last group was i - slots
      const bool ok = mbar_wait(done_bar(dn), dph, abort_flag, p.err, kErrWaitSmemEmpty);
      if (!__all_sync(0xffffffffu, ok)) break;
      load_weights(full_bar(s), slot);
      load_tokens(full_bar(s), slot);
      __syncwarp();
      slot += C::kSlotBytes;
      if (++s == static_cast<uint32_t>(slots)) {
        s = 0;
        slot = smem_base;
      }
      if (++dn == kDone) {
        dn = 0;
        dph ^= 1;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp runs the loop, one elected lane issues ----------------
    const bool issue = elect_one();
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    constexpr uint32_t idesc = umma_idesc_bf16_f32(128, NT);
    uint32_t s = 0, ph = 0, dn = 0;
    for (int i = 0; i < count; ++i) {
      const uint32_t ab = i % kABufs, aph = (i / kABufs) & 1;
      const uint32_t db = i % kDBufs, dph = ((i / kDBufs) & 1) ^ 1;
      const uint32_t a = tmem_u + ab * kI4ACols, d = tmem_u + kABufs * kI4ACols + db * NT;
      const uint32_t x = smem_base + s * C::kSlotBytes + kI4PackedBytes;
      const uint64_t xdesc0 = umma_desc_sw128(x), xdesc1 = umma_desc_sw128(x + C::kXSub);
      const bool ok = mbar_wait(dempty_bar(db), dph, abort_flag, p.err, kErrWaitTmemEmpty) &&
                      mbar_wait(full_bar(s), ph, abort_flag, p.err, kErrWaitSmemFull) &&
                      mbar_wait(aready_bar(ab), aph, abort_flag, p.err, kErrWaitGather);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      if (issue) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          tc_mma_bf16_ts(d, a + k * 8, (k < 4 ? xdesc0 : xdesc1) + 2 * (k & 3), idesc, k ? 1u : 0u);
        tc_commit(done_bar(dn));   // operand, slot and accumulator all wait for this one
      }
      __syncwarp();
      if (++s == static_cast<uint32_t>(slots)) {
        s = 0;
        ph ^= 1;
      }
      if (++dn == kDone) dn = 0;
    }
  } else if (warp >= C::kDqWarp0) {
    // ---------------- dequantisers: a thread is one weight row ----------------
    const int set = (warp - C::kDqWarp0) >> 2;
    const int row = (warp & 3) * 32 + lane;   // the TMEM lanes that this warp may write
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t src = smem_base + static_cast<uint32_t>((row >> 3) * 512 + (row & 7) * 16);
    constexpr uint32_t k128 = 0x43004300u, kQuarter = 0x3E803E80u, kMinus34 = 0xC208C208u, k2e127 = 0x7F007F00u,
                       kMinus2 = 0xC000C000u;
    // slot and completion barrier of the group, and their phases, kept as counters: a division by the ring's depth
    // took as long as the loads
    uint32_t s = set, ph = 0, ab = set, dn = set, dph = 0;
    if (s >= static_cast<uint32_t>(slots)) s = 0;   // a ring of one slot has one group
    for (int i = set; i < count; i += kI4DqSets) {
      const bool have = mbar_wait(full_bar(s), ph, abort_flag, p.err, kErrWaitSmemFull);
      if (!__all_sync(0xffffffffu, have)) break;
      uint32_t w[16];
#pragma unroll
      for (int v = 0; v < 4; ++v)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[4 * v]), "=r"(w[4 * v + 1]), "=r"(w[4 * v + 2]), "=r"(w[4 * v + 3])
                     : "r"(src + s * C::kSlotBytes + 128u * v));
      if (i >= kABufs) {   // the MMAs that read this operand buffer last, group i - kABufs
        const bool ok = mbar_wait(done_bar(dn), dph, abort_flag, p.err, kErrWaitTmemEmpty);
        if (!__all_sync(0xffffffffu, ok)) break;
        if ((dn += kI4DqSets) >= kDone) {
          dn -= kDone;
          dph ^= 1;
        }
      }
      tc_fence_after();
      const uint32_t dst = tmem_base + lane_base + ab * kI4ACols;
#pragma unroll
      for (int v = 0; v < 4; ++v) {   // 16 columns = 32 K elements = four words
        uint32_t o[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t lo = w[4 * v + j], hi = lo >> 8;
          o[4 * j] = fma_bf16x2(and_or(lo, 0x000F000Fu, k128), kQuarter, kMinus34);
          o[4 * j + 1] = fma_bf16x2(lo & 0x00F000F0u, k2e127, kMinus2);
          o[4 * j + 2] = fma_bf16x2(and_or(hi, 0x000F000Fu, k128), kQuarter, kMinus34);
          o[4 * j + 3] = fma_bf16x2(hi & 0x00F000F0u, k2e127, kMinus2);
        }
        tmem_st16(dst + v * 16, o);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_if(aready_bar(ab), lane == 0);   // the wait above is one of the whole warp
      if ((s += kI4DqSets) >= static_cast<uint32_t>(slots)) {
        s -= slots;
        ph ^= 1;
      }
      if ((ab += kI4DqSets) >= kABufs) ab -= kABufs;
    }
  } else {
    // ---------------- epilogue: thread = output column n (accumulator lane) ----------------
    constexpr int EC = C::kEpiCols;
    const int col0 = ((warp - 2) >> 2) * EC;    // this warp's token columns
    const int quad = warp & 3;                  // TMEM lane quadrant this warp may read
    const int n_loc = quad * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    float2 acc[EC / 2];
#pragma unroll
    for (int j = 0; j < EC / 2; ++j) acc[j] = make_float2(0.f, 0.f);
    bool alive = true;
    if (count > 0) {
      const bool have = mbar_wait(scale_bar, 0, abort_flag, p.err, kErrWaitSmemFull);
      alive = __all_sync(0xffffffffu, have);
    }
    uint32_t dn = 0, dph = 0;
    for (int i = 0; i < count && alive; ++i) {
      const float sg = __bfloat162float(sc_s[i * 128 + n_loc]);
      const float2 sg2 = make_float2(sg, sg);
      const uint32_t db = i % kDBufs;
      const bool got = mbar_wait(done_bar(dn), dph, abort_flag, p.err, kErrWaitTmemFull);
      if (!__all_sync(0xffffffffu, got)) {
        alive = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < EC; c += 16) {
        uint32_t v[16];
        tmem_ld<16>(tmem_d + lane_base + db * NT + col0 + c, v);
        tmem_wait_dep<16>(v);
        if (c + 16 == EC) {
          tc_fence_before();
          mbar_arrive_if(dempty_bar(db), lane == 0);   // the wait above is one of the whole warp
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          acc[c / 2 + j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), sg2,
                                      acc[c / 2 + j]);
      }
      if (++dn == kDone) {
        dn = 0;
        dph ^= 1;
      }
    }
    // split-K exchange (same scheme as the fp8 decode kernel): partials as [token][n] into the ring (the
    // last group's MMAs are done, so nobody reads it any more), one bulk copy per owner CTA, owners add in
    // rank order and store.
    float* send = reinterpret_cast<float*>(smem_al);
#pragma unroll
    for (int j = 0; j < EC; ++j)
      if (col0 + j < p.M) send[(col0 + j) * 128 + n_loc] = (j & 1) ? acc[j / 2].y : acc[j / 2].x;
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, %0;" ::"n"(128 * C::kEpiSets) : "memory");   // every epilogue warp comes here, also one that gave up
    if (threadIdx.x == 64 && alive) {
      for (int o = 0; o < p.splits; ++o) {
        const int lo = o * cpc;
        const int cols = min(p.M, lo + cpc) - lo;
        if (cols > 0)
          bulk_copy_to_cta(map_to_cta(recv_base + static_cast<uint32_t>(split * cpc) * 512u, o),
                           smem_base + static_cast<uint32_t>(lo) * 512u,
                           static_cast<uint32_t>(cols) * 512u, map_to_cta(recv_bar, o));
      }
    }
    const int j_lo = split * cpc;
    const int j_hi = min(p.M, j_lo + cpc);
    if (j_hi > j_lo && alive) {
      const bool got = mbar_wait(recv_bar, 0, abort_flag, p.err, kErrWaitExchange);
      if (__all_sync(0xffffffffu, got)) {
        __nv_bfloat16* const out = reinterpret_cast<__nv_bfloat16*>(p.out);
        for (int jb = j_lo + ((warp - 2) >> 2) * 8; jb < j_hi; jb += 8 * C::kEpiSets) {
          float sum[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) sum[u] = 0.f;
          for (int c = 0; c < p.splits; ++c) {  // fixed rank order: deterministic
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (jb + u < j_hi) sum[u] += recv[(c * cpc + (jb - j_lo) + u) * 128 + n_loc];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (jb + u < j_hi)
              out[static_cast<size_t>(jb + u) * p.N + n0 + n_loc] = __float2bfloat16_rn(4.f * sum[u]);   // of q / 4
        }
      }
    }
  }

  // A CTA that gave up no longer waits for the copies sent to it, and behind the barrier below their senders may
  // be gone: time for them, and for its own copies and MMAs in flight, to finish.
  if (__any_sync(0xffffffffu, *abort_flag != 0))
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  // Nobody leaves before every bulk copy that reads its shared memory has been consumed.
  cluster_sync_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// values [N, K] int8 in [-8, 7] + scales [N, K/128] bf16 -> the packed layout above
__global__ void __launch_bounds__(256)
int4_repack_kernel(const int8_t* __restrict__ q, const __nv_bfloat16* __restrict__ scales,
                   uint32_t* __restrict__ wq, __nv_bfloat16* __restrict__ scales_t, int N, int K) {
  const int KB = K / 128;
  const long long words = static_cast<long long>(KB) * N * 16;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < words;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int wi = static_cast<int>(i & 15);
    const long long rn = i >> 4;
    const int n = static_cast<int>(rn % N);
    const int kb = static_cast<int>(rn / N);
    const int8_t* src = q + static_cast<size_t>(n) * K + kb * 128 + wi * 8;
    uint32_t w = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t nib = static_cast<uint32_t>(src[e] + 8) & 0xFu;
      const int pos = (e & 1) ? 4 + (e >> 1) : (e >> 1);   // e0 e2 e4 e6 e1 e3 e5 e7
      w |= nib << (4 * pos);
    }
    // [kb][n / 8][chunk = wi / 4][row = n % 8][word = wi % 4]: a warp reading one chunk of eight
    // consecutive rows touches 128 contiguous bytes of the shared-memory copy (no bank conflicts)
    wq[(((static_cast<long long>(kb) * (N / 8) + n / 8) * 4 + (wi >> 2)) * 8 + (n & 7)) * 4 + (wi & 3)] = w;
    if (wi == 0) scales_t[static_cast<size_t>(kb) * N + n] = scales[static_cast<size_t>(n) * KB + kb];
  }
}

int make_tensor_map_slabs16(CUtensorMap* map, const void* base, int rows, int cols, int box_rows,
                            int box_slabs);  // blockscale_gemm.cu

struct I4Plan {
  int nt, splits, kbps, slots;
};

template <int NT>
static int i4_slots(int kbps) {
  using C = I4Cfg<NT>;
  const int least = kbps < 2 ? kbps : 2;
  // half of an SM's shared memory where two CTAs are to share it, all of it where that does not do
  for (int limit : {tmem_share_bytes(C::kTmemCols), 232448}) {
    int slots = (limit - C::fixed_bytes(kbps)) / C::kSlotBytes;
    slots = slots < kbps ? slots : kbps;
    if (slots > kI4MaxSlots) slots = kI4MaxSlots;
    // A ring that wraps is a multiple of the sets deep, so that a slot's groups all belong to one set: a dequantiser
    // warp waits for the fills of its set's groups only, and a parity wait cannot tell a fill that has not landed
    // yet from the one two later.
    if (slots < kbps) slots -= slots % kI4DqSets;
    if (slots >= least && C::smem_bytes(slots, kbps) <= limit) return slots;
  }
  return 0;
}

const int* max_clusters();   // blockscale_gemm.cu

// Estimated time (us) of the tcgen05 kernel, fitted to 2600 shapes (M 1 to 64, N and K from 128 up; graph replays, cold
// weights), each in every cluster size: 4-6 % off while all CTAs are resident. A CTA alone on an SM takes about
// 0.31 us a group, two of up to 32 tokens 0.48 us for a group of each. Clusters that are not all resident make another
// wave (2048 x 2048, 64 tokens, 16 clusters of 8: 11.6 us, of 4: 6.1).
struct I4Times {
  double fixed, group;   // a call, a K group of every CTA
  double fill, store;    // all SMs taken (or taken twice); the outputs stored by one CTA per tile instead of by many
};
static double int4_us(int nt, int n_tiles, int kbps, int splits, int alone, int sms) {
  const bool two = nt <= 32;   // CTAs per SM
  const int resident = two ? 2 * alone : alone;
  double us = 0.0;
  if (n_tiles > resident) {
    us = n_tiles / resident * (nt == 16 ? 4.66 + 0.479 * kbps : nt == 32 ? 5.9 + 0.503 * kbps : 5.6 + 0.36 * kbps);
    n_tiles %= resident;
    if (!n_tiles) return us;
  }
  const I4Times t = n_tiles <= alone ? (nt == 16 ? I4Times{2.55, 0.306, 0.96, 0.0}
                                        : nt == 32 ? I4Times{3.03, 0.334, 0.71, 0.94}
                                                   : I4Times{3.57, 0.355, 1.50, 1.03})
                                     : (nt == 16 ? I4Times{1.70, 0.479, 1.48, 0.0} : I4Times{2.10, 0.503, 1.71, 0.65});
  // 0.05 us per CTA of a cluster: with it 4 of 1800 other calls (weights cold and in L2) are more than 5 % slower than in the
  // clusters chosen before these estimates, without it 16 (3 x 3712 x 5248 6.4 -> 7.1 us in seven CTAs instead of four)
  return us + t.fixed + t.group * kbps + t.fill * n_tiles * splits / sms + t.store / splits + 0.05 * splits +
         (nt == 64 && splits > 6 ? 0.4 : 0.0);   // clusters of seven and eight place badly
}

// K splits (cluster size) and ring depth: the smallest estimated time; within 1 % of the best cluster size on average
// over those shapes, more than 10 % off in 27 of them.
static I4Plan plan_int4(int M, int N, int K, int sms, int force_splits, bool live) {
  I4Plan best{0, 0, 0, 0};
  const int nt = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
  const int n_tiles = N / 128;
  const int KBt = K / 128;
  const int* clusters = live ? max_clusters() : nullptr;   // otherwise estimated
  double best_cost = 1e30;
  for (int s = 1; s <= 8; ++s) {
    if (force_splits > 0 && s != force_splits) continue;
    const int kbps = (KBt + s - 1) / s;
    const int s_eff = (KBt + kbps - 1) / kbps;
    if (s_eff != s && force_splits <= 0) continue;
    const int slots = nt == 16 ? i4_slots<16>(kbps) : nt == 32 ? i4_slots<32>(kbps) : i4_slots<64>(kbps);
    if (!slots) continue;
    int alone = s > 1 && clusters ? clusters[s] : sms / s;   // clusters at one CTA per SM
    if (alone < 1) alone = 1;
    const double cost = int4_us(nt, n_tiles, kbps, s_eff, alone, sms);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = I4Plan{nt, s_eff, kbps, slots};
    }
  }
  return best;
}

// The mma.sync kernel (int4_stream.cu) has less to set up and is faster where there is little to stream. Measured,
// mma.sync / tcgen05 (us, graph replay, cold weights):
//   M = 1   1536 x 1024 2.75 / 3.34, 2048 x 2048 3.85 / 4.04, 3072 x 2048 4.11 / 4.55, 5120 x 1536 4.39 / 4.71, 9216 x
//           1024 4.46 / 4.69; 2048 x 4096 5.28 / 5.14, 4096 x 3072 5.73 / 4.99, 8192 x 8192 18.4 / 12.0
//   M = 16  2048 x 1024 3.20 / 3.62, 1536 x 4096 4.48 / 4.78, 5120 x 1536 4.96 / 4.98, 9216 x 1024 4.75 / 4.84; 4096 x
//           2048 5.07 / 4.71, 8192 x 8192 19.2 / 12.4
//   M = 32  3072 x 1024 4.25 / 4.52, 5120 x 1024 5.29 / 5.47; 1536 x 1536 4.76 / 4.62, 8192 x 8192 23.4 / 13.3
//   M = 64  1024 x 1024 6.03 / 5.25, 8192 x 8192 35.1 / 18.6
// The limits hold for 2280 drawn shapes of up to 32 tokens: the choice is 1 % slower than the faster kernel on average.
// At the limits the two take turns, with the waves of either (3 x 5760 x 1408 4.4 / 4.7, 3 x 4736 x 1664 5.7 / 5.0).
// Beyond K = 5120 the tcgen05 kernel is never the slower one (5 to 13 % faster, whatever N).
static bool stream_beats_tensor(int M, int N, int K) {
  const double weights = static_cast<double>(N) * K;
  if (M <= 16) return K <= 5120 && weights < (K <= 1280 ? 1e7 : 8e6);
  return M <= 32 && K <= 1024 && weights < (K <= 384 ? 7e6 : 5e6);
}

template <int NT>
static int launch_int4(const CUtensorMap& tmap, const Int4Params& p, cudaStream_t stream) {
  auto kern = int4_gemm_kernel<NT>;
  const int smem = I4Cfg<NT>::smem_bytes(p.slots, p.kbps);
  if (smem > 232448) return set_error(FLYB200_ERR_UNSUPPORTED, "int4 plan needs %d bytes of shared memory", smem);
  static thread_local int configured_dev = -1;
  int dev = 0;
  FLYB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    FLYB200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((p.N / 128) * p.splits), 1, 1);
  cfg.blockDim = dim3(I4Cfg<NT>::kThreads, 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = static_cast<unsigned>(p.splits);
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  FLYB200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmap, p));
  return FLYB200_OK;
}

}  // namespace flyb200

namespace flyb200 {
int launch_int4_stream(void* c, const void* a, const void* wq, const void* scales_t, int M, int N, int K,
                       int force_splits, cudaStream_t stream);  // int4_stream.cu
}

using namespace flyb200;

extern "C" int flyb200_int4_repack(const int8_t* q, const void* scales, int32_t N, int32_t K, void* wq_out,
                                   void* scales_t_out, void* stream) {
  if (!q || !scales || !wq_out || !scales_t_out)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_repack: NULL buffer");
  if (N < 8 || N % 8 || K < 128 || K % 128 || reinterpret_cast<uintptr_t>(wq_out) % 16)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT,
                     "int4_repack: K %% 128 == 0, N %% 8 == 0 and a 16-byte aligned output");
  const int sms = sm_count();
  if (sms <= 0) return FLYB200_ERR_CUDA;
  int4_repack_kernel<<<sms * 8, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      q, static_cast<const __nv_bfloat16*>(scales), static_cast<uint32_t*>(wq_out),
      static_cast<__nv_bfloat16*>(scales_t_out), N, K);
  FLYB200_CUDA_CHECK(cudaGetLastError());
  return FLYB200_OK;
}

extern "C" int flyb200_int4_tensor_plan(int32_t M, int32_t N, int32_t K, int32_t split_k, int32_t sms,
                                        int32_t* plan) {
  if (!plan || M < 1 || M > 64 || N < 128 || N % 128 || K < 128 || K % 128)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_tensor_plan: bad arguments (M=%d N=%d K=%d)", M, N, K);
  const bool live = sms <= 0;
  if (live && (sms = sm_count()) <= 0) return FLYB200_ERR_CUDA;
  const I4Plan p = plan_int4(M, N, K, sms, split_k, live);
  plan[0] = p.splits < 1 || stream_beats_tensor(M, N, K) ? 1 : 2;
  plan[1] = p.nt; plan[2] = p.splits; plan[3] = p.kbps; plan[4] = p.slots;
  plan[5] = p.splits < 1 ? 0 : p.nt == 16 ? I4Cfg<16>::smem_bytes(p.slots, p.kbps)
                           : p.nt == 32 ? I4Cfg<32>::smem_bytes(p.slots, p.kbps)
                                        : I4Cfg<64>::smem_bytes(p.slots, p.kbps);
  plan[6] = p.splits < 1 ? 0 : p.nt == 64 ? I4Cfg<64>::kTmemCols : I4Cfg<16>::kTmemCols;
  return FLYB200_OK;
}

extern "C" int flyb200_int4_gemm(void* c, const void* a, const void* wq, const void* scales_t, int32_t M,
                                 int32_t N, int32_t K, const flyb200_gemm_cfg* cfg, void* stream) {
  if (!c || !a || !wq || !scales_t) return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_gemm: NULL buffer");
  // tokens by TMA, packed weights and group scales by bulk copies
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(scales_t)) % 16)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_gemm: a, wq and scales_t must be 16-byte aligned");
  if (M < 1 || M > 64) return set_error(FLYB200_ERR_UNSUPPORTED, "int4_gemm: 1 <= M <= 64 (got %d)", M);
  if (N < 128 || N % 128 || K < 128 || K % 128)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_gemm: N and K must be multiples of 128 (N=%d K=%d)", N, K);
  // cfg.path: 1 = the register-dequantising mma.sync kernel (int4_stream.cu), 2 = the tcgen05 kernel of this
  // file, 0 = whichever was measured faster
  const int path = cfg ? cfg->path : 0;
  const int sms = sm_count();
  if (sms <= 0) return FLYB200_ERR_CUDA;
  I4Plan plan{0, 0, 0, 0};
  if (path == 2 || (path == 0 && !stream_beats_tensor(M, N, K)))
    plan = plan_int4(M, N, K, sms, cfg ? cfg->split_k : 0, true);
  if (path == 2 && plan.splits < 1)
    return set_error(FLYB200_ERR_INVALID_ARGUMENT, "int4_gemm: no plan for M=%d N=%d K=%d", M, N, K);
  if (plan.splits < 1)   // (also K ranges whose group scales leave no room for this kernel's ring)
    return launch_int4_stream(c, a, wq, scales_t, M, N, K, cfg ? cfg->split_k : 0,
                              reinterpret_cast<cudaStream_t>(stream));
  Int4Params p{};
  p.wq = static_cast<const uint8_t*>(wq);
  p.scales_t = static_cast<const __nv_bfloat16*>(scales_t);
  p.out = c;
  p.err = device_error_word();
  if (!p.err) return FLYB200_ERR_CUDA;
  p.M = M; p.N = N; p.K = K;
  p.splits = plan.splits; p.kbps = plan.kbps; p.slots = plan.slots;
  CUtensorMap tmap;
  int rc = make_tensor_map_slabs16(&tmap, a, M, K, plan.nt, 2);
  if (rc) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (plan.nt) {
    case 16: return launch_int4<16>(tmap, p, st);
    case 32: return launch_int4<32>(tmap, p, st);
    default: return launch_int4<64>(tmap, p, st);
  }
}
