// Dense block-FP8 GEMM with 16 promotion warps, on CTA pairs (tcgen05 cta_group::2) or single CTAs. Two CTAs of a cluster
// compute one 256 x 256 output tile.
// Each CTA loads its own 128 rows of A and HALF of the B tile (128 of its 256 rows); the tensor cores of the pair read
// both halves. Per 128-K block a CTA then moves 32 KB into shared memory and its tensor core reads 32 KB back, which
// fits the 512 clocks its MMAs take at 128 B/clk; the single-CTA tile (48 KB each way) does not.
//
// The fp32 scales change every 128 of K, so every K block is pulled out of TMEM, scaled and added in registers.
// Roles per CTA (640 threads):
//   warps 0-15   promotion: warp w owns TMEM lanes 32 (w % 4).. and columns 64 (w / 4)..; 64 accumulators per thread.
//                Four warps per SM sub-partition: the TMEM round trip of one hides behind the FMAs of the others.
//                What the loop costs in instructions is time (the MMA warp waits for the accumulator buffer half of the
//                time) and, at the power cap, clock: packed FMAs straight on what tcgen05.ld returns, no register copies, one
//                scale read from shared memory, two K blocks per trip. Four times (16 columns, 8 FMAs) instead of twice
//                (32, 16) costs 4 %, plain FMAs instead of packed ones 3 %.
//   warp  16     TMA producer (no multicast: every load has one destination CTA)
//   warp  17     MMA issuer (leader CTA only)
//   warps 18-19  scale loaders: products As[row] * Bs[128-column block] of four K blocks at a time into a
//                shared-memory ring [block][row][K block], so a promotion thread reads one float per K block
// Cross-CTA protocol (rank 0 = leader):
//   full[s]   (leader's)  2 arrivals (one expect_tx per producer) + the bytes of both CTAs' TMA loads
//   empty[s]  (each CTA)  arrival from the leader's tcgen05.commit
//   tfull[b]  (each CTA)  likewise
//   tempty[b] (leader's)  32 arrivals: the promotion warps of both CTAs
// The MMA warp's own trip (two polls, four MMAs, two commits) bounds the 128-wide tile; both barriers are polled at once.
// Shared memory is next: a K block writes 24 KB and reads 24 to 32 KB (128 wide), 384 to 448 clocks at 128 B/clk, against 430 measured.
// The scale reads take four wavefronts each (lanes 8 apart share a bank): 64 of those clocks, 16 without the conflict.
// Polled one after the other, and with 5 stages instead of 7: 203 x 8192 x 7168 20.8 -> 18.7 us, 512 x 4096 x 14336 35.0 -> 32.4.
// Looped, with the copies (120 instructions per warp and K block) and without (97): 8192 x 4096 x 4096 143 -> 134 us,
// 1027 x 7168 x 8192 78.6 -> 73.3, 203 x 6144 x 4096 (128-wide tiles) 15.1 -> 13.2.
#pragma once

#include "gemm_host.cuh"

namespace b200 {

namespace ptx {
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes)
               : "memory");
}
// tiled load whose completion bytes are counted on a barrier of the CTA pair's leader
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, int c0, int c1, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(m), "r"(c0), "r"(c1), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma_f8_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
      "}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// one commit that arrives on the barrier at the same shared-memory offset in every CTA of `mask`
// (tcgen05.commit is the one multicast form used anywhere in this library; no data is moved)
__device__ __forceinline__ void mma_commit_pair_multicast(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}
// The forms that differ between a CTA on its own and a pair
template <int CTAS>
__device__ __forceinline__ void wide_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  if constexpr (CTAS == 2) mma_f8_pair(d, da, db, idesc, acc);
  else mma_f8(d, da, db, idesc, acc);
}
template <int CTAS>
__device__ __forceinline__ void wide_load(uint32_t dst, const CUtensorMap* m, int c0, int c1, uint32_t leader_bar) {
  if constexpr (CTAS == 2) tma_load_2d_pair(dst, m, c0, c1, leader_bar);
  else tma_load_2d(dst, m, c0, c1, leader_bar);
}
template <int CTAS>
__device__ __forceinline__ void wide_sync() {
  __syncthreads();
  if constexpr (CTAS == 2) cluster_sync();
}
// Wait for this thread's outstanding tcgen05.ld. The loaded registers are not operands of the wait (as in tmem_ld_wait):
// what reads them is volatile too and stays behind it, and the compiler makes no copies of them.
__device__ __forceinline__ void tmem_ld_wait_all() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// a += b * s on two packed floats, b just loaded from TMEM
__device__ __forceinline__ void ffma2(uint64_t& a, uint32_t b0, uint32_t b1, uint64_t s) {
  asm volatile("{.reg .b64 b; mov.b64 b, {%1, %2}; fma.rn.f32x2 %0, b, %3, %0;}" : "+l"(a) : "r"(b0), "r"(b1), "l"(s));
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
  uint64_t p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}
__device__ __forceinline__ void st_cluster_2x64(uint32_t addr, uint64_t a, uint64_t b) {
  asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void lds_2x64(uint32_t addr, uint64_t& a, uint64_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint64_t pack2(float v) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %1};" : "=l"(p) : "f"(v));
  return p;
}
}  // namespace ptx

// CTAS = 1: a CTA's own 128 x 256 tile (problems whose rows or waves a pair's 256 rows would waste). CTAS = 2:
// BN: columns of the pair's tile, 256 / 192 / 128. The wide tile does the most work per byte moved and per TMEM round
// trip; the narrow ones are for problems of a few waves, whose last wave they fill better.
template <int CTAS, int BN>
struct Wide {
  static constexpr int kStageA = kBM * kBK;       // this CTA's 128 rows of A
  static constexpr int kStageB = (BN / CTAS) * kBK;  // this CTA's share of the B tile
  static constexpr int kAccBufs = BN == 128 ? 4 : 2, kAccStride = BN == 128 ? 128 : 256;  // TMEM accumulator buffers
  static constexpr int kPromWarps = 16, kProducerWarp = 16, kMmaWarp = 17, kScaleWarp = 18;
  static constexpr int kCols = BN / 4, kChunks = kCols / 16;  // columns of one promotion warp, in 16-column chunks
  static constexpr int kThreads = 640;
  // 20 warps start with 96 registers each (5 per sub-partition); 4 x 104 + 64 = 5 x 96
  static constexpr int kRegsPromotion = 104, kRegsOther = 64;
  static constexpr int kBoxBytes = 32 * kCols * 2;             // a warp's 32 rows of 16-bit output
  static constexpr int kStagingBytes = 16 * kBoxBytes;
  static constexpr int kBlocks = BN == 128 ? 1 : 2;            // 128-column scale blocks a tile touches
  static constexpr int kScaleSlots = 2, kScaleSlotBytes = kBlocks * 128 * 16;  // blocks x rows x four K blocks
  static constexpr int kTmemCols = 512;
  static constexpr int kFixed = kStagingBytes + kScaleSlots * kScaleSlotBytes + 1024 + 256;
  // as many stages as fit: 3 (single CTAs), 4, 6 and 7 (pairs, 256 / 192 / 128 wide)
  static constexpr int kFit = (232448 - kFixed) / (kStageA + kStageB), kStages = kFit < 8 ? kFit : 8;
  static constexpr size_t kSmemBytes = (size_t)kStages * (kStageA + kStageB) + kFixed;
};

// The weights that CTA `rank` of pair `pair` loads first, a row per thread.
template <int CTAS, int BN>
__device__ __forceinline__ void prefetch_first_weights(const GemmParams& p, int pair, int rank) {
  const int t = fast_div(pair, p.k_splits_div), ks = pair - t * p.k_splits, kb0 = ks * p.kb_per_split;
  int mt, nt;
  tile_coords(t, p.m_tiles, p.n_tiles, p.group_m, p.per_group_div, mt, nt);
  const int row = nt * BN + rank * (BN / CTAS) + (int)threadIdx.x;
  if (t < p.m_tiles * p.n_tiles && row < p.N)
    prefetch_weight_row(p.w + (int64_t)row * p.K + (int64_t)kb0 * kBK, min(kPrefetchKb, min(p.num_kb, kb0 + p.kb_per_split) - kb0));
}

// OutT: 16-bit output [M, N], or fp32 (C + split * split_stride: partial sums of a K split, or an fp32 result)
// CS > 0: the K splits of a tile, CS of them (2 or 4), are one cluster. Each of them sums and stores its share of the columns; the
// others hand theirs over through distributed shared memory, in the ring, which is idle by then: 32 or 48 of the 64 KB that a CTA holds, and no
// fp32 partials in memory nor a reduction launch: 203 x 4096 x 4096 12.5 us unsplit -> 10.3 in two splits, 203 x 4096 x 14336 24.5
// with partials in memory -> 19.7.
template <int CTAS, int BN, int CS, typename OutT>
__global__ void __cluster_dims__(CTAS * (CS ? CS : 1), 1, 1) __launch_bounds__(Wide<CTAS, BN>::kThreads, 1)
block_fp8_gemm_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                           const __grid_constant__ CUtensorMap tmap_c, const GemmParams p) {
  using Cfg = Wide<CTAS, BN>;
  constexpr bool CSUM = CS > 0;
  constexpr int S = Cfg::kStages, NB = Cfg::kAccBufs, SQ = Cfg::kScaleSlots, kRows = CTAS * kBM;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t sA = smem_base;
  const uint32_t sB = smem_base + S * Cfg::kStageA;
  const uint32_t staging = smem_base + S * (Cfg::kStageA + Cfg::kStageB);
  float* scales = reinterpret_cast<float*>(smem_al + (size_t)S * (Cfg::kStageA + Cfg::kStageB) + Cfg::kStagingBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(scales) + SQ * Cfg::kScaleSlotBytes);
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
  auto tfull_bar = [&](int b) { return bar0 + 8u * (2 * S + b); };
  auto tempty_bar = [&](int b) { return bar0 + 8u * (2 * S + NB + b); };
  auto sfull_bar = [&](int q) { return bar0 + 8u * (2 * S + 2 * NB + q); };
  auto sempty_bar = [&](int q) { return bar0 + 8u * (2 * S + 2 * NB + SQ + q); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 2 * NB + 2 * SQ);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * S + 2 * NB + 2 * SQ + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t cluster_rank = CTAS == 2 || CSUM ? ptx::cluster_ctarank() : 0;
  // rank in the pair, and the pair's leader in the cluster (a constant where it can be one: it is on the MMA warp's trip)
  const uint32_t rank = CSUM ? cluster_rank & (CTAS - 1) : cluster_rank, leader_rank = CSUM ? cluster_rank - rank : 0u;
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar(s), CTAS);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < NB; ++b) {
      ptx::mbar_init(tfull_bar(b), 1);
      ptx::mbar_init(tempty_bar(b), CTAS * Cfg::kPromWarps);
    }
    for (int q = 0; q < SQ; ++q) {
      ptx::mbar_init(sfull_bar(q), 2);
      ptx::mbar_init(sempty_bar(q), Cfg::kPromWarps);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == Cfg::kMmaWarp) {
    const uint32_t slot = ptx::smem_u32(const_cast<uint32_t*>(tmem_slot));
    if constexpr (CTAS == 2) {
      ptx::tmem_alloc_pair(slot, Cfg::kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(slot, Cfg::kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  if (warp == Cfg::kProducerWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_a);
    ptx::prefetch_tensormap(&tmap_b);
    ptx::prefetch_tensormap(&tmap_c);
  }
  ptx::tc_fence_before();
  ptx::wide_sync<CSUM ? 2 : CTAS>();  // the peer's barriers are initialised before anything signals them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  // What is read and overwritten below belongs to the kernels before, which may still run; the weights of the first K blocks are
  // asked for all the same, as a prefetch into L2, a row each.
  if (warp < Cfg::kPromWarps && (int)threadIdx.x < BN / CTAS) prefetch_first_weights<CTAS, BN>(p, blockIdx.x / CTAS, (int)rank);
  grid_dependency_wait();

  const int S_k = p.k_splits;
  const int total_items = p.m_tiles * p.n_tiles * S_k;
  const int num_kb = p.num_kb;
  const int pair = blockIdx.x / CTAS, npairs = gridDim.x / CTAS;
  struct Item {
    int mt, nt, ks, kb0, kb1;
  };
  auto item_of = [&](int item) {
    Item c;
    const int t = fast_div(item, p.k_splits_div);
    c.ks = item - t * S_k;
    c.kb0 = c.ks * p.kb_per_split;
    c.kb1 = min(num_kb, c.kb0 + p.kb_per_split);
    tile_coords(t, p.m_tiles, p.n_tiles, p.group_m, p.per_group_div, c.mt, c.nt);
    return c;
  };

  if (warp >= Cfg::kPromWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kRegsOther));
    if (warp == Cfg::kProducerWarp) {
      if (ptx::elect_one()) {  // -------------------------------------------------- TMA producer (both CTAs)
        int s = 0;
        uint32_t phase = 1;
        bool ok = true;
        for (int item = pair; item < total_items && ok; item += npairs) {
          const Item c = item_of(item);
          const int a_row = c.mt * kRows + (int)rank * kBM, b_row = c.nt * BN + (int)rank * (BN / CTAS);
          for (int kb = c.kb0; kb < c.kb1; ++kb) {
            ok = ptx::mbar_wait(empty_bar(s), phase, abort_flag);
            if (!ok) break;
            uint32_t lf = full_bar(s);
            if constexpr (CTAS == 2) {
              lf = ptx::mapa(lf, leader_rank);
              ptx::mbar_expect_tx_cluster(lf, Cfg::kStageA + Cfg::kStageB);
            } else {
              ptx::mbar_expect_tx(lf, Cfg::kStageA + Cfg::kStageB);
            }
            ptx::wide_load<CTAS>(sA + s * Cfg::kStageA, &tmap_a, kb * kBK, a_row, lf);
            ptx::wide_load<CTAS>(sB + s * Cfg::kStageB, &tmap_b, kb * kBK, b_row, lf);
            if (++s == S) s = 0, phase ^= 1;
          }
        }
        // the leader's last arrivals on this CTA's empty barriers, before its shared memory may go
        for (int i = 0; i < S && ok; ++i) {
          ok = ptx::mbar_wait(empty_bar(s), phase, abort_flag);
          if (++s == S) s = 0, phase ^= 1;
        }
      }
      __syncwarp();
    } else if (warp == Cfg::kMmaWarp) {
      if (leader && ptx::elect_one()) {  // ------------------------------------------ MMA issuer (leader only)
        constexpr uint32_t idesc = ptx::idesc_e4m3_f32(kRows, BN);
        const uint64_t da0 = ptx::smem_desc_sw128(sA), db0 = ptx::smem_desc_sw128(sB);
        int s = 0, b = 0;
        uint32_t phase = 0, tphase = 1;
        bool ok = true;
        for (int item = pair; item < total_items && ok; item += npairs) {
          const Item c = item_of(item);
#pragma unroll 1
          for (int n = c.kb1 - c.kb0; n > 0; --n) {
            ok = ptx::mbar_wait2(full_bar(s), phase, tempty_bar(b), tphase, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after();
            // a stage further = its bytes >> 4 in the address field, which does not overflow: shared memory ends below 2^18
            const uint64_t da = da0 + (uint32_t)(s * (Cfg::kStageA >> 4)), db = db0 + (uint32_t)(s * (Cfg::kStageB >> 4));
            const uint32_t d = tmem_base + b * Cfg::kAccStride;
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k) ptx::wide_mma<CTAS>(d, da + 2 * k, db + 2 * k, idesc, k > 0);
            if constexpr (CTAS == 2) {
              ptx::mma_commit_pair_multicast(tfull_bar(b), (uint16_t)(3u << leader_rank));
              ptx::mma_commit_pair_multicast(empty_bar(s), (uint16_t)(3u << leader_rank));
            } else {
              ptx::mma_commit(tfull_bar(b));
              ptx::mma_commit(empty_bar(s));
            }
            if (++b == NB) b = 0, tphase ^= 1;
            if (++s == S) s = 0, phase ^= 1;
          }
        }
      }
      __syncwarp();
    } else {  // ------------------------------------------------------------------ scale loaders (both CTAs)
      const int tid = threadIdx.x - Cfg::kScaleWarp * 32;  // 0..63: rows tid and tid + 64
      int q = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int item = pair; item < total_items && ok; item += npairs) {
        const Item c = item_of(item);
        const int row = c.mt * kRows + (int)rank * kBM + tid;
        const float* as0 = p.As + (int64_t)min(row, p.M - 1) * p.as_sm;
        const float* as1 = p.As + (int64_t)min(row + 64, p.M - 1) * p.as_sm;
        const int blk0 = c.nt * BN / 128;  // first scale block of the tile
        for (int kbase = c.kb0; kbase < c.kb1; kbase += 4) {
          float a[4][2], b[4][Cfg::kBlocks];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int kb = min(kbase + j, c.kb1 - 1);
            a[j][0] = __ldg(as0 + (int64_t)kb * p.as_sk);
            a[j][1] = __ldg(as1 + (int64_t)kb * p.as_sk);
#pragma unroll
            for (int n = 0; n < Cfg::kBlocks; ++n)
              b[j][n] = __ldg(p.Bs + (int64_t)min(blk0 + n, p.n_blocks - 1) * num_kb + kb);
          }
          ok = ptx::mbar_wait(sempty_bar(q), phase, abort_flag);
          if (!ok) break;
          float* dst = scales + q * (Cfg::kScaleSlotBytes / 4) + tid * 4;  // [block][row][K block]
#pragma unroll
          for (int n = 0; n < Cfg::kBlocks; ++n) {
            *reinterpret_cast<float4*>(dst + n * 512) =
                make_float4(a[0][0] * b[0][n], a[1][0] * b[1][n], a[2][0] * b[2][n], a[3][0] * b[3][n]);
            *reinterpret_cast<float4*>(dst + n * 512 + 256) =
                make_float4(a[0][1] * b[0][n], a[1][1] * b[1][n], a[2][1] * b[2][n], a[3][1] * b[3][n]);
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(sfull_bar(q));
          if (++q == SQ) q = 0, phase ^= 1;
        }
      }
      __syncwarp();
    }
  } else {
    // -------------------------------------------------------------------- promotion warps (both CTAs)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::kRegsPromotion));
    const int quarter = warp & 3, colq = warp >> 2;
    constexpr int kCols = Cfg::kCols, CH = Cfg::kChunks;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + colq * kCols;
    const uint32_t my_scales = ptx::smem_u32(scales) + (quarter * 32 + lane) * 16;
    const uint32_t leader_tempty = CTAS == 2 ? ptx::mapa(tempty_bar(0), leader_rank) : tempty_bar(0);
    uint32_t tphase = 0, sphase = 0;
    int q = 0, b = 0;
    bool ok = true;
    for (int item = pair; item < total_items && ok; item += npairs) {
      const Item c = item_of(item);
      // a 192-wide tile starts inside a scale block, so a warp's 16-column chunks may lie in two of them
      const int col_in_block = BN == 192 ? c.nt * BN % 128 + colq * kCols : colq * kCols;
      const int first_blk = col_in_block / 128;
      bool second[CH];
#pragma unroll
      for (int h = 0; h < CH; ++h) second[h] = BN == 192 && (col_in_block + 16 * h) / 128 != first_blk;
      uint64_t acc[kCols / 2];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) acc[j] = 0;
      for (int kbase = c.kb0; kbase < c.kb1 && ok; kbase += 4) {
        ok = ptx::mbar_wait(sfull_bar(q), sphase, abort_flag);
        const int n = min(4, c.kb1 - kbase);
#pragma unroll 2
        for (int j = 0; j < n && ok; ++j) {
          float sc1, sc2;  // scale in the warp's first scale block and in its second
          const uint32_t sa = my_scales + q * Cfg::kScaleSlotBytes + first_blk * 2048 + 4 * j;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(sc1) : "r"(sa) : "memory");
          if (BN == 192) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(sc2) : "r"(second[CH - 1] ? sa + 2048 : sa) : "memory");
          ok = ptx::mbar_wait(tfull_bar(b), tphase, abort_flag);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t sc = ptx::pack2(sc1);
          const uint32_t ta = lane_base + b * Cfg::kAccStride;
#pragma unroll
          for (int h = 0; h < CH; h += 2) {  // 32 columns, or the last 16
            uint32_t v[32];
            if (CH - h >= 2) ptx::tmem_ld32(ta + 16 * h, v);
            else ptx::tmem_ld16(ta + 16 * h, v);
            ptx::tmem_ld_wait_all();
            if (h + 2 >= CH) {
              ptx::tc_fence_before();
              __syncwarp();
              if (ptx::elect_one()) {
                if constexpr (CTAS == 2) ptx::mbar_arrive_cluster(leader_tempty + 8 * b);
                else ptx::mbar_arrive(leader_tempty + 8 * b);
              }
              if (++b == NB) b = 0, tphase ^= 1;
            }
#pragma unroll
            for (int i = 0; i < (CH - h >= 2 ? 2 : 1); ++i) {
              const uint64_t sch = BN == 192 && second[h + i] ? ptx::pack2(sc2) : sc;
#pragma unroll
              for (int k = 0; k < 8; ++k) ptx::ffma2(acc[8 * (h + i) + k], v[16 * i + 2 * k], v[16 * i + 2 * k + 1], sch);
            }
          }
        }
        __syncwarp();
        if (ptx::elect_one()) ptx::mbar_arrive(sempty_bar(q));
        if (++q == SQ) q = 0, sphase ^= 1;
      }
      if (!CSUM && !ok) break;
      const uint32_t wstage = staging + warp * Cfg::kBoxBytes;
      const int row0 = c.mt * kRows + (int)rank * kBM + quarter * 32, col0 = c.nt * BN + colq * kCols;
      if constexpr (CSUM) {  // the only item of this CTA; a warp whose wait gave up takes part all the same
        constexpr int G = kCols / 8;  // groups of 8 columns; split s owns G / S_k of them
        constexpr int per = G / (CSUM ? CS : 1);
        const int me = c.ks;
        __syncwarp();
        ptx::cluster_sync();  // every ring is idle
        auto slot = [&](uint32_t base, int src, int g, int half) {
          return base + (uint32_t)(((src * per + g % per) * 2 + half) * Cfg::kPromWarps * 32 + (int)threadIdx.x) * 16;
        };
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int owner = g / per;
          if (owner == me) continue;
          const uint32_t base = ptx::mapa(smem_base, (uint32_t)owner * CTAS + rank);
          ptx::st_cluster_2x64(slot(base, me, g, 0), acc[4 * g], acc[4 * g + 1]);
          ptx::st_cluster_2x64(slot(base, me, g, 1), acc[4 * g + 2], acc[4 * g + 3]);
        }
        __syncwarp();
        ptx::cluster_sync();
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if (g / per != me) continue;
          uint64_t sum[4] = {0, 0, 0, 0};
          for (int src = 0; src < CS; ++src) {  // split order: the same sum on every run
            uint64_t v[4] = {acc[4 * g], acc[4 * g + 1], acc[4 * g + 2], acc[4 * g + 3]};
            if (src != me) {
              ptx::lds_2x64(slot(smem_base, src, g, 0), v[0], v[1]);
              ptx::lds_2x64(slot(smem_base, src, g, 1), v[2], v[3]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i] = ptx::fadd2(sum[i], v[i]);
          }
          float t[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = __uint_as_float((uint32_t)(sum[i / 2] >> (32 * (i & 1))));
          if (ok && row0 + lane < p.M && col0 + g * 8 < p.N)
            store8<OutT>(static_cast<OutT*>(p.C) + (int64_t)(row0 + lane) * p.ldc + col0 + g * 8, t);
        }
        break;
      }

      // ------------------------------------------------------------------------ tile epilogue
      if constexpr (sizeof(OutT) == 2) {
        if (lane == 0) ptx::tma_store_wait_read();  // the last tile's box has left the staging area
        __syncwarp();
#pragma unroll
        for (int ch = 0; ch < kCols / 8; ++ch) {
          float t[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = __uint_as_float((uint32_t)(acc[(ch * 8 + i) / 2] >> (32 * (i & 1))));
          const uint4 v = pack8<OutT>(t);
          // a 64-column box is stored with the TMA 128-byte swizzle; narrower ones row by row
          const uint32_t addr = wstage + lane * kCols * 2 + ((kCols == 64 ? ch ^ (lane & 7) : ch) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                       : "memory");
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (col0 < p.N && row0 < p.M) ptx::tma_store_3d(&tmap_c, wstage, col0, row0, 0);
          ptx::tma_store_commit();
        }
      } else {
        if (row0 + lane < p.M) {
          OutT* dst = static_cast<OutT*>(p.C) + c.ks * p.split_stride + (int64_t)(row0 + lane) * p.ldc + col0;
#pragma unroll
          for (int ch = 0; ch < kCols / 8; ++ch) {
            float t[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = __uint_as_float((uint32_t)(acc[(ch * 8 + i) / 2] >> (32 * (i & 1))));
            if (col0 + ch * 8 < p.N) store8<OutT>(dst + ch * 8, t);
          }
        }
      }
    }
    if (sizeof(OutT) == 2 && lane == 0) ptx::tma_store_wait_all();
  }
  if (CSUM && warp >= Cfg::kPromWarps) {  // the other warps' share of the two cluster barriers above
    __syncwarp();
    ptx::cluster_sync();
    ptx::cluster_sync();
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_flag) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  ptx::tc_fence_before();
  ptx::wide_sync<CSUM ? 2 : CTAS>();  // neither CTA leaves while the other may still signal its barriers or use its smem
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(p.status, 0, 1);
  if (warp == Cfg::kMmaWarp) {
    ptx::tc_fence_after();
    if constexpr (CTAS == 2) ptx::tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    else ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// p.M/N/K/As/Bs/C/ldc (and split_stride) filled by the caller.
template <int CTAS, int BN, int CS, typename OutT>
inline int launch_gemm_wide(const void* A, const void* B, GemmParams p, int k_splits, cudaStream_t st) {
  p.num_kb = (int)cdiv(p.K, kBK);
  p.n_blocks = (int)cdiv(p.N, 128);
  p.n_tiles = (int)cdiv(p.N, BN);
  p.m_tiles = (int)cdiv(p.M, CTAS * kBM);
  p.group_m = row_group(p.M, p.K, CTAS * kBM);
  p.k_splits = k_splits;
  p.kb_per_split = (int)cdiv(p.num_kb, k_splits);
  p.per_group_div = make_fastdiv(p.group_m * p.n_tiles);
  p.k_splits_div = make_fastdiv(p.k_splits);
  p.w = static_cast<const uint8_t*>(B);
  p.status = device_status_word();
  if (!p.status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  const int64_t items = (int64_t)p.m_tiles * p.n_tiles * p.k_splits;
  if (items == 0) return B200_OK;
  const int slots = sm_count() / CTAS;
  const int units = (int)(CS > 0 || items < slots ? items : slots);
  CUtensorMap ta, tb, tc;
  int rc = make_tmap_u8(&ta, A, (uint64_t)p.M, (uint64_t)p.K, kBM, "A");
  if (rc) return rc;
  rc = make_tmap_u8(&tb, B, (uint64_t)p.N, (uint64_t)p.K, BN / CTAS, "B");
  if (rc) return rc;
  tc = ta;
  if (sizeof(OutT) == 2 && CS == 0) {
    rc = make_tmap_out(&tc, p.C, 1, (uint64_t)p.M, (uint64_t)p.N, 2, std::is_same<OutT, __nv_bfloat16>::value, "C", BN / 4);
    if (rc) return rc;
  }
  auto k = block_fp8_gemm_wide_kernel<CTAS, BN, CS, OutT>;
  if (int rc_smem = allow_smem(k, Wide<CTAS, BN>::kSmemBytes, "block_fp8_gemm_wide_kernel")) return rc_smem;
  return launch_dependent(k, dim3((unsigned)(CTAS * units)), Wide<CTAS, BN>::kThreads, Wide<CTAS, BN>::kSmemBytes, st, 1,
                          "block_fp8_gemm_wide_kernel", ta, tb, tc, p);
}
// bn: columns of a pair's tile, or 0: single CTAs. csum: the K splits (2 or 4) are summed within clusters (128-wide pairs).
template <typename OutT>
inline int launch_gemm_wide(int bn, const void* A, const void* B, const GemmParams& p, int k_splits, bool csum, cudaStream_t st) {
  if (csum) {
    B200_UNSUPPORTED(bn != 128 || (k_splits != 2 && k_splits != 4), "gemm: clusters sum 2 or 4 K splits of 128-wide pairs, not %d of %d",
                     k_splits, bn);
    return k_splits == 2 ? launch_gemm_wide<2, 128, 2, OutT>(A, B, p, 2, st) : launch_gemm_wide<2, 128, 4, OutT>(A, B, p, 4, st);
  }
  if (bn == 0) return launch_gemm_wide<1, 256, 0, OutT>(A, B, p, k_splits, st);
  if (bn == 128) return launch_gemm_wide<2, 128, 0, OutT>(A, B, p, k_splits, st);
  if (bn == 192) return launch_gemm_wide<2, 192, 0, OutT>(A, B, p, k_splits, st);
  return launch_gemm_wide<2, 256, 0, OutT>(A, B, p, k_splits, st);
}

}  // namespace b200
