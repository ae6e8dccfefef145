// Block-scaled GEMM (see gemm_ue8m0.cuh) on CTA pairs: a 256 x 240 tile per pair, each CTA with its own 128 rows of A and
// half of B's rows, so a K block moves 31 KB into a CTA's shared memory instead of 44 KB for 128 x 224 columns, and the
// tensor core reads as much less back. Two accumulator stages of 240 columns and the scale columns (2 x 4 for A, 2 x 8
// for B) fill 504 of the 512 TMEM columns. Every CTA's scale loader stages the words of its own rows of A and of all 240
// columns of B; the leader's tcgen05.cp.cta_group::2 copies them from each CTA's shared memory into its TMEM.
#pragma once

#include "gemm_pair.cuh"
#include "gemm_ue8m0.cuh"

namespace b200 {

struct Ue8m0PairCfg {
  static constexpr int BN = 240;
  static constexpr int kStages = 6;
  static constexpr int kStageA = kBM * kBK;       // 16 KB
  static constexpr int kStageB = (BN / 2) * kBK;  // 15 KB
  static constexpr int kSfSlots = 4, kSfSlotBytes = 512 + 1024;
  static constexpr int kThreads = 384;
  static constexpr int kEpiWarps = 8, kProducerWarp = 8, kMmaWarp = 9, kSfWarp = 10;
  static constexpr int kAccCols = BN;
  static constexpr int kSfaCol = 2 * BN;      // 480: two buffers of 4 columns
  static constexpr int kSfbCol = 2 * BN + 8;  // 488: two buffers of 8 columns
  static constexpr int kTmemCols = 512;
  static constexpr size_t kSmemBytes = (size_t)kStages * (kStageA + kStageB) + kSfSlots * kSfSlotBytes + 1024 + 256;
};

namespace ptx {
__device__ __forceinline__ void mma_f8_block_scaled_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                         uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t"
      "}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}
__device__ __forceinline__ void tmem_cp_32x128b_warpx4_pair(uint32_t taddr, uint64_t smem_desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(smem_desc) : "memory");
}
__device__ __forceinline__ void mma_commit_pair_both(uint32_t bar) { mma_commit_pair_multicast(bar, (uint16_t)3); }
__device__ __forceinline__ void mbar_arrive_cluster_release(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
}  // namespace ptx

template <typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Ue8m0PairCfg::kThreads, 1)
block_fp8_gemm_ue8m0_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                            const Ue8m0Params p) {
  using Cfg = Ue8m0PairCfg;
  constexpr int S = Cfg::kStages, BN = Cfg::BN, SFS = Cfg::kSfSlots;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t sA = smem_base;
  const uint32_t sB = smem_base + S * Cfg::kStageA;
  const uint32_t sSF = smem_base + S * (Cfg::kStageA + Cfg::kStageB);
  uint8_t* sSF_ptr = smem_al + (size_t)S * (Cfg::kStageA + Cfg::kStageB);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sSF_ptr + SFS * Cfg::kSfSlotBytes);
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
  auto sf_full_bar = [&](int s) { return bar0 + 8u * (2 * S + s); };
  auto sf_empty_bar = [&](int s) { return bar0 + 8u * (2 * S + SFS + s); };
  auto acc_full_bar = [&](int a) { return bar0 + 8u * (2 * S + 2 * SFS + a); };
  auto acc_empty_bar = [&](int a) { return bar0 + 8u * (2 * S + 2 * SFS + 2 + a); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 2 * SFS + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * S + 2 * SFS + 5);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar(s), 2);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < SFS; ++s) {
      ptx::mbar_init(sf_full_bar(s), 2);
      ptx::mbar_init(sf_empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(acc_full_bar(a), 1);
      ptx::mbar_init(acc_empty_bar(a), 2 * Cfg::kEpiWarps);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == Cfg::kMmaWarp) {
    ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  if (warp == Cfg::kProducerWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_a);
    ptx::prefetch_tensormap(&tmap_b);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // the peer's barriers are initialised before anything signals them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  grid_dependency_wait();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  const int total_tiles = p.m_tiles * p.n_tiles;
  const int num_kb = p.num_kb;
  const int groups = (num_kb + 3) / 4;  // scale groups (four K blocks each) per tile

  if (warp == Cfg::kProducerWarp) {
    if (ptx::elect_one()) {
      // ------------------------------------------------------------------ TMA producer
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += npairs) {
        int mt, nt;
        tile_coords(t, p.m_tiles, p.n_tiles, p.group_m, p.per_group_div, mt, nt);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % S;
          ok = ptx::mbar_wait(empty_bar(s), ((it / S) & 1) ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t lf = ptx::mapa(full_bar(s), 0);
          ptx::mbar_expect_tx_cluster(lf, Cfg::kStageA + Cfg::kStageB);
          ptx::tma_load_2d_pair(sA + s * Cfg::kStageA, &tmap_a, kb * kBK, mt * 2 * kBM + (int)rank * kBM, lf);
          ptx::tma_load_2d_pair(sB + s * Cfg::kStageB, &tmap_b, kb * kBK, nt * BN + (int)rank * (BN / 2), lf);
        }
      }
    }
    __syncwarp();
  } else if (warp >= Cfg::kSfWarp) {
    // ------------------------------------------------------------------ scale loader
    // Atom layout expected by the 32x128b.warpx4 copy: row r of a 128-row atom at byte (r % 32) * 16 + (r / 32) * 4.
    // Lane l therefore holds rows l, 32 + l, 64 + l, 96 + l and writes one 16-byte vector. Two warps take turns, each
    // with the words of its next group in flight while it stores this one: with one warp and no prefetch the L2 round
    // trip of every group paced the tensor core (a CTA pair waited 548 of 943 clocks per K block for scales).
    constexpr int32_t kOne = 0x7F7F7F7F;  // exponent 127 = 2^0 for rows past the edge (their data is zero-filled)
    int t = pair, g = warp - Cfg::kSfWarp;
    auto advance = [&](int by) {
      for (g += by; g >= groups; g -= groups) t += npairs;
    };
    int32_t wa[4], wb[8];
    auto fetch = [&]() {
      int mt, nt;
      tile_coords(t, p.m_tiles, p.n_tiles, p.group_m, p.per_group_div, mt, nt);
      const int m0 = mt * 2 * kBM + (int)rank * kBM, n0 = nt * BN;  // its own rows of A, all columns of the tile
      const int32_t* ga = p.sfa + (int64_t)g * p.sfa_ld;
      const int32_t* gb = p.sfb + (int64_t)g * p.sfb_ld;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = m0 + 32 * j + lane;
        wa[j] = r < p.M ? __ldg(ga + r) : kOne;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = n0 + 32 * j + lane;
        wb[j] = (32 * j < BN && r < p.N) ? __ldg(gb + (p.sfb_rows_per_word == 1 ? r : r / 128)) : kOne;
      }
    };
    advance(0);
    if (t < total_tiles) fetch();
    for (uint32_t gi = warp - Cfg::kSfWarp; t < total_tiles; gi += 2) {
      const int slot = gi % SFS;
      const int4 va = make_int4(wa[0], wa[1], wa[2], wa[3]), vb = make_int4(wb[0], wb[1], wb[2], wb[3]),
                 vc = make_int4(wb[4], wb[5], wb[6], wb[7]);
      if (!ptx::mbar_wait(sf_empty_bar(slot), ((gi / SFS) & 1) ^ 1, abort_flag)) break;
      uint8_t* dst = sSF_ptr + (size_t)slot * Cfg::kSfSlotBytes + lane * 16;
      *reinterpret_cast<int4*>(dst) = va;
      *reinterpret_cast<int4*>(dst + 512) = vb;
      *reinterpret_cast<int4*>(dst + 1024) = vc;
      advance(2);
      if (t < total_tiles) fetch();  // in flight across the fence, the arrival and the next wait
      ptx::fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's copy
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster_release(ptx::mapa(sf_full_bar(slot), 0));
    }
    __syncwarp();
  } else if (warp == Cfg::kMmaWarp) {
    if (leader && ptx::elect_one()) {
      // ------------------------------------------------------- MMA issuer (leader only)
      constexpr uint32_t idesc0 = ptx::idesc_e4m3_block_scaled(2 * kBM, BN);
      uint32_t it = 0, gi = 0, tile_no = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += npairs, ++tile_no) {
        const int as = tile_no & 1;
        ok = ptx::mbar_wait(acc_empty_bar(as), ((tile_no >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        const uint32_t d = tmem_base + as * Cfg::kAccCols;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % S;
          if ((kb & 3) == 0) {
            // scales of the next four K blocks: three 512-byte atoms into the scale columns of buffer gi & 1
            const int slot = gi % SFS;
            ok = ptx::mbar_wait(sf_full_bar(slot), (gi / SFS) & 1, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t src = sSF + slot * Cfg::kSfSlotBytes;
            const uint32_t buf = gi & 1;
            ptx::tmem_cp_32x128b_warpx4_pair(tmem_base + Cfg::kSfaCol + buf * 4, ptx::smem_desc_sf_atom(src));
            ptx::tmem_cp_32x128b_warpx4_pair(tmem_base + Cfg::kSfbCol + buf * 8, ptx::smem_desc_sf_atom(src + 512));
            ptx::tmem_cp_32x128b_warpx4_pair(tmem_base + Cfg::kSfbCol + buf * 8 + 4, ptx::smem_desc_sf_atom(src + 1024));
            ptx::mma_commit_pair_both(sf_empty_bar(slot));  // the slot is free once the copies have read it
            ++gi;
          }
          ok = ptx::mbar_wait(full_bar(s), (it / S) & 1, abort_flag);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t da = ptx::smem_desc_sw128(sA + s * Cfg::kStageA);
          const uint64_t db = ptx::smem_desc_sw128(sB + s * Cfg::kStageB);
          const uint32_t buf = (gi - 1) & 1, byte = kb & 3;
          const uint32_t idesc = idesc0 | (byte << 4) | (byte << 29);  // scale byte of this K block, for A and B
          const uint32_t tsfa = tmem_base + Cfg::kSfaCol + buf * 4;
          const uint32_t tsfb = tmem_base + Cfg::kSfbCol + buf * 8;
#pragma unroll
          for (int k = 0; k < kBK / 32; ++k)
            ptx::mma_f8_block_scaled_pair(d, da + 2 * k, db + 2 * k, idesc, tsfa, tsfb, (kb > 0 || k > 0) ? 1u : 0u);
          ptx::mma_commit_pair_both(empty_bar(s));  // stage free once these MMAs have read it
          if (kb == num_kb - 1) ptx::mma_commit_pair_both(acc_full_bar(as));  // the tile's accumulator is complete
        }
      }
    }
    __syncwarp();
  } else if (warp < Cfg::kEpiWarps) {
    // ------------------------------------------------------------------- epilogue warps
    const int quarter = warp & 3, half = warp >> 2;  // TMEM lanes 32*quarter.., columns BN/2*half..
    const uint32_t leader_acc_empty = ptx::mapa(acc_empty_bar(0), 0);
    uint32_t tile_no = 0;
    bool ok = true;
    for (int t = pair; t < total_tiles && ok; t += npairs, ++tile_no) {
      int mt, nt;
      tile_coords(t, p.m_tiles, p.n_tiles, p.group_m, p.per_group_div, mt, nt);
      const int as = tile_no & 1;
      ok = ptx::mbar_wait(acc_full_bar(as), (tile_no >> 1) & 1, abort_flag);
      if (!ok) break;
      ptx::tc_fence_after();
      const int row = mt * 2 * kBM + (int)rank * kBM + quarter * 32 + lane;
      const int col0 = nt * BN + half * (BN / 2);
      const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16) + as * Cfg::kAccCols + half * (BN / 2);
      OutT* out = static_cast<OutT*>(p.C) + (int64_t)row * p.N + col0;
#pragma unroll 1
      for (int c = 0; c < BN / 2; c += 16) {
        uint32_t v[32];
        ptx::tmem_ld16(ta + c, v);
        ptx::tmem_ld_wait16(v);
        if (row < p.M) {
          float f[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
          if (col0 + c < p.N) store8<OutT>(out + c, f);
          if (c + 8 < BN / 2 && col0 + c + 8 < p.N) store8<OutT>(out + c + 8, f + 8);
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(leader_acc_empty + 8 * as);
    }
  }

  if (*abort_flag) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // neither CTA leaves while the other may still signal its barriers or read its smem
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(p.status, 0, 1);
  if (warp == Cfg::kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
  }
}

template <typename OutT>
inline int launch_gemm_ue8m0_pair(const void* A, const void* B, Ue8m0Params p, cudaStream_t st) {
  using Cfg = Ue8m0PairCfg;
  p.num_kb = (int)cdiv(p.K, kBK);
  p.m_tiles = (int)cdiv(p.M, 2 * kBM);
  p.n_tiles = (int)cdiv(p.N, Cfg::BN);
  p.group_m = row_group(p.M, p.K, 2 * kBM);
  p.per_group_div = make_fastdiv(p.group_m * p.n_tiles);
  p.status = device_status_word();
  if (!p.status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
  if (tiles == 0) return B200_OK;
  const int max_pairs = sm_count() / 2;
  const int pairs = (int)(tiles < max_pairs ? tiles : max_pairs);
  CUtensorMap ta, tb;
  int rc = make_tmap_u8(&ta, A, (uint64_t)p.M, (uint64_t)p.K, kBM, "A");
  if (rc) return rc;
  rc = make_tmap_u8(&tb, B, (uint64_t)p.N, (uint64_t)p.K, (uint32_t)(Cfg::BN / 2), "B (half of 240 rows)");
  if (rc) return rc;
  auto k = block_fp8_gemm_ue8m0_pair_kernel<OutT>;
  if (int rc_smem = allow_smem(k, Cfg::kSmemBytes, "block_fp8_gemm_ue8m0_pair_kernel")) return rc_smem;
  return launch_dependent(k, dim3((unsigned)(2 * pairs)), Cfg::kThreads, Cfg::kSmemBytes, st, 1, "block_fp8_gemm_ue8m0_pair_kernel",
                          ta, tb, p);
}

}  // namespace b200
