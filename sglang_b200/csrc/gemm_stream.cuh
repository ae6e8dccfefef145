// Weight-streaming block-FP8 GEMM for few rows per weight matrix (decode): bound by reading the weights from HBM.
//
// Operands are swapped: 128 weight rows fill the UMMA M dimension and NT = 16 / 32 / 64 tokens are its N, so a K
// block costs NT columns of TMEM traffic and NT FMAs per thread instead of the 256 of the 128-row token tile
// (gemm_kernel.cuh), and no A tile of padding rows is loaded or multiplied. A CTA owns 256 weight rows (two UMMA
// tiles): the gate rows and the up rows of one 128-wide output group, or 256 output columns.
//
// One persistent CTA per SM. The producer's ring (32 KB of weights + NT x 128 B of tokens per K block, as many
// stages as shared memory holds) runs across work items, so the weight stream does not stop for the scales of the
// next item or the epilogue of the last one. With fewer items than SMs, K is split over a thread-block cluster
// instead (one item per cluster) and the partial sums go to the first CTA through distributed shared memory.
//   warps 0-3  promotion of the first 128 rows (lane = weight row, columns = tokens), warps 4-7 of the second
//   warp  8    TMA producer          warp 9  MMA issuer
//   warps 10, 11  scale tables, ids and router weights of the next item into the other of two table buffers: loaded
//              by the promotion warps at the start of an item they stopped the weight stream for the L2 round trips
#pragma once

#include "gemm_host.cuh"

namespace b200 {

enum { STREAM_GATE_UP = 1, STREAM_DOWN = 2 };

struct StreamParams {
  const float* As;  // scales of the sorted token rows: As[kb * as_ld + row]
  int64_t as_ld;
  const float* Bs;  // [experts][row blocks][num_kb]
  int num_kb, kb_per_rank;  // K blocks per cluster rank
  int n_out;                // gate_up: intermediate size I; down: hidden size H
  int n_tiles;              // 256-row weight tiles per expert
  const int32_t* expert_ids;    // [blocks] expert of every NT-row block, -1 = skip
  const int32_t* num_post_pad;  // [1] live rows (a multiple of NT)
  const int32_t* sorted_ids;    // [rows] flat (token * topk + slot), >= numel = pad
  const float* topk_weights;    // router weight per flat index, or null
  int numel, max_blocks, experts;
  const uint8_t* w;  // the stacked weights, rows of num_kb * 128 bytes
  void* C;  // down: OutT [numel][n_out]
  uint8_t* q_out;   // gate_up: FP8 [rows][n_out] and its scales q_scales[(n / 128) * q_ld + row]
  float* q_scales;
  int64_t q_ld;
  int stages, table_kb;  // ring depth; K blocks the scale table holds
  int* status;
};

template <int NT>
struct StreamCfg {
  static constexpr int kThreads = 384;
  static constexpr int kStageW = 256 * kBK, kStageX = NT * kBK, kStage = kStageW + kStageX;
  static constexpr int kAccBufs = 4;  // the tensor core runs this many K blocks ahead of the promotion warps
  static constexpr int kTmemCols = kAccBufs * 2 * NT;
  // behind the ring: barriers, exchange area (the other half's gate / up values), partial row amax, then two buffers
  // of [ids of the rows][their router weights][scale table [kb][NT]][weight-block scales [2][kb]], sized by the K
  // blocks of one CTA
  static constexpr int kExch = NT * 128 * 4, kPart = 4 * NT * 4;
  static constexpr int kFixed = 256 + kExch + kPart + 1024;
  static constexpr int kMaxStages = 8, kSmemLimit = 232448;
  __host__ __device__ static constexpr int table_bytes(int table_kb) { return 2 * NT * 4 + table_kb * NT * 4 + (table_kb * 8 + 15) / 16 * 16; }
  static int stages_for(int table_kb) {
    const int s = (kSmemLimit - kFixed - 2 * table_bytes(table_kb)) / kStage;
    return s < kMaxStages ? s : kMaxStages;
  }
  static size_t smem_for(int stages, int table_kb) { return (size_t)stages * kStage + kFixed + 2 * (size_t)table_bytes(table_kb); }
};

namespace ptx {
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
}  // namespace ptx

// Barrier of `threads` threads that tells all of them whether any of them passed true.
__device__ __forceinline__ bool named_bar_any(int id, int threads, bool mine) {
  uint32_t any;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "bar.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}"
      : "=r"(any)
      : "r"(id), "r"(threads), "r"((uint32_t)mine)
      : "memory");
  return any != 0;
}

template <int NT, int STAGE, typename OutT>
__global__ void __launch_bounds__(StreamCfg<NT>::kThreads, 1)
stream_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const StreamParams p) {
  using Cfg = StreamCfg<NT>;
  constexpr int NB = Cfg::kAccBufs;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const int S = p.stages;
  const uint32_t sW = smem_base, sX = smem_base + S * Cfg::kStageW;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_al + (size_t)S * Cfg::kStage);
  float* exch = reinterpret_cast<float*>(bars + 32);   // [NT][128]
  float* part = exch + NT * 128;                       // [4][NT]
  uint8_t* tables = reinterpret_cast<uint8_t*>(part + 4 * NT);
  const int table_bytes = Cfg::table_bytes(p.table_kb);
  auto row_id_of = [&](int buf) { return reinterpret_cast<int*>(tables + buf * table_bytes); };           // [NT] flat ids
  auto row_w_of = [&](int buf) { return reinterpret_cast<float*>(tables + buf * table_bytes) + NT; };     // [NT] weights
  auto table_of = [&](int buf) { return reinterpret_cast<float*>(tables + buf * table_bytes) + 2 * NT; };  // [kb][NT]
  auto bs_tab_of = [&](int buf) { return table_of(buf) + p.table_kb * NT; };                               // [2][kb]
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (8 + s); };
  auto tfull_bar = [&](int b) { return bar0 + 8u * (16 + b); };
  auto tempty_bar = [&](int b) { return bar0 + 8u * (16 + NB + b); };
  auto tab_full_bar = [&](int b) { return bar0 + 8u * (16 + 2 * NB + b); };
  auto tab_empty_bar = [&](int b) { return bar0 + 8u * (18 + 2 * NB + b); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 20 + 2 * NB);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 20 + 2 * NB + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducerWarp = 8, kMmaWarp = 9;
  uint32_t rank, csize;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < NB; ++b) {
      ptx::mbar_init(tfull_bar(b), 1);
      ptx::mbar_init(tempty_bar(b), 8);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tab_full_bar(b), 2);
      ptx::mbar_init(tab_empty_bar(b), 8);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  if (warp == kProducerWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int item0 = csize == 1 ? blockIdx.x : blockIdx.x / csize;
  const int step = csize == 1 ? gridDim.x : gridDim.x / csize;
  const int kb0 = (int)rank * p.kb_per_rank, kb1 = min(p.num_kb, kb0 + p.kb_per_rank);
  const int nkb = max(kb1 - kb0, 0);
  // first weight row of half h of tile nt of expert e, and its 128-row scale block
  const int row_blocks = (p.n_out + 127) / 128;
  auto weight_row = [&](int e, int nt, int h) {
    return STAGE == STREAM_GATE_UP ? e * 2 * p.n_out + h * p.n_out + nt * 128 : e * p.n_out + nt * 256 + h * 128;
  };
  auto scale_row = [&](int e, int nt, int h) {
    return STAGE == STREAM_GATE_UP ? e * 2 * row_blocks + h * row_blocks + nt
                                   : e * row_blocks + min(nt * 2 + h, row_blocks - 1);
  };

  // Everything read below, and what the epilogue overwrites, belongs to the kernels before. The down GEMM's schedule was
  // written two kernels ago (gate_up lets this grid start after its own wait for it): while gate_up still runs, the
  // promotion warps ask for the first weight tiles, a row each. That is a prefetch into L2 and the id that picks the rows is
  // only a hint: nothing read before the wait is used after it.
  if (STAGE == STREAM_GATE_UP) {
    grid_dependency_wait();
    grid_launch_dependents();
  } else {
    grid_launch_dependents();
    if (warp < 8) {
      const int blk = item0 / p.n_tiles, nt = item0 - blk * p.n_tiles;
      int live, e;
      asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(live) : "l"(p.num_post_pad) : "memory");
      asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(e) : "l"(p.expert_ids + blk) : "memory");
      if (blk * NT < live && e >= 0 && e < p.experts && nt * 256 + (int)threadIdx.x < p.n_out)
        prefetch_weight_row(p.w + ((int64_t)weight_row(e, nt, 0) + threadIdx.x) * p.num_kb * kBK + kb0 * kBK, min(S, nkb));
    }
    grid_dependency_wait();
  }
  const int blocks = min(p.max_blocks, *p.num_post_pad / NT);
  const int total = blocks * p.n_tiles;

  float acc[NT];
  bool sum_ok = false;
  int my_block = -1, my_nt = 0, my_buf = 0;  // item whose sums acc holds

  // Work after the K loop of one item, by the eight promotion warps (256 threads, named barriers 1..3)
  const int half = warp >> 2, r = threadIdx.x & 127;
  auto epilogue = [&]() {
    const float* row_w = row_w_of(my_buf);
    const int* row_id = row_id_of(my_buf);
    const int row0 = my_block * NT;
    if constexpr (STAGE == STREAM_GATE_UP) {
      if (p.topk_weights != nullptr) {  // router weight on the fp32 product, before the activation
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] *= row_w[t];
      }
      // the gate warps finish tokens [0, NT/2), the up warps the others: each hands the other its half
      constexpr int HT = NT / 2;
#pragma unroll
      for (int t = 0; t < HT; ++t) exch[(half ? t : HT + t) * 128 + r] = half ? acc[t] : acc[HT + t];
      named_bar_sync(1, 256);
      const int t0 = half * HT;
      float act[HT];
#pragma unroll
      for (int t = 0; t < HT; ++t) {
        const float mine = half ? acc[HT + t] : acc[t], other = exch[(t0 + t) * 128 + r];
        act[t] = half ? silu_mul_fast(other, mine) : silu_mul_fast(mine, other);
        // largest magnitude of this token over the warp's 32 rows (non-negative floats order like their bits)
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(act[t])));
        if (lane == 0) part[(warp & 3) * NT + t0 + t] = __uint_as_float(m);
      }
      named_bar_sync(2 + half, 128);
#pragma unroll
      for (int t = 0; t < HT; ++t) {
        const float amax = fmaxf(fmaxf(fmaxf(part[t0 + t], part[NT + t0 + t]),
                                       fmaxf(part[2 * NT + t0 + t], part[3 * NT + t0 + t])), 1e-10f);
        const float q = act[t] * __fdividef(448.0f, amax);
        p.q_out[(int64_t)(row0 + t0 + t) * p.n_out + my_nt * 128 + r] =
            (uint8_t)__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3);
        if (r == t) p.q_scales[(int64_t)my_nt * p.q_ld + row0 + t0 + t] = __fdiv_rn(amax, 448.0f);
      }
      named_bar_sync(1, 256);  // exch and part are free again
    } else {
      const int col = my_nt * 256 + half * 128 + r;
      if (col < p.n_out) {
        OutT* out = static_cast<OutT*>(p.C) + col;
#pragma unroll
        for (int t = 0; t < NT; ++t)  // 32 lanes -> 32 consecutive columns of one (token, slot) row
          if (row_id[t] < p.numel) out[(int64_t)row_id[t] * p.n_out] = from_f32<OutT>(acc[t] * row_w[t]);
      }
    }
  };

  if (warp == kProducerWarp) {
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int item = item0; item < total && ok; item += step) {
        const int blk = item / p.n_tiles, nt = item - blk * p.n_tiles;
        const int e = p.expert_ids[blk];
        if (e < 0) continue;
        const int ra = weight_row(e, nt, 0), rb = weight_row(e, nt, 1);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = ptx::mbar_wait(empty_bar(s), phase, abort_flag);
          if (!ok) break;
          ptx::mbar_expect_tx(full_bar(s), Cfg::kStage);
          ptx::tma_load_2d(sW + s * Cfg::kStageW, &tmap_w, kb * kBK, ra, full_bar(s));
          ptx::tma_load_2d(sW + s * Cfg::kStageW + 128 * kBK, &tmap_w, kb * kBK, rb, full_bar(s));
          ptx::tma_load_2d(sX + s * Cfg::kStageX, &tmap_x, kb * kBK, blk * NT, full_bar(s));
          if (++s == S) s = 0, phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    if (ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::idesc_e4m3_f32(128, NT);
      int s = 0;
      uint32_t phase = 0, it = 0;
      bool ok = true;
      for (int item = item0; item < total && ok; item += step) {
        if (p.expert_ids[item / p.n_tiles] < 0) continue;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int b = it % NB;
          ok = ptx::mbar_wait(tempty_bar(b), ((it / NB) & 1) ^ 1, abort_flag) &&
               ptx::mbar_wait(full_bar(s), phase, abort_flag);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t dw = ptx::smem_desc_sw128(sW + s * Cfg::kStageW);
          const uint64_t dx = ptx::smem_desc_sw128(sX + s * Cfg::kStageX);
          const uint32_t d = tmem_base + b * 2 * NT;
#pragma unroll
          for (int h = 0; h < 2; ++h)  // + 128 rows of 128 bytes = + 1024 in the address field
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              ptx::mma_f8(d + h * NT, dw + h * 1024 + 2 * k, dx + 2 * k, idesc, k > 0);
          ptx::mma_commit(empty_bar(s));
          ptx::mma_commit(tfull_bar(b));
          if (++s == S) s = 0, phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp > kMmaWarp) {
    const int tid = threadIdx.x - (kMmaWarp + 1) * 32;  // 0..63
    uint32_t n_item = 0;
    for (int item = item0; item < total; item += step) {
      const int blk = item / p.n_tiles, nt = item - blk * p.n_tiles;
      const int e = p.expert_ids[blk];
      if (e < 0) continue;
      const int tb = n_item & 1;
      if (!ptx::mbar_wait(tab_empty_bar(tb), ((n_item >> 1) & 1) ^ 1, abort_flag)) break;
      float4* table = reinterpret_cast<float4*>(table_of(tb));
      constexpr int V = NT / 4;  // 16-byte vectors per K block: as_ld and the block's first row are multiples of 16
      const float* as = p.As + (int64_t)kb0 * p.as_ld + blk * NT;
#pragma unroll 8
      for (int i = tid; i < nkb * V; i += 64)
        table[i] = __ldg(reinterpret_cast<const float4*>(as + (int64_t)(i / V) * p.as_ld) + i % V);
      float* bs_tab = bs_tab_of(tb);
#pragma unroll 4
      for (int i = tid; i < 2 * nkb; i += 64) {
        const int h = i >= nkb, kb = i - h * nkb;
        bs_tab[h * p.table_kb + kb] = __ldg(p.Bs + (int64_t)scale_row(e, nt, h) * p.num_kb + kb0 + kb);
      }
      if (tid < NT) {
        const int flat = p.sorted_ids[blk * NT + tid];
        row_id_of(tb)[tid] = flat;
        row_w_of(tb)[tid] = p.topk_weights == nullptr ? 1.f : flat < p.numel ? __ldg(p.topk_weights + flat) : 0.f;
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(tab_full_bar(tb));
      ++n_item;
    }
    __syncwarp();
  } else {
    const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half * NT;
    uint32_t it = 0, n_item = 0;
    bool ok = true;
    for (int item = item0; item < total && ok; item += step) {
      const int blk = item / p.n_tiles, nt = item - blk * p.n_tiles;
      if (p.expert_ids[blk] < 0) continue;
      const int tb = n_item & 1;
      ok = ptx::mbar_wait(tab_full_bar(tb), (n_item >> 1) & 1, abort_flag);
      my_block = blk, my_nt = nt, my_buf = tb;
      const float *table = table_of(tb), *bs_tab = bs_tab_of(tb) + half * p.table_kb;
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[t] = 0.f;
      for (int j = 0; j < nkb && ok; ++j, ++it) {
        const int b = it % NB;
        ok = ptx::mbar_wait(tfull_bar(b), (it / NB) & 1, abort_flag);
        if (!ok) break;
        ptx::tc_fence_after();
        const float bs = bs_tab[j];
        const float4* sc = reinterpret_cast<const float4*>(table + j * NT);
        constexpr int CH = NT < 32 ? NT : 32;
#pragma unroll
        for (int c = 0; c < NT; c += CH) {
          uint32_t v[32];
          if (NT == 16) {
            ptx::tmem_ld16(lane_base + b * 2 * NT, v);
            ptx::tmem_ld_wait16(v);
          } else {
            ptx::tmem_ld32(lane_base + b * 2 * NT + c, v);
            ptx::tmem_ld_wait(v);
          }
          if (c + CH == NT) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(tempty_bar(b));
          }
#pragma unroll
          for (int q = 0; q < CH / 4; ++q) {
            const float4 s4 = sc[c / 4 + q];  // same address for every lane: broadcast
            acc[c + 4 * q + 0] = fmaf(__uint_as_float(v[4 * q + 0]), s4.x * bs, acc[c + 4 * q + 0]);
            acc[c + 4 * q + 1] = fmaf(__uint_as_float(v[4 * q + 1]), s4.y * bs, acc[c + 4 * q + 1]);
            acc[c + 4 * q + 2] = fmaf(__uint_as_float(v[4 * q + 2]), s4.z * bs, acc[c + 4 * q + 2]);
            acc[c + 4 * q + 3] = fmaf(__uint_as_float(v[4 * q + 3]), s4.w * bs, acc[c + 4 * q + 3]);
          }
        }
      }
      ++n_item;
      if (csize > 1) break;  // one item per cluster: finished below
      // a warp whose wait gave up must not leave the others alone at the barriers of the epilogue
      if (named_bar_any(1, 256, !ok)) break;
      epilogue();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(tab_empty_bar(tb));
    }
    if (csize > 1) sum_ok = !named_bar_any(1, 256, !ok);
  }

  if (csize > 1) {
    // the first CTA's ring is idle once every rank is here; the others add their sums there, [rank - 1][token][row]
    __syncwarp();
    ptx::cluster_sync();
    const bool live = warp < 8 && my_block >= 0 && sum_ok;
    if (live && rank > 0) {
      const uint32_t dst = ptx::mapa(smem_base, 0) + (((rank - 1) * NT) * 256 + half * 128 + r) * 4;
#pragma unroll
      for (int t = 0; t < NT; ++t) ptx::st_cluster_f32(dst + t * 1024, acc[t]);
    }
    __syncwarp();
    ptx::cluster_sync();
    if (live && rank == 0) {
      const float* src = reinterpret_cast<const float*>(smem_al) + half * 128 + r;
      for (int c = 1; c < (int)csize; ++c)  // rank order: the same sum on every run
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] += src[((c - 1) * NT + t) * 256];
      epilogue();
    }
  }

  if (*abort_flag) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(p.status, 0, 1);
  if (warp == kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// K split over a cluster when even one item per SM would leave at least half of the SMs without weights to
// stream: as many ranks (a power of two, at least two K blocks each) as bring items * ranks up to the SM count.
inline int stream_cluster(int64_t items, int num_kb, int sms, int nt) {
  int c = 1;
  while (c < 8 && items * c * 2 <= sms && num_kb >= 4 * c) c *= 2;
  // the sums of the other ranks must fit the first CTA's ring (at least three stages of it)
  while (c > 1 && (c - 1) * 256 * nt * 4 > 3 * (256 + nt) * kBK) c /= 2;
  return c;
}

// max_blocks: upper bound of the live NT-row blocks (the count is read on the device).
template <int NT, int STAGE, typename OutT>
inline int launch_stream(const void* W, int64_t w_rows, const void* X, int64_t x_rows, int64_t K, StreamParams p,
                         cudaStream_t st) {
  using Cfg = StreamCfg<NT>;
  const int sms = sm_count();
  p.num_kb = (int)cdiv(K, kBK);
  p.n_tiles = STAGE == STREAM_GATE_UP ? p.n_out / 128 : (int)cdiv(p.n_out, 256);
  const int64_t items = (int64_t)p.max_blocks * p.n_tiles;
  const int csize = stream_cluster(items, p.num_kb, sms, NT);
  p.kb_per_rank = (int)cdiv(p.num_kb, csize);
  p.table_kb = p.kb_per_rank;
  p.stages = Cfg::stages_for(p.table_kb);
  if (p.stages < 3) {
    set_error_detail("stream GEMM: K=%lld leaves %d stages of shared memory", (long long)K, p.stages);
    return B200_E_UNSUPPORTED;
  }
  p.status = device_status_word();
  if (!p.status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  p.w = static_cast<const uint8_t*>(W);
  CUtensorMap tw, tx;
  int rc = make_tmap_u8(&tw, W, (uint64_t)w_rows, (uint64_t)K, 128, "W");
  if (rc) return rc;
  rc = make_tmap_u8(&tx, X, (uint64_t)x_rows, (uint64_t)K, (uint32_t)NT, "X");
  if (rc) return rc;
  auto k = stream_gemm_kernel<NT, STAGE, OutT>;
  if (int rc_smem = allow_smem(k, Cfg::kSmemLimit, "stream_gemm_kernel")) return rc_smem;
  const int64_t grid = csize > 1 ? items * csize : items < sms ? items : sms;
  return launch_dependent(k, dim3((unsigned)grid), Cfg::kThreads, Cfg::smem_for(p.stages, p.table_kb), st, csize,
                          "stream_gemm_kernel", tw, tx, p);
}

}  // namespace b200
